// FP32 density plane pass for any pair of fused line lengths (pw_fft_any.cuh).
#include "pw_fft_any.cuh"

namespace pwk {
template <>
cudaError_t launch_any_plane_rho<float>(const FftLaunch &L, const void *A, int nb, int G, int Bg, const double *w, void *rho_part,
                                     cudaStream_t st, int *per_sm) {
    return any::plane_rho<float>(L, A, nb, G, Bg, w, rho_part, st, per_sm);
}
}  // namespace pwk
