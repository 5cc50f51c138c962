// FP64 op_V_loc plane pass for any pair of fused line lengths (pw_fft_any.cuh).
#include "pw_fft_any.cuh"

namespace pwk {
template <> cudaError_t launch_any_plane_vloc<double>(const FftLaunch &L, const void *Vr, void *A, int nb, cudaStream_t st) {
    return any::plane_vloc<double>(L, Vr, A, nb, st);
}
}  // namespace pwk
