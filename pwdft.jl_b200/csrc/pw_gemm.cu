// Complex GEMMs of the FP64 path, on the FP64 tensor cores (mma.sync
// m8n8k4, exact FP64 products and sums; tcgen05 has no FP64 kind), and FP32
// CUDA-core versions of the same products (PW_GEMM=cuda):
//   gemm_tn  C = A^H B      projections betaNL' psi (PsPotNL.jl:252) and the
//                           Rayleigh-Ritz Gram matrices X'HX, Q'HQ, Q'Q
//                           (diag_LOBPCG.jl:85,152-153,183-184); long K =
//                           Ngw is split across CTAs (deterministic two-pass
//                           reduction in FP64).
//   gemm_nn  C (+)= A B     betaNL * (D * P) (op_V_Ps_nloc.jl:59-76) and the
//                           subspace rotations Q*U, HQ*U (diag_LOBPCG.jl:188-194)
#include <algorithm>
#include <cmath>

#include "pw_launch.h"

namespace pwk {

namespace {

constexpr int TN_BM = 32, TN_BN = 32, TN_BK = 32;

template <typename T>
__global__ void __launch_bounds__(256)
k_gemm_tn(int64_t K, int m, int n, const Cx<T> *__restrict__ A, int64_t lda, const Cx<T> *__restrict__ B, int64_t ldb,
          double2 *__restrict__ W, int64_t kchunk, int upper) {
    __shared__ Cx<T> As[TN_BK][TN_BM + 1];
    __shared__ Cx<T> Bs[TN_BK][TN_BN + 1];
    const int m0 = blockIdx.x * TN_BM, n0 = blockIdx.y * TN_BN;
    if (upper && m0 > n0 + TN_BN - 1) return;  // tile strictly below the diagonal
    const int64_t kbeg = (int64_t)blockIdx.z * kchunk;
    const int64_t kend = min(K, kbeg + kchunk);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    Cx<T> acc[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j] = cmake((T)0, (T)0);
    for (int64_t k0 = kbeg; k0 < kend; k0 += TN_BK) {
        for (int e = threadIdx.x; e < TN_BK * TN_BM; e += 256) {
            const int kk = e % TN_BK, mm = e / TN_BK;
            const int64_t k = k0 + kk;
            As[kk][mm] = (k < kend && m0 + mm < m) ? A[(size_t)(m0 + mm) * lda + k] : cmake((T)0, (T)0);
            Bs[kk][mm] = (k < kend && n0 + mm < n) ? B[(size_t)(n0 + mm) * ldb + k] : cmake((T)0, (T)0);
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < TN_BK; ++kk) {
            Cx<T> a0 = As[kk][tx], a1 = As[kk][tx + 16];
            Cx<T> b0 = Bs[kk][ty], b1 = Bs[kk][ty + 16];
            acc[0][0] = cadd(acc[0][0], cmulc(a0, b0));
            acc[0][1] = cadd(acc[0][1], cmulc(a0, b1));
            acc[1][0] = cadd(acc[1][0], cmulc(a1, b0));
            acc[1][1] = cadd(acc[1][1], cmulc(a1, b1));
        }
        __syncthreads();
    }
    double2 *Wz = W + (size_t)blockIdx.z * m * n;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int mm = m0 + tx + 16 * i, nn = n0 + ty + 16 * j;
            if (mm < m && nn < n) Wz[(size_t)nn * m + mm] = make_double2((double)acc[i][j].x, (double)acc[i][j].y);
        }
}

// ------------------------------------------------------- FP64, tensor cores
// One CTA of four warps (2 x 2) forms a 16 WM x 16 WN tile of C, each warp
// WM x WN blocks of 8 x 8 complex values in registers: per step of four k it
// reads WM + WN fragments of 16 bytes a lane (one complex value) and issues
// 4 WM WN m8n8k4 products (Re Re, Im Im, Re Im, Im Re), so shared memory
// serves at most 0.4 of the time the FP64 pipe needs (64 multiply-adds a
// clock and SM).  Operands come in BK = 8 steps through a ring of three
// cp.async stages.  Rows are padded to 12 (k-contiguous operands) or 16 WM + 2
// (row-contiguous ones) complex values, which puts the eight lanes of each
// 128-byte phase of a fragment read on different banks.
// Sums: the 16 products of a step of eight k are summed from zero, then added to the
// accumulator, which so is rounded once in eight values.  Every instruction
// accumulating into the long sum (two roundings in four values, each of the long
// sum's size) is 2 to 15 % faster and loses accuracy: against extended precision, 180
// columns over 24,000 5.0e-15 against 4.8e-16 here and 1.7e-15 on CUDA cores; 480
// columns times 480 x 160 1.0e-15, 3.0e-16, 7.4e-16.
// TN: C = A^H B, A and B k-contiguous.  NN: C = A B, A row-contiguous.
// Bound by the FP64 pipe (36.9 TFLOP/s measured for a loop of nothing else).
// The 32 x 32 CUDA-core tiles before it were bound by shared-memory reads
// (two 16-byte reads per complex multiply-add and thread).  Measured, 480
// columns over K = 23,871 (Q'HQ, Q'Q and Q U of 160 bands together):
// 6.66 -> 3.01 ms, 27 TFLOP/s; op_H of 32 atoms (81 bands) 664 -> 546 us.
constexpr int ZBK = 8, ZST = 3, ZKP = ZBK + 4;
__device__ __forceinline__ void dmma0(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
                 : "=d"(c[0]), "=d"(c[1])
                 : "d"(a), "d"(b), "d"(0.0));
}
template <int WM, int WN, bool TN> constexpr size_t zgemm_smem() {
    return (size_t)ZST * ((TN ? 16 * WM * ZKP : ZBK * (16 * WM + 2)) + 16 * WN * ZKP) * sizeof(double2);
}

__device__ __forceinline__ void cp16(double2 *smem, const double2 *g, bool in) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    const int n = in ? 16 : 0;   // 0: the 16 bytes are zero-filled, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(g), "r"(n) : "memory");
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// k range of the CTA: [kbeg, kend).  direct: C is written (or added to)
// here, else the partial sums go to C[z][n][m] (ld m) for k_splitk_reduce.
// upper (TN): tiles strictly below the diagonal are skipped; 2: with direct, the
// other triangle gets the conjugates.  tri (NN):
// triangular structure the caller guarantees (the k-loop skips the zero
// blocks, whole tiles are skipped where no needed output lies):
//   1  A lower triangular (A[g][l] = 0 for l > g)
//   2  B upper triangular (B[l][j] = 0 for l > j) and only C[g][j], g <= j,
//      needed (tiles entirely below the diagonal are not formed)
//   3  A upper triangular (A[g][l] = 0 for l < g)
template <int WM, int WN, bool TN>
__global__ void __launch_bounds__(128, WM *WN >= 12 ? 2 : (WM * WN >= 6 ? 3 : 4))
k_zgemm(int64_t K, int64_t m, int n, const double2 *__restrict__ A, int64_t lda, const double2 *__restrict__ B,
        int64_t ldb, double2 *__restrict__ C, int64_t ldc, int64_t kchunk, int direct, int accumulate, int upper, int tri) {
    constexpr int BM = 16 * WM, BN = 16 * WN;
    constexpr int AP = TN ? ZKP : BM + 2;                       // row pitch of the A stage
    constexpr int ASZ = TN ? BM * ZKP : ZBK * (BM + 2), BSZ = BN * ZKP;
    extern __shared__ __align__(16) unsigned char zsm[];
    double2 *As = reinterpret_cast<double2 *>(zsm), *Bs = As + ZST * ASZ;
    const int64_t m0 = (int64_t)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    if (upper && m0 > n0 + BN - 1) return;
    if (!TN && tri == 2 && m0 > n0 + BN - 1) return;
    int64_t kbeg = (int64_t)blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
    if (!TN && tri == 1) kend = min(kend, m0 + BM);
    if (!TN && tri == 2) kend = min(kend, (int64_t)n0 + BN);
    if (!TN && tri == 3) kbeg = min(K, m0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp & 1) * 8 * WM, wn = (warp >> 1) * 8 * WN;
    const int g = lane >> 2, t = lane & 3;

    const int nk = kend > kbeg ? (int)((kend - kbeg + ZBK - 1) / ZBK) : 0;
    const int ck = tid & 7, cc = tid >> 3;                      // k-contiguous operands: 8 k x 16 columns a round
    auto load = [&](int it) {
        const int64_t k0 = kbeg + (int64_t)it * ZBK;
        double2 *as = As + (it % ZST) * ASZ, *bs = Bs + (it % ZST) * BSZ;
        const bool kin = k0 + ck < kend;
        if constexpr (TN) {
#pragma unroll
            for (int u = 0; u < WM; ++u) {
                const int64_t r = m0 + cc + 16 * u;
                const bool in = kin && r < m;
                cp16(&as[(cc + 16 * u) * ZKP + ck], in ? &A[(size_t)r * lda + k0 + ck] : A, in);
            }
        } else {
#pragma unroll
            for (int u = 0; u < WM; ++u) {
                const int e = tid + 128 * u, kk = e / BM, r = e - kk * BM;
                const bool in = k0 + kk < kend && m0 + r < m;
                cp16(&as[kk * AP + r], in ? &A[(size_t)(k0 + kk) * lda + m0 + r] : A, in);
            }
        }
#pragma unroll
        for (int u = 0; u < WN; ++u) {
            const int c = n0 + cc + 16 * u;
            const bool in = kin && c < n;
            cp16(&bs[(cc + 16 * u) * ZKP + ck], in ? &B[(size_t)c * ldb + k0 + ck] : B, in);
        }
    };

    double re[WM][WN][2], im[WM][WN][2];
#pragma unroll
    for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int j = 0; j < WN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
#pragma unroll
    for (int p = 0; p < ZST - 1; ++p) {
        if (p < nk) load(p);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int it = 0; it < nk; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ZST - 2) : "memory");
        __syncthreads();   // stage it has landed for every thread, and everyone is done with stage it - 1
        if (it + ZST - 1 < nk) load(it + ZST - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double2 *as = As + (it % ZST) * ASZ, *bs = Bs + (it % ZST) * BSZ;
        double2 b[2][WN];
#pragma unroll
        for (int j = 0; j < WN; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) b[h][j] = bs[(wn + 8 * j + g) * ZKP + 4 * h + t];
#pragma unroll
        for (int i = 0; i < WM; ++i) {
            double2 a[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                a[h] = TN ? as[(wm + 8 * i + g) * ZKP + 4 * h + t] : as[(4 * h + t) * AP + wm + 8 * i + g];
#pragma unroll
            for (int j0 = 0; j0 < WN; j0 += 2) {
                double tr[2][2], ti[2][2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int p = 0; p < 4; ++p)
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (j0 + u >= WN) continue;
                            const double2 bb = b[h][j0 + u];
                            if (p == 0) h ? dmma(tr[u], a[h].x, bb.x) : dmma0(tr[u], a[h].x, bb.x);
                            if (p == 1) h ? dmma(ti[u], a[h].x, bb.y) : dmma0(ti[u], a[h].x, bb.y);
                            if (p == 2) dmma(tr[u], TN ? a[h].y : -a[h].y, bb.y);
                            if (p == 3) dmma(ti[u], TN ? -a[h].y : a[h].y, bb.x);
                        }
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        if (j0 + u < WN) {
                            re[i][j0 + u][q] += tr[u][q];
                            im[i][j0 + u][q] += ti[u][q];
                        }
            }
        }
    }
    if (!direct) C += (size_t)blockIdx.z * m * n;
#pragma unroll
    for (int i = 0; i < WM; ++i) {
        const int64_t mm = m0 + wm + 8 * i + g;
#pragma unroll
        for (int j = 0; j < WN; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int nn = n0 + wn + 8 * j + 2 * t + q;
                if (mm < m && nn < n) {
                    double2 *p = direct ? &C[(size_t)nn * ldc + mm] : &C[(size_t)nn * m + mm];
                    const double2 v = make_double2(re[i][j][q], im[i][j][q]);
                    if (!(direct && upper && mm > nn)) *p = direct && accumulate ? cadd(*p, v) : v;
                    if (direct && upper == 2 && mm < nn) {
                        double2 *h = &C[(size_t)mm * ldc + nn];
                        const double2 cv = make_double2(v.x, -v.y);
                        *h = accumulate ? cadd(*h, cv) : cv;
                    }
                }
            }
    }
}

// Tile and split-K count of a product: the candidate with the shortest
// modelled time in clocks.  A CTA's tile costs 16 WM WN clocks of its SM's
// FP64 pipe per k, more by 0.8 (TN) or 0.3 (NN) times 1 / WM + 1 / WN for the
// fragments it reads per product, but not less than 45 (the ring waits for L2: 350
// clocks a step of 8), plus about 32 k for filling the ring and storing; the SM with
// the most CTAs decides, its last ones alone at 1.3 (one left over) or 1.05 (two) times
// their share; a split adds the partial sums' trip through L2 (about 2400 bytes a
// clock) and the reduction's launch (4000 clocks).  The three factors are a fit to 16
// products with each of the 15 tiles measured; the choice is within 5 % of the best
// there (A^H A of 180 columns over 24,000: 173 us with 64 x 64 tiles, 289 with the 32 x
// 16 ones that a model without them takes).  Splitting stops at four CTAs an SM, which also bounds the workspace: 592
// tiles, 49 MB, and up to about twice that for a triangular product, where only the
// formed tiles count but every split has room for all.  Few values are split too
// (betaNL' psi of 8 bands over about 730 plane waves: 35.8 us on one CTA, 5.0 in 23
// parts).
// fused: the caller's next pass sums the splits.
TnPlan zplan(int64_t K, int64_t m, int n, bool tn, int upper, bool fused = false) {
    TnPlan best{2, 2, 1, K, 0, 1};
    double tbest = 1e300;
    for (int wm = 2; wm <= 4; ++wm)
        for (int wn = 1; wn <= 5; ++wn) {
            if (!tn && wm == 3) continue;
            const int64_t tm = (m + 16 * wm - 1) / (16 * wm), tc = (n + 16 * wn - 1) / (16 * wn);
            if (tc > 65535 || (tn && tm > 65535)) continue;
            double tiles = (double)tm * (double)tc;
            if (upper) {
                tiles = 0;
                for (int64_t c = 0; c < tc; ++c) tiles += (double)std::min<int64_t>(tm, (c * 16 * wn + 16 * wn - 1) / (16 * wm) + 1);
            }
            const double f = 1.0 + (tn ? 0.8 : 0.3) * (1.0 / wm + 1.0 / wn);
            const int res = wm * wn >= 12 ? 2 : wm * wn >= 6 ? 3 : 4;   // CTAs that an SM holds
            // splits that fill whole rounds of the 148 SMs, or as many as
            // leave 32 values each
            for (int w = 0; w <= (tn ? 4 : 0); ++w) {
                const int S = w == 0 ? 1 : (int)std::min<int64_t>((int64_t)(148.0 * w / tiles), K / 32);
                if (w > 0 && S < 2) continue;
                const double kc = (double)((K + S - 1) / S);
                const int per = (int)std::ceil(tiles * S / 148.0), left = per % res;
                const double busy = per + (left == 1 ? 0.3 : left == 2 ? 0.1 : 0.0);
                double t = std::max(busy * 16.0 * wm * wn * f, 45.0) * (kc + 32.0);
                if (S > 1) t += (fused ? 0.0 : 4000.0) + (double)S * m * n * 32.0 / 2400.0;
                if (t < tbest * (1.0 - 1e-9)) {
                    tbest = t;
                    best = TnPlan{wm, wn, S, K, 0, 1};
                }
            }
        }
    const int64_t kc = (K + best.S - 1) / best.S;
    best.kchunk = (kc + ZBK - 1) / ZBK * ZBK;
    return best;
}

template <int WM, int WN, bool TN>
cudaError_t launch_z(const TnPlan &p, int64_t K, int64_t m, int n, const double2 *A, int64_t lda, const double2 *B,
                     int64_t ldb, double2 *C, int64_t ldc, int direct, int accumulate, int upper, int tri, cudaStream_t st) {
    constexpr size_t smem = zgemm_smem<WM, WN, TN>();
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_zgemm<WM, WN, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid((unsigned)((m + 16 * WM - 1) / (16 * WM)), (n + 16 * WN - 1) / (16 * WN), p.S);
    k_zgemm<WM, WN, TN><<<grid, 128, smem, st>>>(K, m, n, A, lda, B, ldb, C, ldc, p.kchunk, direct, accumulate, upper, tri);
    return cudaGetLastError();
}
template <bool TN>
cudaError_t launch_zgemm(const TnPlan &p, int64_t K, int64_t m, int n, const void *A, int64_t lda, const void *B, int64_t ldb,
                         double2 *C, int64_t ldc, int direct, int accumulate, int upper, int tri, cudaStream_t st) {
    const double2 *a = (const double2 *)A, *b = (const double2 *)B;
#define PW_Z(WM, WN)               \
    if (p.wm == WM && p.wn == WN) \
        return launch_z<WM, WN, TN>(p, K, m, n, a, lda, b, ldb, C, ldc, direct, accumulate, upper, tri, st);
#define PW_ZR(WM) PW_Z(WM, 1) PW_Z(WM, 2) PW_Z(WM, 3) PW_Z(WM, 4) PW_Z(WM, 5)
    PW_ZR(2)
    PW_ZR(4)
    if constexpr (TN) {
        PW_ZR(3)
    }
#undef PW_ZR
#undef PW_Z
    return cudaErrorInvalidValue;
}

// C[j ldc + i] (+)= sum over the S partial sums W[z][j][i].  upper: 1 = only
// i <= j is formed and written, 2 = only i <= j was formed and the other
// triangle gets its conjugate transpose (A^H A).
__device__ __forceinline__ void put_sum(double2 *C, int64_t ldc, int mm, int nn, double2 s, int accumulate, int upper) {
    double2 *p = &C[(size_t)nn * ldc + mm];
    *p = accumulate ? cadd(*p, s) : s;
    if (upper == 2 && mm < nn) {
        double2 *q = &C[(size_t)mm * ldc + nn];
        const double2 h = make_double2(s.x, -s.y);
        *q = accumulate ? cadd(*q, h) : h;
    }
}
__global__ void k_splitk_reduce(const double2 *__restrict__ W, int S, int m, int n, double2 *__restrict__ C, int64_t ldc,
                                int accumulate, int upper) {
    const size_t total = (size_t)m * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int nn = (int)(t / m), mm = (int)(t - (size_t)nn * m);
        if (upper && mm > nn) continue;
        double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int z = 0; z < S; ++z) s = cadd(s, W[(size_t)z * total + t]);
        put_sum(C, ldc, mm, nn, s, accumulate, upper);
    }
}
// The same with eight lanes to an element, for many parts and few elements (4 x 4
// values over 24,000 in FP64, 148 parts: the product 41 us with one thread an
// element, 14 with eight).
__global__ void k_splitk_reduce8(const double2 *__restrict__ W, int S, int m, int n, double2 *__restrict__ C, int64_t ldc,
                                 int accumulate, int upper) {
    const size_t total = (size_t)m * n;
    const int l8 = threadIdx.x & 7;
    for (size_t t0 = (blockIdx.x * (size_t)blockDim.x + (threadIdx.x & ~31)) >> 3; t0 < total;
         t0 += ((size_t)gridDim.x * blockDim.x) >> 3) {
        const size_t t = t0 + ((threadIdx.x & 31) >> 3);
        const int nn = (int)(t / m), mm = (int)(t - (size_t)nn * m);
        const bool in = t < total && !(upper && mm > nn);
        double2 s = make_double2(0.0, 0.0);
        if (in) {
#pragma unroll 4
            for (int z = l8; z < S; z += 8) s = cadd(s, W[(size_t)z * total + t]);
        }
        for (int o = 4; o > 0; o >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (in && l8 == 0) put_sum(C, ldc, mm, nn, s, accumulate, upper);
    }
}

constexpr int NN_BM = 64, NN_BN = 32, NN_BK = 16;

template <typename T>
__global__ void __launch_bounds__(256)
k_gemm_nn(int64_t M, int n, int k, const Cx<T> *__restrict__ A, int64_t lda, const double2 *__restrict__ B, int64_t ldb,
          Cx<T> *__restrict__ C, int64_t ldc, int accumulate) {
    __shared__ Cx<T> As[NN_BK][NN_BM];
    __shared__ Cx<T> Bs[NN_BK][NN_BN];
    const int64_t g0 = (int64_t)blockIdx.x * NN_BM;
    const int n0 = blockIdx.y * NN_BN;
    const int tg = threadIdx.x & 63, tn = threadIdx.x >> 6;  // 64 rows x 4 column groups of 8
    Cx<T> acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = cmake((T)0, (T)0);
    for (int j0 = 0; j0 < k; j0 += NN_BK) {
        for (int e = threadIdx.x; e < NN_BK * NN_BM; e += 256) {
            const int gg = e % NN_BM, jj = e / NN_BM;
            As[jj][gg] = (g0 + gg < M && j0 + jj < k) ? A[(size_t)(j0 + jj) * lda + g0 + gg] : cmake((T)0, (T)0);
        }
        for (int e = threadIdx.x; e < NN_BK * NN_BN; e += 256) {
            const int jj = e % NN_BK, nn = e / NN_BK;
            double2 v = (j0 + jj < k && n0 + nn < n) ? B[(size_t)(n0 + nn) * ldb + j0 + jj] : make_double2(0.0, 0.0);
            Bs[jj][nn] = cmake((T)v.x, (T)v.y);
        }
        __syncthreads();
#pragma unroll 4
        for (int jj = 0; jj < NN_BK; ++jj) {
            const Cx<T> a = As[jj][tg];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] = cadd(acc[q], cmul(a, Bs[jj][tn * 8 + q]));
        }
        __syncthreads();
    }
    const int64_t g = g0 + tg;
    if (g < M) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int nn = n0 + tn * 8 + q;
            if (nn < n) {
                Cx<T> *p = C + (size_t)nn * ldc + g;
                *p = accumulate ? cadd(*p, acc[q]) : acc[q];
            }
        }
    }
}

__global__ void k_dcsr(int nbeta, int nb, const int *__restrict__ rowptr, const int *__restrict__ col,
                       const double *__restrict__ val, const double2 *__restrict__ P, double2 *__restrict__ P2) {
    const size_t total = (size_t)nbeta * nb;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(t / nbeta), i = (int)(t - (size_t)b * nbeta);
        double2 s = make_double2(0.0, 0.0);
        for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
            const double2 p = P[(size_t)b * nbeta + col[e]];
            s.x += val[e] * p.x;
            s.y += val[e] * p.y;
        }
        P2[t] = s;
    }
}

// P2[b][i] = sum_j D[i][j] sum_z W[z][b][j]: the split-K sum of P = betaNL' psi and
// D P in one pass (P itself is not needed by op_V_Ps_nloc).
// Eight lanes share an element's splits (one thread summing 23 of them for 20 x 40
// values took 11 us).
__global__ void k_dcsr_splits(int nbeta, int nb, const int *__restrict__ rowptr, const int *__restrict__ col,
                              const double *__restrict__ val, const double2 *__restrict__ W, int S, double2 *__restrict__ P2) {
    const size_t total = (size_t)nbeta * nb;
    const int l8 = threadIdx.x & 7;
    for (size_t t0 = (blockIdx.x * (size_t)blockDim.x + (threadIdx.x & ~31)) >> 3; t0 < total;
         t0 += ((size_t)gridDim.x * blockDim.x) >> 3) {
        const size_t t = t0 + ((threadIdx.x & 31) >> 3);
        double2 s = make_double2(0.0, 0.0);
        if (t < total) {
            const int b = (int)(t / nbeta), i = (int)(t - (size_t)b * nbeta);
            for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
                const double2 *w = W + (size_t)b * nbeta + col[e];
                double2 p = make_double2(0.0, 0.0);
#pragma unroll 4
                for (int z = l8; z < S; z += 8) p = cadd(p, w[(size_t)z * total]);
                s.x += val[e] * p.x;
                s.y += val[e] * p.y;
            }
        }
        for (int o = 4; o > 0; o >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (t < total && l8 == 0) P2[t] = s;
    }
}

__global__ void k_c128_to_c64(const double2 *in, float2 *out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = make_float2((float)in[i].x, (float)in[i].y);
}
__global__ void k_c64_to_c128(const float2 *in, double2 *out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = make_double2((double)in[i].x, (double)in[i].y);
}
__global__ void k_d_to_f(const double *in, float *out, size_t n, double s) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (float)(in[i] * s);
}
__global__ void k_scale_d(const double *in, double *out, size_t n, double s) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = in[i] * s;
}

int blocks_for(size_t total) {
    size_t b = (total + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    return b < 1 ? 1 : (int)b;
}

int splitk_count(int64_t K, int m, int n) {
    const int tiles = ((m + TN_BM - 1) / TN_BM) * ((n + TN_BN - 1) / TN_BN);
    int64_t S = (600 + tiles - 1) / tiles;
    const int64_t Smax = (K + 255) / 256;
    if (S > Smax) S = Smax;
    if (S < 1) S = 1;
    return (int)S;
}

}  // namespace

TnPlan gemm_tn_plan(int real_bytes, int64_t K, int m, int n, int upper) {
    if (real_bytes == 8) {
        TnPlan p = zplan(K, m, n, true, upper);
        if (p.S > 1) {
            p.ws_bytes = (size_t)p.S * m * n * sizeof(double2);
            p.launches = 2;
        }
        return p;
    }
    TnPlan p{0, 0, splitk_count(K, m, n), 0, 0, 2};
    p.kchunk = ((K + p.S - 1) / p.S + TN_BK - 1) / TN_BK * TN_BK;
    p.ws_bytes = (size_t)p.S * m * n * sizeof(double2);
    return p;
}

template <typename T>
cudaError_t gemm_tn(const TnPlan &p, int64_t K, int m, int n, const void *A, int64_t lda, const void *B, int64_t ldb,
                    double2 *C, int64_t ldc, int accumulate, void *ws, cudaStream_t st, int upper) {
    if (m <= 0 || n <= 0) return cudaSuccess;
    const int S = p.S;
    cudaError_t e;
    if constexpr (sizeof(T) == 8) {
        const int direct = p.ws_bytes == 0;
        e = launch_zgemm<true>(p, K, m, n, A, lda, B, ldb, direct ? C : (double2 *)ws, ldc, direct, accumulate, upper, 0, st);
        if (e != cudaSuccess || direct) return e;
    } else {
        dim3 grid((m + TN_BM - 1) / TN_BM, (n + TN_BN - 1) / TN_BN, S);
        k_gemm_tn<T><<<grid, 256, 0, st>>>(K, m, n, (const Cx<T> *)A, lda, (const Cx<T> *)B, ldb, (double2 *)ws, p.kchunk, upper);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const size_t total = (size_t)m * n;
    if (S >= 16 && total <= 65536)
        k_splitk_reduce8<<<blocks_for(total * 8), 256, 0, st>>>((const double2 *)ws, S, m, n, C, ldc, accumulate, upper);
    else
        k_splitk_reduce<<<blocks_for(total), 256, 0, st>>>((const double2 *)ws, S, m, n, C, ldc, accumulate, upper);
    return cudaGetLastError();
}

template <typename T>
cudaError_t gemm_nn(int64_t M, int n, int k, const void *A, int64_t lda, const double2 *B, int64_t ldb, void *C,
                    int64_t ldc, int accumulate, cudaStream_t st, int tri) {
    if (M <= 0 || n <= 0) return cudaSuccess;
    if constexpr (sizeof(T) == 8) {
        return launch_zgemm<false>(zplan(k, M, n, false, tri == 2), k, M, n, A, lda, B, ldb, (double2 *)C, ldc, 1, accumulate,
                                   0, tri, st);
    } else {
        dim3 grid((unsigned)((M + NN_BM - 1) / NN_BM), (n + NN_BN - 1) / NN_BN);
        k_gemm_nn<T><<<grid, 256, 0, st>>>(M, n, k, (const Cx<T> *)A, lda, B, ldb, (Cx<T> *)C, ldc, accumulate);
        return cudaGetLastError();
    }
}

template cudaError_t gemm_tn<float>(const TnPlan &, int64_t, int, int, const void *, int64_t, const void *, int64_t, double2 *, int64_t,
                                    int, void *, cudaStream_t, int);
template cudaError_t gemm_tn<double>(const TnPlan &, int64_t, int, int, const void *, int64_t, const void *, int64_t, double2 *, int64_t,
                                     int, void *, cudaStream_t, int);
template cudaError_t gemm_nn<float>(int64_t, int, int, const void *, int64_t, const double2 *, int64_t, void *, int64_t,
                                    int, cudaStream_t, int);
template cudaError_t gemm_nn<double>(int64_t, int, int, const void *, int64_t, const double2 *, int64_t, void *, int64_t,
                                     int, cudaStream_t, int);

size_t project_ws_bytes(int64_t K, int nbeta, int nb) {
    return (size_t)zplan(K, nbeta, nb, true, 0, true).S * nbeta * nb * sizeof(double2);
}
cudaError_t project_dcsr(int64_t K, int nbeta, int nb, const double2 *beta, const double2 *psi, int64_t ldp, const int *rowptr,
                         const int *col, const double *val, double2 *P2, void *ws, cudaStream_t st) {
    const TnPlan p = zplan(K, nbeta, nb, true, 0, true);
    cudaError_t e = launch_zgemm<true>(p, K, nbeta, nb, beta, K, psi, ldp, (double2 *)ws, 0, 0, 0, 0, 0, st);
    if (e != cudaSuccess) return e;
    k_dcsr_splits<<<blocks_for((size_t)nbeta * nb * 8), 256, 0, st>>>(nbeta, nb, rowptr, col, val, (const double2 *)ws, p.S, P2);
    return cudaGetLastError();
}
cudaError_t apply_dcsr(int nbeta, int nb, const int *rowptr, const int *col, const double *val, const double2 *P,
                       double2 *P2, cudaStream_t st) {
    k_dcsr<<<blocks_for((size_t)nbeta * nb), 256, 0, st>>>(nbeta, nb, rowptr, col, val, P, P2);
    return cudaGetLastError();
}
cudaError_t convert_c128_to_c64(const double2 *in, float2 *out, size_t n, cudaStream_t st) {
    k_c128_to_c64<<<blocks_for(n), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t convert_c64_to_c128(const float2 *in, double2 *out, size_t n, cudaStream_t st) {
    k_c64_to_c128<<<blocks_for(n), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t convert_d_to_f(const double *in, float *out, size_t n, double scale, cudaStream_t st) {
    k_d_to_f<<<blocks_for(n), 256, 0, st>>>(in, out, n, scale);
    return cudaGetLastError();
}
cudaError_t scale_d(const double *in, double *out, size_t n, double scale, cudaStream_t st) {
    k_scale_d<<<blocks_for(n), 256, 0, st>>>(in, out, n, scale);
    return cudaGetLastError();
}

}  // namespace pwk
