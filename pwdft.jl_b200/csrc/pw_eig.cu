// FP64 small dense Hermitian (generalised) eigensolver on the GPU: the
// eigen(T, G) / eigvals(XHX) / eigen(S) calls of diag_LOBPCG.jl:86,185,216
// (LAPACK zhegv / zheev in the reference).
//
//   1. hermitise T and G from their upper triangles (Julia's Hermitian(A))
//   2. G = L L^H                        blocked right-looking elimination of
//   3. Linv = L^-1                      [G | I] on 32 x 32 tiles, two grid
//                                       barriers per 32-column panel
//                                       (cooperative kernel)
//   4. C = Linv T Linv^H                two FP64 complex GEMMs
//   5. C = Q Tr Q^H                     Householder tridiagonalisation (LAPACK
//                                       zhetd2 conventions: H = I - tau v v^H,
//                                       real tridiagonal Tr): the last 256
//                                       columns in one cluster's registers,
//                                       those before in registers across the
//                                       grid (n <= 1024) or in L2 with one grid
//                                       barrier per column
//   6. lowest k eigenvalues of Tr       multisection on Sturm counts, one warp
//                                       per eigenvalue; the block reflectors
//                                       of step 8 meanwhile
//   7. eigenvectors of Tr               inverse iteration (tridiagonal LU with
//                                       partial pivoting), re-orthogonalised
//                                       (modified Gram-Schmidt) inside clusters
//                                       of near-degenerate eigenvalues, one
//                                       warp per cluster
//   8. Z = Q Ztr                        block reflectors (32 columns) applied
//                                       in reverse order, 1-4 eigenvectors a CTA
//   9. S = Linv^H Z                     FP64 complex GEMM
// The cooperative kernels synchronise with a grid barrier of their own whose
// waits are bounded; on expiry they record an error and run to completion.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "pw_eig.h"
#include "pw_launch.h"
#include "pw_tri.h"

namespace pwk {
namespace eig {

constexpr long long GSYNC_LIMIT = 1ll << 22;   // acquire polls of gsync (a few seconds)
constexpr int COOP_THREADS = 256;
constexpr int TU = 8;   // global loads kept in flight per thread in the tridiagonalisation

struct GridBar {  // barrier counter storage
    unsigned int count;
    unsigned int gen;
};

// Bounded grid-wide barrier on a monotonic counter (zeroed before the
// launch): every CTA adds one and waits until the counter reaches the
// number of CTAs times the barriers passed so far.  `tgt` is the calling
// CTA's running target (same value in every thread).
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Failure-detection test hooks, written only through pwk_test_gsync (a
// test-only export): the poll limit of every wait, and one CTA that withholds
// its arrivals so that the others' waits run out.  The library itself never
// changes them.
__device__ long long g_gsync_limit = GSYNC_LIMIT;
__device__ int g_gsync_withhold = -1;

__device__ __forceinline__ void gsync(unsigned *ctr, unsigned &tgt, int *err) {
    __syncthreads();
    tgt += gridDim.x;
    if (threadIdx.x == 0) {
        __threadfence();
        if ((int)blockIdx.x != g_gsync_withhold) atomicAdd(ctr, 1u);
        if (!*(volatile int *)err) {
            const long long lim = g_gsync_limit;
            long long it = 0;
            while (ld_acquire_u32(ctr) < tgt) {
                if (++it > lim) {
                    atomicExch(err, 1);
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
}

__device__ __forceinline__ double2 cmulc_d(double2 a, double2 b) {  // conj(a) b
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double2 cmul_d(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

template <typename V>
__device__ V block_sum(V v, V *red) {
    for (int o = 16; o > 0; o >>= 1) {
        if constexpr (sizeof(V) == sizeof(double2)) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        } else {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    V s = red[0];
    for (int i = 1; i < nw; ++i) {
        if constexpr (sizeof(V) == sizeof(double2)) {
            s.x += red[i].x;
            s.y += red[i].y;
        } else {
            s += red[i];
        }
    }
    return s;
}

// A (n x n, column-major): lower := conj(upper)^T, diagonal made real.
__global__ void k_herm_upper(double2 *A, int n) {
    const size_t total = (size_t)n * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / n), i = (int)(t - (size_t)j * n);
        if (i > j) {
            const double2 u = A[(size_t)i * n + j];
            A[t] = make_double2(u.x, -u.y);
        } else if (i == j) {
            A[t].y = 0.0;
        }
    }
}

__global__ void k_conj_transpose(const double2 *__restrict__ A, double2 *__restrict__ B, int n) {
    const size_t total = (size_t)n * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / n), i = (int)(t - (size_t)j * n);
        const double2 a = A[(size_t)i * n + j];
        B[t] = make_double2(a.x, -a.y);
    }
}

// ---------------------------------------------------------------- blocked
// Cholesky and triangular inverse on 32 x 32 tiles, in one elimination of the
// augmented matrix [G | I] -> [L^H | L^-1] (cooperative kernel).
constexpr int TB = 32;
constexpr int TLD = TB + 1;  // leading dimension of the diagonal block (row-major)
constexpr int KLD = TB + 2;  // tiles stored [k][row]: the 8 lanes of a 128-byte phase of a fragment
constexpr int CLD = TB + 4;  // read (4 k x 2 rows) fall on different banks; tiles stored [column][k]

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Cholesky of the diagonal block at (p, p) (rows and columns past n read as
// the unit matrix) into D (row-major, ld TLD, lower part), 1 / L_tt into rdiag.
// Right-looking with the elements in registers (thread (tx, ty) owns rows
// tx + 16 a, columns ty + 16 b): a step publishes one raw column, and
// everyone subtracts raw_r conj(raw_c) / pivot; one block barrier a step.
// Returns the first failing local column + 1, or 0; a non-positive pivot is
// replaced by a tiny one so the factorisation runs to completion.
__device__ int chol_tile(const double2 *A, int n, int p, double2 *D, double *rdiag, double2 (*col)[TB]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double2 v[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int r = tx + 16 * a, c = ty + 16 * b;
            v[a][b] = (p + r < n && p + c < n) ? __ldcg(&A[(size_t)(p + c) * n + p + r]) : make_double2(r == c ? 1.0 : 0.0, 0.0);
        }
    int fail = 0;
#pragma unroll
    for (int b = 0; b < 2; ++b)
        for (int tt = 0; tt < 16; ++tt) {
            const int t = 16 * b + tt;
            double2 *cb = col[t & 1];
            if (ty == tt) {
                cb[tx] = v[0][b];
                cb[tx + 16] = v[1][b];
            }
            __syncthreads();   // the buffer two steps back is free: everyone passed the last barrier after reading it
            const double dt = cb[t].x;
            if (!(dt > 0.0) && fail == 0) fail = t + 1;
            const double inv = 1.0 / fmax(dt, 1e-300);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double2 rc = cb[ty + 16 * q];
                const double2 f = make_double2(rc.x * inv, -rc.y * inv);
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    if (ty + 16 * q > t) {
                        const double2 m = cmul_d(cb[tx + 16 * a], f);
                        v[a][q].x -= m.x;
                        v[a][q].y -= m.y;
                    }
                }
            }
            // column t stays raw in its owners' registers; its scale 1 / sqrt(pivot)
            if (threadIdx.x == t) rdiag[t] = 1.0 / sqrt(fmax(dt, 1e-300));
        }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int r = tx + 16 * a, c = ty + 16 * b;
            D[r * TLD + c] = make_double2(v[a][b].x * rdiag[c], v[a][b].y * rdiag[c]);
        }
    return fail;
}

// G = L L^H and X = L^-1 together, right-looking over 32-column panels:
//   phase 1 (one warp per row or column, after every CTA has factored the
//           diagonal block L11 for itself): the panel rows L21 = A21 L11^-H
//           and the block row X_p = L11^-1 X_p, by substitution;
//   barrier;
//   phase 2: A_IJ -= L_I L_J^H on the lower trailing tiles and
//           X_IJ -= L_I X_pJ below the block row (cyclic over CTAs), on the
//           FP64 tensor cores;
//   barrier.
// G's lower triangle is overwritten, its upper triangle left; X is written in
// full (zero above the diagonal).  info = first failing column (1-based) or 0.
// Latency-bound (15 panels at n = 480): 306 us at n = 480 and 117 us at n = 160;
// two kernels, Cholesky and inverse, with three block barriers a column in the
// diagonal block, took 549 + 307 and 181 + 109 us.
constexpr size_t CHOL_SMEM = (size_t)(TB * TLD + 2 * TB * CLD) * sizeof(double2);
__global__ void __launch_bounds__(COOP_THREADS) k_chol_inv(double2 *A, double2 *X, int n, unsigned *ctr, int *err, int *info) {
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *D = reinterpret_cast<double2 *>(sm);  // diagonal block
    double2 *Ta = D + TB * TLD;                     // L_I, [k][row]
    double2 *Tb = Ta + TB * CLD;                    // L_J, [k][row], or X_pJ, [column][k]
    __shared__ double rdiag[TB];
    __shared__ double2 col[2][TB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = COOP_THREADS >> 5;
    unsigned tgt = 0;
    for (int p = 0; p < n; p += TB) {
        const int bs = min(TB, n - p), q0 = p + bs, P = p / TB;
        // the first row or column of this warp: loaded before the factorisation
        auto load = [&](int i) {
            double2 z = make_double2(0.0, 0.0);
            if (lane >= bs) return z;
            if (i >= q0) return i < n ? __ldcg(&A[(size_t)(p + lane) * n + i]) : z;                 // row i of A21
            if (i >= p) return make_double2(i - p == lane ? 1.0 : 0.0, 0.0);                        // X_pp = I
            return __ldcg(&X[(size_t)i * n + p + lane]);                                             // column i of X_p
        };
        const int i0 = blockIdx.x * nw + warp, step = gridDim.x * nw;
        double2 acc = i0 < n ? load(i0) : make_double2(0.0, 0.0);
        const int f = chol_tile(A, n, p, D, rdiag, col);
        if (f && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(info, 0, p + f);
        __syncthreads();
        // l[t] = (a[t] - sum_{s<t} l[s] L11[t][s]^(*)) / L11[t][t], lane t holding
        // entry t: conjugated for the rows of L21, plain for the columns of X
        for (int i = i0; i < n; i += step) {
            if (i != i0) acc = load(i);
            const double cj = i >= q0 ? -1.0 : 1.0;
            double2 l = make_double2(0.0, 0.0);
#pragma unroll 8
            for (int s = 0; s < TB; ++s) {
                const double is = rdiag[s];
                const double2 ls = make_double2(__shfl_sync(0xffffffffu, acc.x, s) * is, __shfl_sync(0xffffffffu, acc.y, s) * is);
                if (lane == s) l = ls;
                if (lane > s) {
                    double2 m = D[lane * TLD + s];
                    m.y *= cj;
                    const double2 q = cmul_d(m, ls);
                    acc.x -= q.x;
                    acc.y -= q.y;
                }
            }
            if (lane < bs) {
                if (i >= q0)
                    A[(size_t)(p + lane) * n + i] = l;
                else
                    X[(size_t)i * n + p + lane] = l;
            }
        }
        // zeros above X's block diagonal (nobody reads them here)
        for (int e = blockIdx.x * COOP_THREADS + threadIdx.x; e < p * bs; e += gridDim.x * COOP_THREADS)
            X[(size_t)(p + e / p) * n + e % p] = make_double2(0.0, 0.0);
        gsync(ctr, tgt, err);
        if (q0 >= n) break;
        const int nt = (n - q0 + TB - 1) / TB, ng = nt * (nt + 1) / 2, ntile = ng + nt * (P + 1);
        for (int tt = blockIdx.x; tt < ntile; tt += gridDim.x) {
            int I, J;
            const bool isx = tt >= ng;
            if (isx) {
                I = (tt - ng) % nt;
                J = (tt - ng) / nt;
            } else {
                I = 0;
                int rem = tt;
                while (rem > I) {
                    rem -= I + 1;
                    ++I;
                }
                J = rem;
            }
            const int r0 = q0 + I * TB, c0 = isx ? J * TB : q0 + J * TB;
            double2 *M = isx ? X : A;
            // this lane's entries of the target: rows rr, columns cc .. cc + 1 of two 8 x 8 blocks
            const int g = lane >> 2, t4 = lane & 3, rr = r0 + (warp & 3) * 8 + g;
            double2 old[2][2];
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int cc = c0 + (warp >> 2) * 16 + 8 * b + 2 * t4 + q;
                    // X's block column p starts from zero
                    old[b][q] = rr < n && cc < n && !(isx && J == P) ? __ldcg(&M[(size_t)cc * n + rr]) : make_double2(0.0, 0.0);
                }
#pragma unroll
            for (int e = threadIdx.x; e < TB * TB; e += COOP_THREADS) {
                const int hi = e / TB, lo = e % TB;
                Ta[hi * KLD + lo] = hi < bs && r0 + lo < n ? __ldcg(&A[(size_t)(p + hi) * n + r0 + lo]) : make_double2(0.0, 0.0);
                if (isx)
                    Tb[hi * CLD + lo] = lo < bs ? __ldcg(&X[(size_t)(c0 + hi) * n + p + lo]) : make_double2(0.0, 0.0);
                else
                    Tb[hi * KLD + lo] = hi < bs && c0 + lo < n ? __ldcg(&A[(size_t)(p + hi) * n + c0 + lo]) : make_double2(0.0, 0.0);
            }
            __syncthreads();
            double re[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, im[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
            const int ra = (warp & 3) * 8 + g;
#pragma unroll
            for (int kk = 0; kk < TB; kk += 4) {
                const double2 a = Ta[(kk + t4) * KLD + ra];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int cb = (warp >> 2) * 16 + 8 * b + g;
                    double2 m = isx ? Tb[cb * CLD + kk + t4] : Tb[(kk + t4) * KLD + cb];
                    if (!isx) m.y = -m.y;
                    dmma(re[b], a.x, m.x);
                    dmma(im[b], a.x, m.y);
                    dmma(re[b], -a.y, m.y);
                    dmma(im[b], a.y, m.x);
                }
            }
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int cc = c0 + (warp >> 2) * 16 + 8 * b + 2 * t4 + q;
                    if (rr < n && cc < n && (isx || rr >= cc))
                        M[(size_t)cc * n + rr] = make_double2(old[b][q].x - re[b][q], old[b][q].y - im[b][q]);
                }
            __syncthreads();
        }
        gsync(ctr, tgt, err);
    }
}

// Householder tridiagonalisation of the Hermitian C (full storage), LAPACK
// zhetd2 (lower) conventions: H_j = I - tau_j v_j v_j^H with v_j[j+1] = 1,
// real tridiagonal (d, e); v_j is left in C[j+2:n, j].  One grid barrier per
// column:
//   phase M (distributed): the owner of each trailing column i > j applies
//     the previous step's rank-2 update  A -= v w^H + w v^H  to rows > j and,
//     in the same pass, forms y_i = (column i)^H v_j;
//   barrier;
//   phase R (every CTA, redundantly): w_j = tau y + alpha v_j with
//     alpha = -tau/2 (tau y)^H v_j; the next column j+1 is read, given the
//     step-j update, and its Householder vector v_{j+1} formed.
// Every CTA therefore holds v_j, w_j, v_{j-1}, w_{j-1} in shared memory and
// the trailing matrix is read and written once per column.  y alternates
// between two buffers so that a CTA running ahead into the next phase M
// cannot overwrite values a slower CTA still reads.
__global__ void __launch_bounds__(COOP_THREADS)
k_tridiag(double2 *C, int n, int jend, double *d, double *e, double2 *tau, double2 *ybuf, unsigned *ctr, int *err) {
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *vc = reinterpret_cast<double2 *>(sm);  // v_j         [n]
    double2 *vp = vc + n;                           // v_{j-1}     [n]
    double2 *wp = vp + n;                           // w_{j-1}     [n]
    double2 *red = wp + n;                          // [32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned tgt = 0;
    double2 tj = make_double2(0.0, 0.0);

    // Householder vector of x = vc[j+1 .. n) in place (vc[j] := 0,
    // vc[j+1] := 1); returns tau.  CTA 0 records e[j] = beta and tau[j].
    auto householder = [&](int j) -> double2 {
        double s2 = 0.0;
        for (int i = j + 2 + threadIdx.x; i < n; i += blockDim.x) s2 += vc[i].x * vc[i].x + vc[i].y * vc[i].y;
        s2 = block_sum<double>(s2, (double *)red);
        const double2 alpha = vc[j + 1];
        double2 t, scal;
        double beta;
        if (s2 == 0.0 && alpha.y == 0.0) {
            t = make_double2(0.0, 0.0);
            beta = alpha.x;
            scal = make_double2(0.0, 0.0);
        } else {
            beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s2), alpha.x);
            t = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
            const double ar = alpha.x - beta, ai = alpha.y, den = ar * ar + ai * ai;
            scal = make_double2(ar / den, -ai / den);
        }
        __syncthreads();  // everyone has read vc[j+1]
        for (int i = j + threadIdx.x; i < n; i += blockDim.x)
            vc[i] = (i == j) ? make_double2(0.0, 0.0) : (i == j + 1) ? make_double2(1.0, 0.0) : cmul_d(vc[i], scal);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            e[j] = beta;
            tau[j] = t;
        }
        __syncthreads();
        return t;
    };

    // column 0
    for (int i = threadIdx.x; i < n; i += blockDim.x) vc[i] = __ldcg(&C[i]);
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) d[0] = vc[0].x;
    if (n >= 2) tj = householder(0);

    for (int j = 0; j < jend; ++j) {
        double2 *yb = ybuf + (size_t)(j & 1) * n;
        // ---- phase M: update owned columns i > j with (v_{j-1}, w_{j-1}), y_i = col_i^H v_j
        for (int i = j + 1 + blockIdx.x + gridDim.x * warp; i < n; i += gridDim.x * nw) {
            double2 *col = C + (size_t)i * n;
            double2 acc = make_double2(0.0, 0.0);
            // (v, w) = (0, 0) at j = 0: no previous update
            const double2 cw = j > 0 ? make_double2(wp[i].x, -wp[i].y) : make_double2(0.0, 0.0);
            const double2 cv = j > 0 ? make_double2(vp[i].x, -vp[i].y) : make_double2(0.0, 0.0);
            // TU loads in flight per lane: the column streams from L2
            for (int r0 = j + 1 + lane; r0 < n; r0 += 32 * TU) {
                double2 a[TU];
#pragma unroll
                for (int u = 0; u < TU; ++u) {
                    const int r = r0 + 32 * u;
                    a[u] = r < n ? __ldcg(&col[r]) : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int u = 0; u < TU; ++u) {
                    const int r = r0 + 32 * u;
                    if (r < n) {
                        if (j > 0) {
                            const double2 p = cmul_d(vp[r], cw), q = cmul_d(wp[r], cv);
                            a[u].x -= p.x + q.x;
                            a[u].y -= p.y + q.y;
                            col[r] = a[u];
                        }
                        const double2 s = cmulc_d(a[u], vc[r]);
                        acc.x += s.x;
                        acc.y += s.y;
                    }
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            if (lane == 0) yb[i] = acc;
        }
        gsync(ctr, tgt, err);
        // ---- phase R (redundant).  Column j is no longer read by anyone:
        // its owner stores v_j there for the back-transformation.
        if ((j % gridDim.x) == blockIdx.x)
            for (int i = j + 2 + threadIdx.x; i < n; i += blockDim.x) C[(size_t)j * n + i] = vc[i];
        // v_{j-1}, w_{j-1} are dead now.  One batch of loads brings in both
        // y (scaled by tau, into wp) and the raw next column j+1 (into vp).
        const int c1 = j + 1;
        const double2 *col = C + (size_t)c1 * n;
        for (int base = threadIdx.x; base < n; base += blockDim.x * TU) {
            double2 ya[TU], ca[TU];
#pragma unroll
            for (int u = 0; u < TU; ++u) {
                const int i = base + u * blockDim.x;
                ya[u] = (i > j && i < n) ? __ldcg(&yb[i]) : make_double2(0.0, 0.0);
                ca[u] = (i >= c1 && i < n) ? __ldcg(&col[i]) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < TU; ++u) {
                const int i = base + u * blockDim.x;
                if (i < n) {
                    wp[i] = cmul_d(tj, ya[u]);
                    vp[i] = ca[u];
                }
            }
        }
        __syncthreads();
        // w_j = tau y + alpha v_j, alpha = -tau/2 (tau y)^H v_j
        double2 yv = make_double2(0.0, 0.0);
        for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) {
            const double2 s = cmulc_d(wp[i], vc[i]);
            yv.x += s.x;
            yv.y += s.y;
        }
        yv = block_sum<double2>(yv, red);
        const double2 al = cmul_d(make_double2(-0.5 * tj.x, -0.5 * tj.y), yv);
        for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) {
            const double2 p = cmul_d(al, vc[i]);
            wp[i].x += p.x;
            wp[i].y += p.y;
        }
        __syncthreads();
        // v_j becomes v_{j-1} for the next step; the next column (in the
        // old v_{j-1} buffer) becomes vc and gets the step-j update
        double2 *t = vp;
        vp = vc;
        vc = t;
        const double2 cw = make_double2(wp[c1].x, -wp[c1].y), cv = make_double2(vp[c1].x, -vp[c1].y);
        for (int r = c1 + threadIdx.x; r < n; r += blockDim.x) {
            const double2 p = cmul_d(vp[r], cw), q = cmul_d(wp[r], cv);
            vc[r].x -= p.x + q.x;
            vc[r].y -= p.y + q.y;
        }
        __syncthreads();
        if (blockIdx.x == 0 && threadIdx.x == 0) d[c1] = vc[c1].x;
        if (c1 < jend) tj = householder(c1);
    }
    // the trailing matrix from column jend on, with the last step's update, for
    // the next kernel
    if (jend < n - 1) {
        gsync(ctr, tgt, err);   // everyone has read column jend
        for (int i = jend + blockIdx.x; i < n; i += gridDim.x) {
            const double2 cw = make_double2(wp[i].x, -wp[i].y), cv = make_double2(vp[i].x, -vp[i].y);
            for (int r = jend + threadIdx.x; r < n; r += blockDim.x) {
                const double2 p = cmul_d(vp[r], cw), q = cmul_d(wp[r], cv), a = __ldcg(&C[(size_t)i * n + r]);
                C[(size_t)i * n + r] = make_double2(a.x - (p.x + q.x), a.y - (p.y + q.y));
            }
        }
    }
}

// The same tridiagonalisation for n <= 1024 with the trailing matrix in
// registers (CPW columns a warp, row lane + 32 u in register u) and no grid
// barrier.  What the CTAs exchange per column, for each column i > j its y_i =
// (column i)^H v_j and its entry of row j + 1 (the conjugate of column j + 1, by
// symmetry), is written once to its own place (ybuf, filled with all-ones words
// before the launch), and every CTA reads it as soon as the words it polls are
// there: the data is its own flag, and a column costs one store-to-load trip
// through L2 instead of a fence, an atomic, a poll and then the loads.  A CTA's
// values lie together and leave in one store: with eight SMs writing to a line
// that others poll, a column took 1.5 to 3 us more.  Each thread keeps its EPT
// elements of v_j in registers through the redundant step (y, the next column
// and its Householder vector), which takes three block barriers.  A word that
// stays all-ones past the poll limit sets *err, after which nobody waits long
// any more.  Latency-bound: n = 160 / 480 / 900 take 0.54 / 1.95 / 4.72 ms, the
// grid-barrier kernel 0.78 / 2.71 / 6.21 ms.
__device__ __forceinline__ bool unset(double2 v) {
    return __double_as_longlong(v.x) == -1ll || __double_as_longlong(v.y) == -1ll;
}
__device__ __forceinline__ double2 ld_relaxed(const double2 *p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(double2 *p, double2 v) {
    // a NaN that carries the all-ones pattern would read as "not there yet"
    if (__double_as_longlong(v.x) == -1ll) v.x = __longlong_as_double(0x7ff8000000000000ll);
    if (__double_as_longlong(v.y) == -1ll) v.y = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}

// Warp sum of a complex value: the real part in lanes 0..15, the imaginary
// part in lanes 16..31.
__device__ __forceinline__ double half_sums(double2 v, int lane) {
    const double o = __shfl_xor_sync(0xffffffffu, lane < 16 ? v.y : v.x, 16);
    double s = (lane < 16 ? v.x : v.y) + o;
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    return s;
}

template <int NR, int W, int CPW>
__global__ void __launch_bounds__(32 * W)
k_tridiag_r(double2 *C, int n, int jend, double *d, double *e, double2 *tau, double2 *ybuf, int *err) {
    constexpr int TH = 32 * W, EPT = 32 * NR / TH, NN = 32 * NR;
    static_assert(EPT * TH == NN, "every row has a thread");
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *vc = reinterpret_cast<double2 *>(sm), *vp = vc + NN, *wp = vp + NN;   // v_j, v_{j-1}, w_{j-1}
    constexpr int SL = W * CPW;                      // columns of a CTA
    __shared__ double2 ysm[2 * SL];                  // (y, row j+1 of the column) pairs
    __shared__ double2 red[2][W + 1];               // block sums, and one broadcast value each
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool mute = (int)blockIdx.x == g_gsync_withhold;
    const long long lim = g_gsync_limit;
    // this warp's columns (rows >= its index matter)
    int ci[CPW];
    double2 a[CPW][NR];
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
        ci[c] = 1 + blockIdx.x + gridDim.x * (warp + W * c);
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const int r = lane + 32 * u;
            a[c][u] = ci[c] < n && r < n ? __ldcg(&C[(size_t)ci[c] * n + r]) : make_double2(0.0, 0.0);
        }
    }
    const int ldy = gridDim.x * SL;
    double2 x[EPT], v[EPT];                         // this thread's elements of column j+1 and of v_j
    auto row = [&](int u) { return tid + TH * u; };
#pragma unroll
    for (int u = 0; u < EPT; ++u) x[u] = row(u) < n ? __ldcg(&C[row(u)]) : make_double2(0.0, 0.0);
    // y of column i sits with its CTA's other columns: one writer a line
    int pos[EPT];
#pragma unroll
    for (int u = 0; u < EPT; ++u) {
        const int i = max(row(u) - 1, 0);
        pos[u] = (i % gridDim.x) * SL + i / gridDim.x;
    }
    double2 tj = make_double2(0.0, 0.0);

    // Householder vector of x = column j (rows > j) into v, vc; returns tau
    auto householder = [&](int j) {
        double s2 = 0.0;
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            if (row(u) > j + 1) s2 += x[u].x * x[u].x + x[u].y * x[u].y;
            if (row(u) == j + 1) red[1][W] = x[u];
        }
        for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        if (lane == 0) red[1][warp].x = s2;
        __syncthreads();
        s2 = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) s2 += red[1][w].x;
        const double2 alpha = red[1][W];
        double2 t = make_double2(0.0, 0.0), scal = t;
        double beta = alpha.x;
        if (s2 != 0.0 || alpha.y != 0.0) {
            beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s2), alpha.x);
            const double ib = 1.0 / beta;
            t = make_double2((beta - alpha.x) * ib, -alpha.y * ib);
            const double ar = alpha.x - beta, ai = alpha.y, den = 1.0 / (ar * ar + ai * ai);
            scal = make_double2(ar * den, -ai * den);
        }
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            v[u] = row(u) <= j ? make_double2(0.0, 0.0) : row(u) == j + 1 ? make_double2(1.0, 0.0) : cmul_d(x[u], scal);
            vc[row(u)] = v[u];
        }
        if (blockIdx.x == 0 && tid == 0) {
            e[j] = beta;
            tau[j] = t;
        }
        __syncthreads();
        return t;
    };

    if (blockIdx.x == 0 && tid == 0) d[0] = x[0].x;
    if (n >= 2) tj = householder(0);
    for (int j = 0; j < jend; ++j) {
        const int c1 = j + 1;
        double2 *yb = ybuf + (size_t)j * ldy * 2;
        // ---- the warp's column: rank-2 update with (v_{j-1}, w_{j-1}), then y = column^H v_j
        {
            double2 cw[CPW], cv[CPW], acc[CPW], pick[CPW];
            bool any = false;
#pragma unroll
            for (int c = 0; c < CPW; ++c) {
                const bool on = ci[c] > j && ci[c] < n;
                any |= on;
                cw[c] = cv[c] = acc[c] = pick[c] = make_double2(0.0, 0.0);
                if (on && j > 0) {
                    cw[c] = make_double2(wp[ci[c]].x, -wp[ci[c]].y);
                    cv[c] = make_double2(vp[ci[c]].x, -vp[ci[c]].y);
                }
            }
            if (any) {
#pragma unroll
                for (int u = 0; u < NR; ++u) {
                    const int r = lane + 32 * u;
                    if (32 * u + 31 > j && 32 * u < n) {
                        const double2 pv = vp[r], pw = wp[r], pc = vc[r];
#pragma unroll
                        for (int c = 0; c < CPW; ++c) {
                            if (j > 0) {
                                double2 &t = a[c][u];
                                t.x = fma(-pv.x, cw[c].x, fma(pv.y, cw[c].y, fma(-pw.x, cv[c].x, fma(pw.y, cv[c].y, t.x))));
                                t.y = fma(-pv.x, cw[c].y, fma(-pv.y, cw[c].x, fma(-pw.x, cv[c].y, fma(-pw.y, cv[c].x, t.y))));
                            }
                            if (u == (c1 >> 5)) pick[c] = a[c][u];
                            if (r > j) {
                                acc[c].x = fma(a[c][u].x, pc.x, fma(a[c][u].y, pc.y, acc[c].x));
                                acc[c].y = fma(a[c][u].x, pc.y, fma(-a[c][u].y, pc.x, acc[c].y));
                            }
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < CPW; ++c) {
                    const double h = half_sums(acc[c], lane);
                    if ((lane & 15) == 0) (lane ? ysm[2 * (warp + W * c)].y : ysm[2 * (warp + W * c)].x) = h;
                    if (lane == (c1 & 31)) ysm[2 * (warp + W * c) + 1] = make_double2(pick[c].x, -pick[c].y);
                }
            }
        }
        __syncthreads();
        if (tid < 2 * SL) {
            const int i = 1 + blockIdx.x + gridDim.x * (tid >> 1);
            if (i > j && i < n && !mute) st_relaxed(&yb[2 * blockIdx.x * SL + tid], ysm[tid]);
        }
        // ---- every CTA: y and the raw column j+1, as they arrive
        double2 y[EPT];
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const bool in = row(u) > j && row(u) < n;
            y[u] = in ? ld_relaxed(&yb[2 * pos[u]]) : make_double2(0.0, 0.0);
            x[u] = in ? ld_relaxed(&yb[2 * pos[u] + 1]) : make_double2(0.0, 0.0);
        }
        for (long long it = 0;; ++it) {
            bool wait = false;
#pragma unroll
            for (int u = 0; u < EPT; ++u) {
                if (unset(y[u])) {
                    y[u] = ld_relaxed(&yb[2 * pos[u]]);
                    wait = true;
                }
                if (unset(x[u])) {
                    x[u] = ld_relaxed(&yb[2 * pos[u] + 1]);
                    wait = true;
                }
            }
            if (!wait) break;
            if (it > lim) {
                atomicExch(err, 1);
                break;
            }
            if ((it & 63) == 63 && *(volatile int *)err) break;
        }
        // v_j to its place in C (all of column j has been read: every CTA has published this step)
        if ((j % gridDim.x) == blockIdx.x) {
#pragma unroll
            for (int u = 0; u < EPT; ++u)
                if (row(u) > c1 && row(u) < n) C[(size_t)j * n + row(u)] = v[u];
        }
        // w_j = tau y + alpha v_j, alpha = -tau/2 (tau y)^H v_j
        double2 yv = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            y[u] = cmul_d(tj, y[u]);
            const double2 q = cmulc_d(y[u], v[u]);
            yv.x += q.x;
            yv.y += q.y;
            if (row(u) == c1) red[0][W] = y[u];
        }
        const double h = half_sums(yv, lane);
        if ((lane & 15) == 0) (lane ? red[0][warp].y : red[0][warp].x) = h;
        __syncthreads();   // also: every warp is done with vp, wp of this column's update
        yv = make_double2(0.0, 0.0);
#pragma unroll
        for (int w = 0; w < W; ++w) yv = cadd(yv, red[0][w]);
        const double2 al = cmul_d(make_double2(-0.5 * tj.x, -0.5 * tj.y), yv);
        // column j+1 given the step-j update: x -= v conj(w_{j+1}) + w (v_{j+1} = 1)
        const double2 wc = cadd(red[0][W], al), cw = make_double2(wc.x, -wc.y);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const double2 w = cadd(y[u], cmul_d(al, v[u])), p = cmul_d(v[u], cw);
            vp[row(u)] = v[u];
            wp[row(u)] = w;
            x[u].x -= p.x + w.x;
            x[u].y -= p.y + w.y;
            if (row(u) == c1 && blockIdx.x == 0) d[c1] = x[u].x;
        }
        if (c1 < jend) tj = householder(c1);
    }
    // the trailing matrix from column jend on, with the last step's update, for
    // the next kernel
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CPW; ++c)
        if (jend < n - 1 && ci[c] >= jend && ci[c] < n) {
            const double2 cw = make_double2(wp[ci[c]].x, -wp[ci[c]].y), cv = make_double2(vp[ci[c]].x, -vp[ci[c]].y);
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int r = lane + 32 * u;
                if (r >= jend && r < n) {
                    const double2 p = cmul_d(vp[r], cw), q = cmul_d(wp[r], cv);
                    C[(size_t)ci[c] * n + r] = make_double2(a[c][u].x - (p.x + q.x), a[c][u].y - (p.y + q.y));
                }
            }
        }
}

// The same for n <= 256 (or the last 256 columns of a larger matrix, leading
// dimension ld) inside one thread-block cluster of 16 CTAs: every warp owns
// CPW columns in registers, and the pairs (y_i, entry of row j + 1) go straight
// into every CTA's shared memory (st.async), whose mbarrier counts their bytes: a
// column costs a distributed-shared-memory store instead of a trip through L2
// that other SMs poll.  Two exchange buffers suffice, because a CTA leaves the
// column loop, and is sent to no more, after its own last column (pw_tri.h); the
// owner of column n - 1, which stays to the end, records d, e and tau.  Waits are
// bounded by polls of the mbarrier; when one
// runs out the CTA sets *err and waits no more, and the cluster barrier at the
// end keeps every CTA's shared memory alive until all have finished.  n = 160 /
// 250 take 0.34 / 0.58 ms (k_tridiag_r 0.54 / 0.93, k_tridiag 0.77 / 1.27); with
// 32 columns a CTA, n = 480, the update bounds it: 2.20 ms, k_tridiag_r 1.92.
template <int NR, int W, int CPW> constexpr size_t tridiag_c_smem() {
    constexpr int SL = W * CPW;
    return ((size_t)3 * 32 * NR + 2 * (size_t)TRC * SL * 2 + 2 * SL) * sizeof(double2);
}
template <int NR, int W, int CPW>
__global__ void __launch_bounds__(32 * W, 1)
k_tridiag_c(double2 *C, int n, int ld, double *d, double *e, double2 *tau, int *err) {
    constexpr int TH = 32 * W, NN = 32 * NR, EPT = NN / TH, SL = W * CPW, SR = TRC * 2 * SL / TH;
    static_assert(TRC * SL >= NN, "every column has a warp");
    static_assert(SR * TH == TRC * 2 * SL, "a thread sends the same number of pairs");
    static_assert(EPT * TH == NN, "every row has a thread");
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *vc = reinterpret_cast<double2 *>(sm), *vp = vc + NN, *wp = vp + NN;   // v_j, v_{j-1}, w_{j-1}
    double2 *ex = wp + NN;                       // exchange buffers [2][TRC][SL][2]
    double2 *ysm = ex + 2 * TRC * SL * 2;        // this CTA's pairs [SL][2]
    __shared__ double2 red[2][W + 1];
    __shared__ __align__(8) unsigned long long bar[2];
    __shared__ int failed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const bool mute = (int)rank == g_gsync_withhold;
    const int steps = tri_steps(n, (int)rank);   // this CTA takes part in the steps j < steps
    const bool rec = (int)rank == tri_last_rank(n);
    int to[SR];                                  // steps of the CTAs that this thread's pairs go to
#pragma unroll
    for (int u = 0; u < SR; ++u) to[u] = tri_steps(n, (tid + TH * u) / (2 * SL));
    const long long lim = g_gsync_limit;
    const unsigned bar0 = (unsigned)__cvta_generic_to_shared(&bar[0]), ex0 = (unsigned)__cvta_generic_to_shared(ex);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
    }
    int ci[CPW];
    double2 a[CPW][NR];
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
        ci[c] = 1 + (int)rank + TRC * (warp + W * c);
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const int r = lane + 32 * u;
            a[c][u] = ci[c] < n && r < n ? __ldcg(&C[(size_t)ci[c] * ld + r]) : make_double2(0.0, 0.0);
        }
    }
    auto row = [&](int u) { return tid + TH * u; };
    double2 x[EPT], v[EPT];
    int pos[EPT];
#pragma unroll
    for (int u = 0; u < EPT; ++u) {
        x[u] = row(u) < n ? __ldcg(&C[row(u)]) : make_double2(0.0, 0.0);
        const int i = max(row(u) - 1, 0);
        pos[u] = 2 * ((i % TRC) * SL + i / TRC);
    }
    double2 tj = make_double2(0.0, 0.0);
    // every mbarrier is ready, and everyone has read column 0
    asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");

    auto householder = [&](int j) {
        double s2 = 0.0;
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            if (row(u) > j + 1) s2 += x[u].x * x[u].x + x[u].y * x[u].y;
            if (row(u) == j + 1) red[1][W] = x[u];
        }
        for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        if (lane == 0) red[1][warp].x = s2;
        __syncthreads();
        s2 = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) s2 += red[1][w].x;
        const double2 alpha = red[1][W];
        double2 t = make_double2(0.0, 0.0), scal = t;
        double beta = alpha.x;
        if (s2 != 0.0 || alpha.y != 0.0) {
            beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s2), alpha.x);
            const double ib = 1.0 / beta;
            t = make_double2((beta - alpha.x) * ib, -alpha.y * ib);
            const double ar = alpha.x - beta, ai = alpha.y, den = 1.0 / (ar * ar + ai * ai);
            scal = make_double2(ar * den, -ai * den);
        }
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            v[u] = row(u) <= j ? make_double2(0.0, 0.0) : row(u) == j + 1 ? make_double2(1.0, 0.0) : cmul_d(x[u], scal);
            vc[row(u)] = v[u];
        }
        if (rec && tid == 0) {
            e[j] = beta;
            tau[j] = t;
        }
        __syncthreads();
        return t;
    };

    if (rec && tid == 0) d[0] = x[0].x;
    if (steps > 0) tj = householder(0);
    for (int j = 0; j < steps; ++j) {
        const int c1 = j + 1, b = j & 1;
        // this CTA's mbarrier of the step expects 32 bytes a column i > j
        const bool dead = *(volatile int *)&failed;   // a wait ran out: no more exchange
        if (tid == 0 && !dead)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar0 + 8 * b),
                         "r"(tri_bytes(n, j))
                         : "memory");
        // ---- the warp's columns: rank-2 update with (v_{j-1}, w_{j-1}), then y = column^H v_j
        double2 cw[CPW], cv[CPW], acc[CPW];
        bool any = false;
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
            const bool on = ci[c] > j && ci[c] < n;
            any |= on;
            cw[c] = cv[c] = acc[c] = make_double2(0.0, 0.0);
            if (on && j > 0) {
                cw[c] = make_double2(wp[ci[c]].x, -wp[ci[c]].y);
                cv[c] = make_double2(vp[ci[c]].x, -vp[ci[c]].y);
            }
        }
        if (any) {
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                const int r = lane + 32 * u;
                if (32 * u + 31 > j && 32 * u < n) {
                    const double2 pv = vp[r], pw = wp[r], pc = vc[r];
#pragma unroll
                    for (int c = 0; c < CPW; ++c) {
                        double2 t = a[c][u];
                        if (j > 0) {
                            t.x = fma(-pv.x, cw[c].x, fma(pv.y, cw[c].y, fma(-pw.x, cv[c].x, fma(pw.y, cv[c].y, t.x))));
                            t.y = fma(-pv.x, cw[c].y, fma(-pv.y, cw[c].x, fma(-pw.x, cv[c].y, fma(-pw.y, cv[c].x, t.y))));
                            a[c][u] = t;
                        }
                        if (r == c1) ysm[2 * (warp + W * c) + 1] = make_double2(t.x, -t.y);
                        if (r > j) {
                            acc[c].x = fma(t.x, pc.x, fma(t.y, pc.y, acc[c].x));
                            acc[c].y = fma(t.x, pc.y, fma(-t.y, pc.x, acc[c].y));
                        }
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < CPW; ++c) {
                const double h = half_sums(acc[c], lane);
                if ((lane & 15) == 0) (lane ? ysm[2 * (warp + W * c)].y : ysm[2 * (warp + W * c)].x) = h;
            }
        }
        __syncthreads();
        // ---- the CTA's pairs to every CTA that takes part in the step
#pragma unroll
        for (int u = 0; u < SR; ++u) {
            const int q = tid + TH * u, it = q % (2 * SL), dst = q / (2 * SL), i = 1 + (int)rank + TRC * (it >> 1);
            if (i > j && i < n && j < to[u] && !mute && !dead) {
                const double2 val = ysm[it];
                unsigned ra, rb;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(ra)
                             : "r"(ex0 + 16u * (unsigned)(b * TRC * SL * 2 + (int)rank * 2 * SL + it)), "r"(dst));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bar0 + 8 * b), "r"(dst));
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(ra),
                             "d"(val.x), "d"(val.y), "r"(rb)
                             : "memory");
            }
        }
        // ---- everyone's pairs have arrived
        {
            const unsigned ph = (unsigned)((j >> 1) & 1);
            for (long long it = 0; !*(volatile int *)&failed; ++it) {
                unsigned ok;
                asm volatile(
                    "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                    : "=r"(ok)
                    : "r"(bar0 + 8 * b), "r"(ph)
                    : "memory");
                if (ok) break;
                if (it > lim) {
                    failed = 1;
                    atomicExch(err, 1);
                }
            }
        }
        double2 y[EPT];
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const bool in = row(u) > j && row(u) < n;
            const double2 *p = ex + (size_t)b * TRC * SL * 2 + pos[u];
            y[u] = in ? p[0] : make_double2(0.0, 0.0);
            x[u] = in ? p[1] : make_double2(0.0, 0.0);
        }
        // v_j to its place in C (all of column j has been read: every CTA has published this step)
        if (tri_writer(j) == (int)rank) {
#pragma unroll
            for (int u = 0; u < EPT; ++u)
                if (row(u) > c1 && row(u) < n) C[(size_t)j * ld + row(u)] = v[u];
        }
        // w_j = tau y + alpha v_j, alpha = -tau/2 (tau y)^H v_j
        double2 yv = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            y[u] = cmul_d(tj, y[u]);
            const double2 q = cmulc_d(y[u], v[u]);
            yv.x += q.x;
            yv.y += q.y;
            if (row(u) == c1) red[0][W] = y[u];
        }
        const double h = half_sums(yv, lane);
        if ((lane & 15) == 0) (lane ? red[0][warp].y : red[0][warp].x) = h;
        __syncthreads();   // also: every warp is done with vp, wp of this column's update
        yv = make_double2(0.0, 0.0);
#pragma unroll
        for (int w = 0; w < W; ++w) yv = cadd(yv, red[0][w]);
        const double2 al = cmul_d(make_double2(-0.5 * tj.x, -0.5 * tj.y), yv);
        // column j+1 given the step-j update: x -= v conj(w_{j+1}) + w (v_{j+1} = 1)
        const double2 wc = cadd(red[0][W], al), cw1 = make_double2(wc.x, -wc.y);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const double2 w = cadd(y[u], cmul_d(al, v[u])), p = cmul_d(v[u], cw1);
            vp[row(u)] = v[u];
            wp[row(u)] = w;
            x[u].x -= p.x + w.x;
            x[u].y -= p.y + w.y;
            if (row(u) == c1 && rec) d[c1] = x[u].x;
        }
        if (c1 < steps) tj = householder(c1);
    }
    // no CTA leaves while another may still store into its shared memory
    if (failed) __nanosleep(20000);
    asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
}

// Number of eigenvalues of a tridiagonal matrix below x from the signs of the
// Sturm polynomials p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (a sign change
// per eigenvalue; the quotients p_i / p_{i-1} are the pivots of LDL^T).  One
// dependent multiply-add per row (8 clocks) where the pivot recurrence has a
// division (115); n = 480, 160 values: 536 -> 164 us.  de[i] = (d_i, e_{i-1}^2) of the matrix scaled to norm 1..2,
// with e^2 >= 2^-200 so that no two consecutive p vanish (a change of e by
// 2^-100 of the norm); p grows at most 5-fold and shrinks at most 2^-200 per
// two rows, so rescaling by a power of two every 8 rows stays in range.
__device__ int sturm_count(const double2 *de, int n, double x) {
    double pp = 1.0, p = de[0].x - x;
    int c = (unsigned)__double2hiint(p) >> 31;
    auto row = [&](int i) {
        const double2 q = de[i];
        const double pn = fma(q.x - x, p, -(q.y * pp));
        c += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
        pp = p;
        p = pn;
    };
    int i = 1;
    for (; i + 8 <= n; i += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) row(i + u);
        const int ex = (__double2hiint(fmax(fabs(p), fabs(pp))) >> 20) & 0x7ff;
        const double f = __hiloint2double((2046 - min(max(ex, 1), 2045)) << 20, 0);
        p *= f;
        pp *= f;
    }
    for (; i < n; ++i) row(i);
    return c;
}

// Block reflectors of the back-transformation: H_{j0} ... H_{j0+31} =
// I - V T V^H with T (32 x 32, upper triangular, row-major) from the Gram
// V^H V of the panel's Householder vectors.  128 threads; V in 32-row chunks
// through shared memory (sm: 2 x 32 x 33 complex values).
constexpr int WYB = 32;
__device__ void wy_panel(const double2 *__restrict__ C, const double2 *__restrict__ tau, int n, int j0,
                         double2 *__restrict__ T, double2 *sm) {
    constexpr int LD = WYB + 1;
    double2 *Vs = sm, *S = sm + WYB * LD;
    const int tid = threadIdx.x, nv = min(WYB, n - 1 - j0);
    const int a0 = (tid & 15) * 2, b0 = (tid >> 4) * 4;     // 2 x 4 pairs (a, b) a thread
    double2 acc[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = make_double2(0.0, 0.0);
    for (int r0 = j0 + 1; r0 < n; r0 += WYB) {
        for (int e = tid; e < WYB * WYB; e += 128) {
            const int j = e / WYB, i = r0 + e % WYB;        // vector j0 + j, row i
            double2 v = make_double2(0.0, 0.0);
            if (j < nv && i < n && i > j0 + j) v = i == j0 + j + 1 ? make_double2(1.0, 0.0) : C[(size_t)(j0 + j) * n + i];
            Vs[(e % WYB) * LD + j] = v;
        }
        __syncthreads();
        if (b0 + 3 > a0)
            for (int i = 0; i < WYB; ++i) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        const double2 q = cmulc_d(Vs[i * LD + a0 + u], Vs[i * LD + b0 + v]);
                        acc[u][v].x += q.x;
                        acc[u][v].y += q.y;
                    }
            }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) S[(a0 + u) * LD + b0 + v] = acc[u][v];
    __syncthreads();
    // T[:, i] = -tau_i T[0:i, 0:i] (V^H v_i)[0:i], T_ii = tau_i (Vs holds T), zero
    // past the panel's nv vectors
    for (int i = 0; i < nv; ++i) {
        const double2 ti = tau[j0 + i];
        if (tid < WYB) {
            double2 y = make_double2(0.0, 0.0);
            for (int q = tid; q < i; ++q) {
                const double2 w = cmul_d(Vs[tid * LD + q], S[q * LD + i]);
                y.x += w.x;
                y.y += w.y;
            }
            y = cmul_d(make_double2(-ti.x, -ti.y), y);
            Vs[tid * LD + i] = tid < i ? y : tid == i ? ti : make_double2(0.0, 0.0);
        }
        __syncthreads();
    }
    for (int e = tid; e < WYB * WYB; e += 128)
        T[e] = e % WYB < nv ? Vs[(e / WYB) * LD + e % WYB] : make_double2(0.0, 0.0);
}

// lowest k eigenvalues of the real symmetric tridiagonal (d, e), ascending.
// Multisection: one warp per eigenvalue; each round the 32 lanes take Sturm
// counts at 32 interior points of the current interval [a, b], which then
// shrinks 33-fold to the sub-interval that holds eigenvalue i.  The first nwy
// CTAs form the block reflectors of the back-transformation meanwhile (they
// need the Householder vectors only).  Latency-bound: n dependent
// multiply-adds a round, about 12 rounds.
constexpr int BIS_THREADS = 128;
inline size_t bisect_smem(int n) { return std::max((size_t)n, (size_t)2 * WYB * (WYB + 1)) * sizeof(double2); }
__global__ void __launch_bounds__(BIS_THREADS)
k_bisect(const double *__restrict__ d, const double *__restrict__ e, int n, int k, double *__restrict__ lam,
         double *__restrict__ nrm_out, const double2 *__restrict__ C, const double2 *__restrict__ tau, int nwy,
         double2 *__restrict__ T) {
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *de = reinterpret_cast<double2 *>(sm);
    if ((int)blockIdx.x < nwy) {
        wy_panel(C, tau, n, blockIdx.x * WYB, T + (size_t)blockIdx.x * WYB * WYB, de);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int i = (blockIdx.x - nwy) * (BIS_THREADS >> 5) + (threadIdx.x >> 5);
    double lo = 1e300, hi = -1e300;
    for (int r = lane; r < n; r += 32) {
        const double rad = (r > 0 ? fabs(e[r - 1]) : 0.0) + (r < n - 1 ? fabs(e[r]) : 0.0);
        lo = fmin(lo, d[r] - rad);
        hi = fmax(hi, d[r] + rad);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const double nrm = fmax(fabs(lo), fabs(hi));
    // exact scaling by a power of two to a norm of 1..2 (a zero or non-finite
    // matrix stays as it is)
    const int ex = (__double2hiint(nrm) >> 20) & 0x7ff;
    const bool ok = ex > 0 && ex < 2046;
    const double sc = ok ? __hiloint2double((2046 - ex) << 20, 0) : 1.0, un = ok ? __hiloint2double(ex << 20, 0) : 1.0;
    for (int r = threadIdx.x; r < n; r += BIS_THREADS) {
        const double es = r > 0 ? e[r - 1] * sc : 0.0;
        de[r] = make_double2(d[r] * sc, fmax(es * es, 6.223015277861142e-61));   // 2^-200
    }
    __syncthreads();
    if (i >= k) return;
    const double nrs = nrm * sc;
    double a = lo * sc - 1e-14 * nrs - 1e-300, b = hi * sc + 1e-14 * nrs + 1e-300;
    for (int it = 0; it < 64; ++it) {
        if (b - a <= 2.0 * 2.220446049250313e-16 * fmax(fabs(a), fabs(b))) break;
        const double h = (b - a) / 33.0;
        const double x = fmin(fmax(a + (lane + 1) * h, a), b);
        const bool above = sturm_count(de, n, x) > i;             // eigenvalue i lies below x
        const unsigned m = __ballot_sync(0xffffffffu, above);
        const int f = m ? __ffs(m) - 1 : 32;                       // first sample point above it (warp-uniform)
        const double xl = __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
        const double xr = __shfl_sync(0xffffffffu, x, f < 32 ? f : 31);
        const double na = f > 0 ? xl : a, nb = f < 32 ? xr : b;
        if (na == a && nb == b) break;  // no representable progress
        a = na;
        b = nb;
    }
    if (lane == 0) {
        lam[i] = 0.5 * (a + b) * un;
        if (i == 0) *nrm_out = nrm;
    }
}

// LU factorisation with partial pivoting of (Tr - lam I) (LAPACK dgttrf
// pattern): rows i and i+1 swap when |sub| > |pivot|.  Per row, what the
// solve below multiplies by: rd = 1 / U[i][i], du = U[i][i+1] rd, du2 =
// U[i][i+2] rd, lm = multiplier, pv = 1 where rows i, i+1 were swapped.  A
// pivot below `tiny` is replaced by it (the shift sits on an eigenvalue to working
// precision; 1e-30 of the norm, so that the solution's norm stays finite).
// One lane runs it; rows go through registers 8 at a time so that
// only the recurrence itself is serial.
constexpr int TRB = 8;
__device__ void tri_factor(const double *__restrict__ d, const double *__restrict__ e, int n, double lam, double tiny,
                           double *__restrict__ rd, double *__restrict__ du, double *__restrict__ du2,
                           double *__restrict__ lm, unsigned char *__restrict__ pv) {
    double di = d[0] - lam, ui = n > 1 ? e[0] : 0.0;
    for (int i0 = 0; i0 < n - 1; i0 += TRB) {
        double dd[TRB], ee[TRB + 1];
#pragma unroll
        for (int u = 0; u < TRB; ++u) {
            dd[u] = i0 + u + 1 < n ? d[i0 + u + 1] - lam : 0.0;
            ee[u] = i0 + u < n - 1 ? e[i0 + u] : 0.0;
        }
        ee[TRB] = i0 + TRB < n - 1 ? e[i0 + TRB] : 0.0;
#pragma unroll
        for (int u = 0; u < TRB; ++u) {
            const int i = i0 + u;
            if (i < n - 1) {
                const double sub = ee[u], dn = dd[u], un = ee[u + 1];
                const bool keep = fabs(di) >= fabs(sub);
                if (keep && fabs(di) < tiny) di = copysign(tiny, di);
                const double r = 1.0 / (keep ? di : sub);
                const double f = (keep ? sub : di) * r;
                rd[i] = r;
                du[i] = (keep ? ui : dn) * r;
                du2[i] = keep ? 0.0 : un * r;
                lm[i] = f;
                pv[i] = keep ? 0 : 1;
                di = keep ? fma(-f, ui, dn) : fma(-f, dn, ui);
                ui = keep ? un : -f * un;
            }
        }
    }
    if (fabs(di) < tiny) di = copysign(tiny, di);
    rd[n - 1] = 1.0 / di;
    du[n - 1] = 0.0;
    du2[n - 1] = 0.0;
}

// b := (Tr - lam I)^-1 b with the factorisation of tri_factor.
__device__ void tri_solve(int n, const double *__restrict__ rd, const double *__restrict__ du,
                          const double *__restrict__ du2, const double *__restrict__ lm,
                          const unsigned char *__restrict__ pv, double *b) {
    double bi = b[0];
    for (int i0 = 0; i0 < n - 1; i0 += TRB) {
        double bn[TRB], l[TRB], o[TRB];
        bool sw[TRB];
#pragma unroll
        for (int u = 0; u < TRB; ++u) {
            const int i = min(i0 + u, n - 2);
            bn[u] = b[i + 1];
            l[u] = lm[i];
            sw[u] = pv[i] != 0;
        }
#pragma unroll
        for (int u = 0; u < TRB; ++u)
            if (i0 + u < n - 1) {
                o[u] = sw[u] ? bn[u] : bi;
                bi = sw[u] ? fma(-l[u], bn[u], bi) : fma(-l[u], bi, bn[u]);
            }
#pragma unroll
        for (int u = 0; u < TRB; ++u)
            if (i0 + u < n - 1) b[i0 + u] = o[u];
    }
    double x2 = 0.0, x1 = bi * rd[n - 1];
    b[n - 1] = x1;
    for (int i0 = n - 2; i0 >= 0; i0 -= TRB) {
        double c[TRB], p[TRB], q[TRB];
#pragma unroll
        for (int u = 0; u < TRB; ++u) {
            const int i = max(i0 - u, 0);
            c[u] = b[i] * rd[i];
            p[u] = du[i];
            q[u] = du2[i];
        }
#pragma unroll
        for (int u = 0; u < TRB; ++u)
            if (i0 - u >= 0) {
                const double x = fma(-p[u], x1, fma(-q[u], x2, c[u]));
                x2 = x1;
                x1 = x;
                c[u] = x;
            }
#pragma unroll
        for (int u = 0; u < TRB; ++u)
            if (i0 - u >= 0) b[i0 - u] = c[u];
    }
}

// One warp per cluster of near-degenerate eigenvalues (gap <= ortol):
// inverse iteration for each member (one factorisation, INVIT_STEPS solves),
// re-orthogonalised against the earlier members of its cluster.  The
// factorisation and the iterate live in shared memory (lane 0 runs the
// sequential recurrences).  Z: n x k real (column-major).
constexpr int INVIT_STEPS = 3;
__global__ void k_invit(const double *__restrict__ d, const double *__restrict__ e, int n, int k,
                        const double *__restrict__ lam, const double *__restrict__ nrmp, double reltol,
                        double *__restrict__ Z) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int wid = blockIdx.x * (blockDim.x >> 5) + wl;
    double *rd = reinterpret_cast<double *>(sm) + (size_t)wl * 5 * n;
    double *du = rd + n, *du2 = du + n, *lm = du2 + n, *x = lm + n;
    unsigned char *pv = sm + (size_t)(blockDim.x >> 5) * 5 * n * sizeof(double) + (size_t)wl * n;
    if (wid >= k) return;
    const double nrm = *nrmp;
    const double ortol = reltol * nrm;
    const double eps = 2.220446049250313e-16;
    // a warp owns eigenvalue wid only if it starts a cluster
    if (wid > 0 && lam[wid] - lam[wid - 1] <= ortol) return;
    int end = wid + 1;
    while (end < k && lam[end] - lam[end - 1] <= ortol) ++end;
    double lprev = 0.0;
    for (int i = wid; i < end; ++i) {
        double li = lam[i];
        if (i > wid && li - lprev < 10.0 * eps * nrm) li = lprev + 10.0 * eps * nrm;  // separate degenerate shifts
        lprev = li;
        // deterministic pseudo-random start
        for (int r = lane; r < n; r += 32) {
            unsigned int h = (unsigned int)(r * 2654435761u) ^ (unsigned int)(i * 2246822519u + 12345u);
            h ^= h >> 15;
            h *= 2246822519u;
            h ^= h >> 13;
            x[r] = ((double)(h & 0xFFFFFF) / 16777216.0) - 0.5;
        }
        if (lane == 0) tri_factor(d, e, n, li, nrm > 0.0 ? 1e-30 * nrm : 1e-30, rd, du, du2, lm, pv);
        __syncwarp();
        for (int it = 0; it < INVIT_STEPS; ++it) {
            if (lane == 0) tri_solve(n, rd, du, du2, lm, pv, x);
            __syncwarp();
            for (int jj = wid; jj < i; ++jj) {  // modified Gram-Schmidt inside the cluster
                const double *q = Z + (size_t)jj * n;
                double s = 0.0;
                for (int r = lane; r < n; r += 32) s += q[r] * x[r];
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                for (int r = lane; r < n; r += 32) x[r] -= s * q[r];
                __syncwarp();
            }
            double s = 0.0;
            for (int r = lane; r < n; r += 32) s += x[r] * x[r];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const double inv = 1.0 / sqrt(fmax(s, 1e-300));
            for (int r = lane; r < n; r += 32) x[r] *= inv;
            __syncwarp();
        }
        double *z = Z + (size_t)i * n;
        for (int r = lane; r < n; r += 32) z[r] = x[r];
        __syncwarp();
    }
}

// shared memory of k_invit per warp
inline size_t invit_smem_per_warp(int n) { return (size_t)n * (5 * sizeof(double) + 1); }

// Z[:, c] = Q Ztr[:, c], Q = H_0 H_1 ... H_{n-2}: 32 reflectors at a time,
// z -= V T (V^H z), in reverse order; NV eigenvectors a CTA, held in shared
// memory.  Per panel: the 32 dot products (4 vectors a warp), t = T s, the
// update (rows over threads), one block barrier each, where one reflector at a
// time took three (n = 480, 160 vectors: 655 -> 199 us).  Bound by reading V
// (n^2 / 2 values twice a CTA, the second time mostly from L1), so NV grows
// with k.
template <int NV>
__global__ void __launch_bounds__(256)
k_backtr(const double2 *__restrict__ C, const double2 *__restrict__ T, int n, int k, const double *__restrict__ Zt,
         double2 *__restrict__ Z) {
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *z = reinterpret_cast<double2 *>(sm);           // [NV][n]
    double2 *s = z + (size_t)NV * n, *t = s + NV * WYB;     // [NV][32] each
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = blockIdx.x * NV;
#pragma unroll
    for (int q = 0; q < NV; ++q)
        for (int i = threadIdx.x; i < n; i += 256)
            z[q * n + i] = make_double2(c0 + q < k ? Zt[(size_t)(c0 + q) * n + i] : 0.0, 0.0);
    __syncthreads();
    for (int p = (n - 2) / WYB; p >= 0; --p) {
        const int j0 = p * WYB, nv = min(WYB, n - 1 - j0);
        double2 acc[4][NV];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < NV; ++q) acc[u][q] = make_double2(0.0, 0.0);
        const int jw = j0 + warp * 4;                       // this warp's vectors jw .. jw + 3
        if (warp * 4 < nv) {
#pragma unroll 2
            for (int i = jw + 1 + lane; i < n; i += 32) {
                double2 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = jw + u;
                    v[u] = (j < j0 + nv && i > j + 1) ? C[(size_t)j * n + i]
                                                      : make_double2(j < j0 + nv && i == j + 1 ? 1.0 : 0.0, 0.0);
                }
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    const double2 x = z[q * n + i];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const double2 w = cmulc_d(v[u], x);
                        acc[u][q].x += w.x;
                        acc[u][q].y += w.y;
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                double2 a = acc[u][q];
                for (int o = 16; o > 0; o >>= 1) {
                    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
                    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
                }
                if (lane == 0) s[q * WYB + warp * 4 + u] = a;
            }
        // t = T s, 8 lanes a row (the loads of T do not wait for s)
        const int r = threadIdx.x >> 3, l8 = threadIdx.x & 7;
        double2 tr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) tr[u] = T[(size_t)p * WYB * WYB + r * WYB + l8 + 8 * u];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double2 a = make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 w = cmul_d(tr[u], s[q * WYB + l8 + 8 * u]);
                a.x += w.x;
                a.y += w.y;
            }
            for (int o = 4; o > 0; o >>= 1) {
                a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
                a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
            }
            if (l8 == 0) t[q * WYB + r] = a;
        }
        __syncthreads();
        // rows i of z; T's zero rows make t vanish beyond nv
        for (int i = j0 + 1 + threadIdx.x; i < n; i += 256) {
            double2 x[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) x[q] = z[q * n + i];
#pragma unroll 8
            for (int j = 0; j < nv; ++j) {
                const double2 v = i > j0 + j + 1 ? C[(size_t)(j0 + j) * n + i]
                                                 : make_double2(i == j0 + j + 1 ? 1.0 : 0.0, 0.0);
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    const double2 w = cmul_d(v, t[q * WYB + j]);
                    x[q].x -= w.x;
                    x[q].y -= w.y;
                }
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) z[q * n + i] = x[q];
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < NV; ++q)
        if (c0 + q < k)
            for (int i = threadIdx.x; i < n; i += 256) Z[(size_t)(c0 + q) * n + i] = z[q * n + i];
}

template <int NV>
cudaError_t launch_backtr(const double2 *C, const double2 *T, int n, int k, const double *Zt, double2 *Z, cudaStream_t st) {
    const size_t smem = (size_t)NV * (n + 2 * WYB) * sizeof(double2);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute((const void *)k_backtr<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k_backtr<NV><<<(k + NV - 1) / NV, 256, smem, st>>>(C, T, n, k, Zt, Z);
    return cudaGetLastError();
}

int blocks_for(size_t total) {
    size_t b = (total + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    return b < 1 ? 1 : (int)b;
}

// CTAs of fn that are resident at once on the current device; one_per_sm: at
// most that many
cudaError_t resident_ctas(const void *fn, int threads, size_t smem, int *n, bool one_per_sm = false) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if (smem > 48 * 1024 && (e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
        return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem)) != cudaSuccess) return e;
    *n = sms * (one_per_sm ? std::min(per, 1) : per);
    return cudaSuccess;
}

// The last (or only) 256 columns of the tridiagonalisation, what one cluster holds in
// registers, go to it, those before them to the grid: in registers up to n = 1024,
// through L2 above that.  At 2.3 against 4.0 us a column the whole reduced problem goes
// from 2.94 to 2.65 ms at n = 480, from 1.14 to 0.75 at 160 (k = n / 3); with 384
// columns in a cluster of 384 threads a CTA it spills, 2.73 at 480.
const auto tri_c = k_tridiag_c<8, 8, 2>;
static_assert(32 * 8 == TRI_NC, "the cluster's columns");
struct TriKernels {
    TriRoute route;
    const void *fn_r;           // the register kernel for n, and its shared memory
    size_t smem_r;
    cudaLaunchConfig_t cf;      // the cluster's launch
    cudaLaunchAttribute at;
};
cudaError_t tri_kernels(int n, cudaStream_t st, TriKernels *k) {
    cudaError_t e;
    constexpr size_t smem_c = tridiag_c_smem<8, 8, 2>();
    static_assert(smem_c <= 48 << 10, "no opt-in");
    k->cf = {};
    k->cf.gridDim = TRC;
    k->cf.blockDim = 256;
    k->cf.dynamicSmemBytes = smem_c;
    k->cf.stream = st;
    k->at.id = cudaLaunchAttributeClusterDimension;
    k->at.val.clusterDim.x = TRC;
    k->at.val.clusterDim.y = k->at.val.clusterDim.z = 1;
    k->cf.attrs = &k->at;
    k->cf.numAttrs = 1;
    if ((e = cudaFuncSetAttribute(tri_c, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    // no room for 16 neighbouring SMs (a partitioned device): the grid does all
    int ncl = 0;
    if (cudaOccupancyMaxActiveClusters(&ncl, tri_c, &k->cf) != cudaSuccess) {
        cudaGetLastError();
        ncl = 0;
    }
    // few CTAs keep the exchange short, few columns a CTA the update (n =
    // 480, us a column: 120 CTAs of 4 columns 4.1, 60 of 8 4.5, 30 of 16 5.4)
    k->fn_r = n <= 512 ? (const void *)k_tridiag_r<16, 4, 1> : (const void *)k_tridiag_r<32, 8, 1>;
    k->smem_r = 3 * (size_t)(n <= 512 ? 512 : 1024) * sizeof(double2);
    int res = 0;
    if (n <= 1024 && (n > TRI_NC || ncl < 1)) {
        // (48 KB and the static arrays need the opt-in, or none would be resident)
        if ((e = cudaFuncSetAttribute(k->fn_r, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k->smem_r)) != cudaSuccess) return e;
        if ((e = resident_ctas(k->fn_r, 32 * tri_r_warps(n), k->smem_r, &res)) != cudaSuccess) return e;
    }
    k->route = tri_route(n, res, ncl);
    return cudaSuccess;
}

cudaError_t coop_blocks(const void *fn, size_t smem, int *nblk) {
    const cudaError_t e = resident_ctas(fn, COOP_THREADS, smem, nblk, true);   // one CTA per SM keeps the barrier cheap
    return e != cudaSuccess ? e : *nblk < 1 ? cudaErrorCooperativeLaunchTooLarge : cudaSuccess;
}

}  // namespace eig

using namespace eig;

size_t eig_work_bytes(int n, int k) {
    const size_t nn = (size_t)n * n * sizeof(double2);
    return 2 * nn + (size_t)32 * n * sizeof(double2)  // L^-1, scratch n x n (or the tridiagonalisation's exchange)
           + (size_t)2 * n * sizeof(double2)          // y (two buffers)
           + (size_t)(3 * n) * sizeof(double)         // d, e, lam
           + (size_t)n * sizeof(double2)              // tau
           + (size_t)n * k * sizeof(double)           // Ztr
           + (size_t)n * k * sizeof(double2)          // Z
           + (size_t)((n + WYB - 1) / WYB) * WYB * WYB * sizeof(double2)   // block reflectors
           + 16 * 256;                                // barrier, status, norm + 256-byte rounding of 13 pieces
}

// Linv = L^-1 with G = L L^H (G's lower triangle is overwritten).  ctr:
// barrier counter, err: [0] barrier expiry, [1] first failing Cholesky column
// (1-based).
cudaError_t chol_and_inverse(double2 *G, int n, double2 *Linv, unsigned *ctr, int *err, cudaStream_t st) {
    cudaError_t e_;
    const int nt = (n + TB - 1) / TB;
    int nblk = 0;
    if ((e_ = coop_blocks((const void *)k_chol_inv, CHOL_SMEM, &nblk)) != cudaSuccess) return e_;
    nblk = std::max(1, std::min(nblk, nt * (nt + 1) / 2));
    if ((e_ = cudaMemsetAsync(ctr, 0, sizeof(unsigned), st)) != cudaSuccess) return e_;
    int *info = err + 1;
    void *args[] = {(void *)&G, (void *)&Linv, (void *)&n, (void *)&ctr, (void *)&err, (void *)&info};
    return cudaLaunchCooperativeKernel((const void *)k_chol_inv, nblk, COOP_THREADS, args, CHOL_SMEM, st);
}

// flag[0] = 1 if any diagonal or off-diagonal entry of the tridiagonal
// matrix is not finite
__global__ void k_check_finite(const double *__restrict__ d, const double *__restrict__ e, int n, int *flag) {
    bool bad = false;
    for (int i = threadIdx.x; i < n; i += blockDim.x) bad |= !isfinite(d[i]) || (i + 1 < n && !isfinite(e[i]));
    if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 1;
}

cudaError_t hegv_lowest(double2 *T, double2 *G, int n, int k, double *lam_out, double2 *S, void *work, size_t work_bytes,
                        int *launches, int *d_status, cudaStream_t st) {
    if (n <= 0 || k <= 0 || k > n || work_bytes < eig_work_bytes(n, k)) return cudaErrorInvalidValue;
    unsigned char *p = (unsigned char *)work;
    auto take = [&](size_t bytes) {
        unsigned char *q = p;
        p += (bytes + 255) & ~(size_t)255;
        return (void *)q;
    };
    const size_t nn = (size_t)n * n;
    // L^-1 and a scratch matrix, and after them the exchange buffer of the
    // register tridiagonalisation (n rows of pairs for at most n + 16 columns)
    double2 *ybuf = (double2 *)take((2 * nn + 32 * (size_t)n) * sizeof(double2));
    double2 *Linv = ybuf, *M1 = ybuf + nn;
    double2 *xg = (double2 *)take(2 * (size_t)n * sizeof(double2));
    double *d = (double *)take(n * sizeof(double));
    double *e = (double *)take(n * sizeof(double));
    double *lam = (double *)take(n * sizeof(double));
    double2 *tau = (double2 *)take(n * sizeof(double2));
    double *Zt = (double *)take((size_t)n * k * sizeof(double));
    double2 *Z = (double2 *)take((size_t)n * k * sizeof(double2));
    double2 *Tw = (double2 *)take((size_t)((n + WYB - 1) / WYB) * WYB * WYB * sizeof(double2));   // block reflectors' T
    GridBar *gb = (GridBar *)take(sizeof(GridBar));
    int *err = (int *)take(sizeof(int) * 4);
    double *nrm = (double *)take(sizeof(double));
    unsigned *ctr = &gb->count;
    cudaError_t e_;
    if ((e_ = cudaMemsetAsync(gb, 0, sizeof(GridBar), st)) != cudaSuccess) return e_;
    if ((e_ = cudaMemsetAsync(err, 0, sizeof(int) * 4, st)) != cudaSuccess) return e_;
    const int nb = blocks_for(nn);
    int nl = 1;   // kernels launched
    k_herm_upper<<<nb, 256, 0, st>>>(T, n);
    double2 *Cm = T;
    if (G) {
        nl += 6;
        k_herm_upper<<<nb, 256, 0, st>>>(G, n);
        if ((e_ = chol_and_inverse(G, n, Linv, ctr, err, st)) != cudaSuccess) return e_;
        // C = Linv T Linv^H: Linv lower triangular, only C's upper triangle
        // is read (n = 1440: the two full products took 3.06 ms)
        if ((e_ = gemm_nn<double>(n, n, n, Linv, n, T, n, M1, n, 0, st, 1)) != cudaSuccess) return e_;
        k_conj_transpose<<<nb, 256, 0, st>>>(Linv, G, n);  // G no longer needed: holds Linv^H
        if ((e_ = gemm_nn<double>(n, n, n, M1, n, G, n, T, n, 0, st, 2)) != cudaSuccess) return e_;
        k_herm_upper<<<nb, 256, 0, st>>>(T, n);
    }
    TriKernels tk;
    if ((e_ = tri_kernels(n, st, &tk)) != cudaSuccess) return e_;
    const TriRoute route = tk.route;
    const void *fn = tk.fn_r;
    const size_t smem_r = tk.smem_r;
    const int W = tri_r_warps(n), ctas_r = tri_r_ctas(n), jend = route.jend;
    if ((jend > 0 || !route.cluster) && route.registers) {
        if ((e_ = cudaMemsetAsync(ybuf, 0xff, (size_t)jend * 2 * ctas_r * W * sizeof(double2), st)) != cudaSuccess) return e_;
        void *args[] = {(void *)&Cm, (void *)&n, (void *)&jend, (void *)&d, (void *)&e, (void *)&tau, (void *)&ybuf, (void *)&err};
        if ((e_ = cudaLaunchCooperativeKernel(fn, ctas_r, 32 * W, args, smem_r, st)) != cudaSuccess) return e_;
        nl += 1;
    } else if (jend > 0) {
        const size_t smem = (size_t)(3 * n + 32) * sizeof(double2);
        int nblk = 0;
        if ((e_ = coop_blocks((const void *)k_tridiag, smem, &nblk)) != cudaSuccess) return e_;
        // about one trailing column per warp at the start: fewer CTAs keep
        // the per-column barrier cheap for small n
        nblk = std::max(1, std::min(nblk, (n + 7) / 8));
        if ((e_ = cudaMemsetAsync(ctr, 0, sizeof(unsigned), st)) != cudaSuccess) return e_;
        void *args[] = {(void *)&Cm, (void *)&n, (void *)&jend, (void *)&d, (void *)&e, (void *)&tau, (void *)&xg, (void *)&ctr, (void *)&err};
        if ((e_ = cudaLaunchCooperativeKernel((const void *)k_tridiag, nblk, COOP_THREADS, args, smem, st)) != cudaSuccess)
            return e_;
        nl += 1;
    }
    if (route.cluster) {
        if ((e_ = cudaLaunchKernelEx(&tk.cf, tri_c, Cm + (size_t)jend * (n + 1), n - jend, n, d + jend, e + jend, tau + jend, err)) !=
            cudaSuccess)
            return e_;
        nl += 1;
    }
    // a non-finite T or G reaches the tridiagonal matrix: report it (the
    // Sturm counts would otherwise turn it into finite, meaningless values)
    k_check_finite<<<1, 256, 0, st>>>(d, e, n, err + 2);
    {
        const size_t smem = bisect_smem(n);
        const int nwy = S ? (n - 1 + WYB - 1) / WYB : 0, per = BIS_THREADS / 32;
        if (smem > 48 * 1024 &&
            (e_ = cudaFuncSetAttribute((const void *)k_bisect, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
            return e_;
        k_bisect<<<nwy + (k + per - 1) / per, BIS_THREADS, smem, st>>>(d, e, n, k, lam, nrm, Cm, tau, nwy, Tw);
        nl += 2;
    }
    if ((e_ = cudaMemcpyAsync(lam_out, lam, k * sizeof(double), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e_;
    if (S) {
        {
            // as many warps per CTA as fit in about 200 KB of shared memory
            const size_t per = invit_smem_per_warp(n);
            const int wpc = (int)std::max<size_t>(1, std::min<size_t>(8, (200u << 10) / per));
            const size_t smem = ((per * wpc) + 15) & ~(size_t)15;
            if (smem > 48 * 1024 &&
                (e_ = cudaFuncSetAttribute((const void *)k_invit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
                    cudaSuccess)
                return e_;
            k_invit<<<(k + wpc - 1) / wpc, 32 * wpc, smem, st>>>(d, e, n, k, lam, nrm, 1e-7, Zt);
        }
        // one eigenvector a CTA until there are enough for every SM several times
        double2 *Zo = G ? Z : S;
        if (k >= 4 * 148 && n <= 2048)
            e_ = launch_backtr<4>(Cm, Tw, n, k, Zt, Zo, st);
        else if (k >= 2 * 148 && n <= 4096)
            e_ = launch_backtr<2>(Cm, Tw, n, k, Zt, Zo, st);
        else
            e_ = launch_backtr<1>(Cm, Tw, n, k, Zt, Zo, st);
        if (e_ != cudaSuccess) return e_;
        if (G) {
            // S = Linv^H Z  (Linv^H sits in G)
            if ((e_ = gemm_nn<double>(n, k, n, G, n, Z, n, S, n, 0, st, 3)) != cudaSuccess) return e_;
        }
        nl += G ? 3 : 2;
    }
    *launches = nl;
    if ((e_ = cudaGetLastError()) != cudaSuccess) return e_;
    // status: [0] barrier expiry, [1] Cholesky breakdown column (1-based),
    // [2] non-finite tridiagonal matrix
    return cudaMemcpyAsync(d_status, err, 3 * sizeof(int), cudaMemcpyDeviceToDevice, st);
}

cudaError_t chol_inverse_upper(double2 *C, int n, double2 *Rinv, void *work, int *d_status, cudaStream_t st) {
    unsigned char *p = (unsigned char *)work;
    double2 *Linv = (double2 *)p;
    p += (((size_t)n * n * sizeof(double2)) + 255) & ~(size_t)255;
    unsigned *ctr = (unsigned *)p;
    p += 256;
    int *err = (int *)p;
    cudaError_t e_;
    if ((e_ = cudaMemsetAsync(err, 0, sizeof(int) * 4, st)) != cudaSuccess) return e_;
    const int nb = blocks_for((size_t)n * n);
    k_herm_upper<<<nb, 256, 0, st>>>(C, n);
    if ((e_ = chol_and_inverse(C, n, Linv, ctr, err, st)) != cudaSuccess) return e_;
    k_conj_transpose<<<nb, 256, 0, st>>>(Linv, Rinv, n);
    if ((e_ = cudaGetLastError()) != cudaSuccess) return e_;
    return cudaMemcpyAsync(d_status, err, 2 * sizeof(int), cudaMemcpyDeviceToDevice, st);
}

}  // namespace pwk

// Test-only export (not in pwb200.h): the kernels that an order-n problem takes on
// `device`: 1 the register kernel, 2 the cluster, 3 both, 0 the grid-barrier kernel
// alone, negative on an error.
extern "C" int pwk_test_tri_route(int device, int n) {
    pwk::eig::TriKernels k;
    if (cudaSetDevice(device) != cudaSuccess || pwk::eig::tri_kernels(n, nullptr, &k) != cudaSuccess) return -1;
    return (k.route.registers && (k.route.jend > 0 || !k.route.cluster) ? 1 : 0) + (k.route.cluster ? 2 : 0);
}

// Test-only export (not in pwb200.h): sets the grid-barrier poll limit
// (limit <= 0 restores the default) and the CTA that withholds its arrivals
// (-1: none) on `device`, for the tests that make a bounded wait expire
// without faulting or hanging the GPU.
extern "C" int pwk_test_gsync(int device, long long limit, int withhold_cta) {
    if (cudaSetDevice(device) != cudaSuccess) return 2;
    const long long lim = limit > 0 ? limit : pwk::eig::GSYNC_LIMIT;
    if (cudaMemcpyToSymbol(pwk::eig::g_gsync_limit, &lim, sizeof(lim)) != cudaSuccess) return 2;
    if (cudaMemcpyToSymbol(pwk::eig::g_gsync_withhold, &withhold_cta, sizeof(withhold_cta)) != cudaSuccess) return 2;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}
