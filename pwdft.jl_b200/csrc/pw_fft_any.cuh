// Plane passes of the pruned FFT for grids whose x and y lengths are any two of
// the fused plans' (pw_fft_fused.cuh): the x-fused kernels of the 27-, 75- and
// 120-point cubes with the two directions chosen independently at run time.
// A kernel calls the y pass and the x pass of its lengths (one switch each,
// uniform over the launch), so the code grows with the number of lengths and not with
// its square.  The run-time-plan kernels that these sizes ran on before spend
// most of their time on index arithmetic (radix stages of run-time length,
// integer divisions), table reads for every twiddle and separate zero-fill,
// scatter, V and gather passes over the plane; they remain for lengths without
// a fused plan.  Measured: op_H of 8 atoms (40-point cube, 20 bands, FP32) 129 ->
// 92 us, of 32 atoms (75 x 75 x 40, 81 bands, FP64) 546 -> 490 us (z passes),
// density and op_H on 36- to 108-point boxes 2.0 to 3.2 times faster.
#pragma once
#include <algorithm>

#include "pw_fft_fused.cuh"
#include "pw_launch.h"

namespace pwk {
namespace any {

#define PW_ANY_SIZES(X)                                                                                              \
    X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48) X(50) X(54) X(60) X(64) X(72) X(75) X(80) X(81) X(90) \
    X(96) X(100) X(108) X(120) X(125) X(128)

constexpr int THREADS = 256, NW = THREADS / 32;
// Twiddles: all N entries of a direction, in both precisions (powers formed in
// registers cost accuracy, see pwf::FullTw).
constexpr int TWN = 128;
template <typename T> using Tw = pwf::FullTw<T>;
// entry i = r R0 + j of the table, 1 <= r < R1, j < R0: exp(-2 pi i r j / N)
__host__ __device__ __forceinline__ int tw_entry(int i, int R0) { return i / R0 * (i % R0); }

// What the host chooses for a launch.
struct Shape {
    int bpc;      // bands of one z-plane per CTA
    int LD;       // row stride of the sub-plane S[active x][y]
    int padm;     // y -> y + (y * padm >> 16): the y plan's padding (0: none)
    int R0x, R0y; // first radices (twiddle table lengths)
    int xw;       // elements of a warp's x-line buffer
    int vst;      // row stride of V(r) or the density plane in shared memory (0: not kept there)
};
__device__ __forceinline__ int ypos(const Shape &h, int y) { return y + ((y * h.padm) >> 16); }


// shared memory: twiddles of x and y, nsub sub-planes, the warps' x lines, the
// V(r) or density plane, the active-x map
template <typename T> struct Sm {
    Cx<T> *tx, *ty, *S, *Xw;
    T *P;
    short *iax;
    __device__ __forceinline__ Sm(const Shape &h, int nsub, int Nxa, int N2) {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        tx = reinterpret_cast<Cx<T> *>(smem_raw);
        ty = tx + TWN;
        S = ty + TWN;
        Cx<T> *x = S + (size_t)nsub * Nxa * h.LD;
        Xw = x + (threadIdx.x >> 5) * h.xw;
        P = reinterpret_cast<T *>(x + NW * h.xw);
        iax = reinterpret_cast<short *>(P + (size_t)N2 * h.vst);
    }
};

// The passes are functions of their own (a length's registers are allocated for
// it alone) and take the shared arrays from the launch's shape, so that their
// accesses stay shared-memory ones.
template <typename T, int N2> __device__ __noinline__ void y_pass(Shape h, int nsub, int Nxa, int nl, int sign) {
    const Sm<T> m(h, nsub, Nxa, N2);
    pwf::lines<T, N2, true, (pwf::fp_pad<N2>() > 0)>(m.S, nl, 1, h.LD, Tw<T>{m.ty}, sign);   // ends with __syncthreads
}

// Active-x rows of the elements a lane reads in the first inverse x stage (and
// writes in the last forward one), one byte each (255: not active); one-stage
// plans look iax up directly.
template <int N1> struct XRows {
    static constexpr bool TWO = pwf::FPlan<N1>::nst == 2;
    static constexpr int G = pwf::fp_group<N1>();
    static constexpr int R0 = pwf::FPlan<N1>::r(0), R1 = TWO ? pwf::FPlan<N1>::r(1) : 1;
    static constexpr int NPK = TWO ? (R0 + 3) / 4 : 1;
    unsigned pk[NPK];
    int line;
    __device__ __forceinline__ XRows(const short *iax, int lane) {
        line = lane;
        if constexpr (TWO) {
            static_assert(R1 <= 16 && pwf::LaneMap<R1, G>::ROUNDS == 1, "one x butterfly slot per lane");
            int jl;
            pwf::LaneMap<R1, G>::at(lane, 0, G, line, jl);
#pragma unroll
            for (int w = 0; w < NPK; ++w) {
                unsigned u = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int r = 4 * w + b;
                    const int ia = r < R0 && jl < R1 ? iax[jl + R1 * r] : -1;
                    u |= (unsigned)(ia >= 0 ? ia : 255) << (8 * b);
                }
                pk[w] = u;
            }
        }
    }
    __device__ __forceinline__ int at(const short *iax, int x, int r) const {
        if constexpr (TWO) {
            const int v = (pk[r >> 2] >> (8 * (r & 3))) & 255;
            return v == 255 ? -1 : v;
        } else {
            return iax[x];
        }
    }
};

template <typename T, int N1, bool VS>
__device__ __noinline__ void x_vloc(Shape h, int Nxa, int N2, int nbh, const T *__restrict__ Vp) {
    constexpr int G = pwf::fp_group<N1>();
    const Sm<T> m(h, h.bpc, Nxa, N2);
    const T *Vs = m.P;
    const short *iax = m.iax;
    const int SP = Nxa * h.LD;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const XRows<N1> rows(iax, lane);
    const int ngrp = (N2 + G - 1) / G, LD = h.LD;
    for (int q = warp; q < nbh * ngrp; q += NW) {
        const int bb = q / ngrp, g0 = (q - bb * ngrp) * G, nl = min(G, N2 - g0);
        Cx<T> *Sb = m.S + bb * SP + ypos(h, g0 + rows.line);
        auto ld_s = [&](int, int x, int r) {
            const int ia = rows.at(iax, x, r);
            return ia >= 0 ? Sb[ia * LD] : cmake((T)0, (T)0);
        };
        auto vsc = [&](int line, int x) { return VS ? Vs[(g0 + line) * h.vst + x] : __ldg(&Vp[(g0 + line) * N1 + x]); };
        auto st_s = [&](int, int x, int r, Cx<T> v) {
            const int ia = rows.at(iax, x, r);
            if (ia >= 0) Sb[ia * LD] = v;
        };
        pwf::group_fft_vpair<T, N1>(m.Xw, nl, Tw<T>{m.tx}, lane, ld_s, vsc, st_s);
    }
}

template <typename T, int N1, bool RS>
__device__ __noinline__ void x_rho(Shape h, int Nxa, int N2, T *__restrict__ rp, T wb) {
    constexpr int G = pwf::fp_group<N1>();
    const Sm<T> m(h, 1, Nxa, N2);
    T *Rs = m.P;
    const short *iax = m.iax;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const XRows<N1> rows(iax, lane);
    const int LD = h.LD;
    for (int g0 = warp * G; g0 < N2; g0 += NW * G) {
        const int nl = min(G, N2 - g0);
        const Cx<T> *Sb = m.S + ypos(h, g0 + rows.line);
        auto ld_s = [&](int, int x, int r) {
            const int ia = rows.at(iax, x, r);
            return ia >= 0 ? Sb[ia * LD] : cmake((T)0, (T)0);
        };
        auto st_r = [&](int line, int x, int, Cx<T> v) {
            T *p = RS ? &Rs[(g0 + line) * h.vst + x] : &rp[(g0 + line) * N1 + x];
            *p += wb * (v.x * v.x + v.y * v.y);
        };
        pwf::group_fft<T, N1>(m.Xw, nl, Tw<T>{m.tx}, +1, lane, ld_s, st_r);
    }
}

template <typename T> size_t sm_bytes(const Shape &h, int nsub, int Nxa, int N1, int N2) {
    return ((size_t)2 * TWN + (size_t)nsub * Nxa * h.LD + (size_t)NW * h.xw) * sizeof(Cx<T>) + (size_t)N2 * h.vst * sizeof(T) +
           N1 * sizeof(short);
}

// the pass of a line length (uniform over the launch)
template <typename T> using YFn = void (*)(Shape, int, int, int, int);
template <typename T> __device__ __forceinline__ YFn<T> y_function(int n) {
    YFn<T> f = nullptr;
    switch (n) {
#define PW_C(N)            \
    case N:                \
        f = y_pass<T, N>; \
        break;
        PW_ANY_SIZES(PW_C)
#undef PW_C
    }
    return f;
}
template <typename T> using XFn = void (*)(Shape, int, int, int, const T *);
template <typename T, bool VS> __device__ __forceinline__ XFn<T> x_vloc_function(int n) {
    XFn<T> f = nullptr;
    switch (n) {
#define PW_C(N)                \
    case N:                    \
        f = x_vloc<T, N, VS>; \
        break;
        PW_ANY_SIZES(PW_C)
#undef PW_C
    }
    return f;
}
template <typename T> using RFn = void (*)(Shape, int, int, T *, T);
template <typename T, bool RS> __device__ __forceinline__ RFn<T> x_rho_function(int n) {
    RFn<T> f = nullptr;
    switch (n) {
#define PW_C(N)               \
    case N:                   \
        f = x_rho<T, N, RS>; \
        break;
        PW_ANY_SIZES(PW_C)
#undef PW_C
    }
    return f;
}

template <typename T>
__device__ __forceinline__ void setup(const KPlan &kp, const Shape &h, const Sm<T> &m, const Cx<T> *__restrict__ twx,
                                      const Cx<T> *__restrict__ twy) {
    for (int i = threadIdx.x; i < kp.N1; i += THREADS) m.iax[i] = -1;
    // (one-stage plans: R0 = 0, no twiddles)
    const int nx = h.R0x ? kp.N1 : 0, ny = h.R0y ? kp.N2 : 0;
    for (int i = h.R0x + threadIdx.x; i < nx; i += THREADS) m.tx[i] = twx[tw_entry(i, h.R0x)];
    for (int i = h.R0y + threadIdx.x; i < ny; i += THREADS) m.ty[i] = twy[tw_entry(i, h.R0y)];
}
// S := the plane's columns (zeros elsewhere), nbh bands
template <typename T>
__device__ __forceinline__ void fill(const KPlan &kp, const Shape &h, const Sm<T> &m, const Cx<T> *__restrict__ Ap, size_t astr,
                                     int nbh) {
    const int SP = kp.Nxa * h.LD;
    for (int i = threadIdx.x; i < nbh * SP; i += THREADS) m.S[i] = cmake((T)0, (T)0);
    __syncthreads();
    for (int i = threadIdx.x; i < kp.Nxa; i += THREADS) m.iax[kp.xa[i]] = (short)i;
    for (int bb = 0; bb < nbh; ++bb) {
        const Cx<T> *a = Ap + bb * astr;
        Cx<T> *Sb = m.S + (size_t)bb * SP;
#pragma unroll 4
        for (int c = threadIdx.x; c < kp.Ncol; c += THREADS) Sb[kp.col_ia[c] * h.LD + ypos(h, kp.col_j[c])] = a[c];
    }
    __syncthreads();
}

template <typename T> struct MinB { static constexpr int v = sizeof(T) == 4 ? 2 : 1; };

// op_V_loc on plane blockIdx.x of bands [bpc blockIdx.y, ...): inverse y and x,
// times V(r)/N, forward x and y, in place in A.
template <typename T, bool VS>
__global__ void __launch_bounds__(THREADS, MinB<T>::v)
ka_plane_vloc(KPlan kp, Shape h, const Cx<T> *__restrict__ twx, const Cx<T> *__restrict__ twy, const T *__restrict__ Vr,
              Cx<T> *__restrict__ A, int nb) {
    const Sm<T> m(h, h.bpc, kp.Nxa, kp.N2);
    const int kz = blockIdx.x, b0 = blockIdx.y * h.bpc, nbh = min(h.bpc, nb - b0);
    const size_t astr = (size_t)kp.N3 * kp.Ncol;
    Cx<T> *Ap = A + b0 * astr + (size_t)kz * kp.Ncol;
    const T *Vp = Vr + (size_t)kz * kp.N1 * kp.N2;
    if constexpr (VS) {
        for (int y = threadIdx.x >> 5; y < kp.N2; y += NW)
            for (int x = threadIdx.x & 31; x < kp.N1; x += 32) {
                const unsigned sa = (unsigned)__cvta_generic_to_shared(&m.P[y * h.vst + x]);
                if constexpr (sizeof(T) == 4)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(&Vp[y * kp.N1 + x]) : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(&Vp[y * kp.N1 + x]) : "memory");
            }
    }
    setup<T>(kp, h, m, twx, twy);
    fill<T>(kp, h, m, Ap, astr, nbh);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        y_function<T>(kp.N2)(h, h.bpc, kp.Nxa, nbh * kp.Nxa, pass ? -1 : +1);
        if (pass) break;
        if constexpr (VS) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
        x_vloc_function<T, VS>(kp.N1)(h, kp.Nxa, kp.N2, nbh, Vp);
        __syncthreads();
    }
    for (int bb = 0; bb < nbh; ++bb) {
        Cx<T> *a = Ap + bb * astr;
        const Cx<T> *Sb = m.S + (size_t)bb * kp.Nxa * h.LD;
#pragma unroll 4
        for (int c = threadIdx.x; c < kp.Ncol; c += THREADS) a[c] = Sb[kp.col_ia[c] * h.LD + ypos(h, kp.col_j[c])];
    }
}

// calc_rhoe: bands [g Bg, min(nb, (g + 1) Bg)) of plane kz into partial sum g.
template <typename T, bool RS>
__global__ void __launch_bounds__(THREADS, MinB<T>::v)
ka_plane_rho(KPlan kp, Shape h, const Cx<T> *__restrict__ twx, const Cx<T> *__restrict__ twy, const Cx<T> *__restrict__ A,
             int nb, int Bg, const double *__restrict__ w, T *__restrict__ rho_part) {
    const Sm<T> m(h, 1, kp.Nxa, kp.N2);
    const int kz = blockIdx.x, g = blockIdx.y, N12 = kp.N1 * kp.N2;
    T *rp = rho_part + ((size_t)g * kp.N3 + kz) * N12;
    setup<T>(kp, h, m, twx, twy);
    if constexpr (RS) {
        for (int i = threadIdx.x; i < kp.N2 * h.vst; i += THREADS) m.P[i] = (T)0;
    } else {
        for (int i = threadIdx.x; i < N12; i += THREADS) rp[i] = (T)0;
    }
    const int b1 = min(nb, (g + 1) * Bg);
    for (int b = g * Bg; b < b1; ++b) {
        fill<T>(kp, h, m, A + ((size_t)b * kp.N3 + kz) * kp.Ncol, 0, 1);
        y_function<T>(kp.N2)(h, 1, kp.Nxa, kp.Nxa, +1);
        x_rho_function<T, RS>(kp.N1)(h, kp.Nxa, kp.N2, rp, (T)w[b]);
        __syncthreads();
    }
    if constexpr (RS)
        for (int y = threadIdx.x >> 5; y < kp.N2; y += NW)
            for (int x = threadIdx.x & 31; x < kp.N1; x += 32) rp[(size_t)y * kp.N1 + x] = m.P[y * h.vst + x];
}

// ------------------------------------------------------------------- host
struct Line {
    int R0 = 0, R1 = 0, G = 0, xs = 0, pad = 0;
};
inline bool line_of(int n, Line &l) {
#define PW_C(N)                                                                                                   \
    if (n == N) {                                                                                                 \
        l.R0 = pwf::FPlan<N>::r(0);                                                                               \
        l.R1 = pwf::FPlan<N>::nst == 2 ? pwf::FPlan<N>::r(1) : 0;                                                 \
        l.G = pwf::fp_group<N>();                                                                                 \
        l.xs = pwf::fp_xs<N>();                                                                                   \
        l.pad = pwf::fp_pad<N>();                                                                                 \
        return true;                                                                                              \
    }
    PW_ANY_SIZES(PW_C)
#undef PW_C
    return false;
}

// Bands per CTA: the line groups of a direction go to 8 warps in rounds, and a
// last round with few groups wastes the rest; the bpc (1-4) with the fewest
// rounds per band (an x round, inverse and forward, counted twice a y one)
// among those that leave two CTAs an SM (FP32; one for FP64) and at least two
// per SM to launch.  (Also fewer barriers and V(r) loads per band.)
template <typename T> int pick_bpc(const KPlan &kp, const Shape &h0, const Line &lx, const Line &ly, int nb) {
    const size_t lim = sizeof(T) == 4 ? 113 * 1024 : 227 * 1024;
    int best = 1;
    double cost = 1e300;
    for (int b = 1; b <= 4; ++b) {
        if (b > 1 && (sm_bytes<T>(h0, b, kp.Nxa, kp.N1, kp.N2) > lim || (int64_t)kp.N3 * ((nb + b - 1) / b) < 2 * 148)) break;
        const int gy = b * kp.Nxa, ry = ((gy + ly.G - 1) / ly.G + NW - 1) / NW;
        const int gx = b * ((kp.N2 + lx.G - 1) / lx.G), rx = (gx + NW - 1) / NW;
        const double c = (2.0 * ry * ly.G * kp.N2 + 2.0 * rx * lx.G * kp.N1 + 64.0) / b;
        if (c < 0.98 * cost) {
            cost = c;
            best = b;
        }
    }
    return best;
}

template <typename T> bool shape_of(const KPlan &kp, size_t plane_max, Shape &h, Line &lx, Line &ly) {
    if (!line_of(kp.N1, lx) || !line_of(kp.N2, ly) || kp.Nxa > 255) return false;
    h.bpc = 1;
    h.LD = ly.xs;
    h.padm = ly.pad ? 65536 / ly.R0 + 1 : 0;
    h.R0x = lx.R1 ? lx.R0 : 0;
    h.R0y = ly.R1 ? ly.R0 : 0;
    h.xw = lx.R1 ? lx.G * lx.xs : 0;
    // rows of an FP32 plane 16 words apart modulo 32: the two half-warps of an
    // x group read adjacent rows
    h.vst = sizeof(T) == 4 ? kp.N1 + ((16 - kp.N1) % 32 + 32) % 32 : kp.N1;
    if ((size_t)kp.N2 * h.vst * sizeof(T) > plane_max) h.vst = 0;
    return true;
}

template <typename T>
cudaError_t plane_vloc(const FftLaunch &L, const void *Vr, void *A, int nb, cudaStream_t st) {
    const KPlan &kp = L.kp;
    Shape h;
    Line lx, ly;
    if (!shape_of<T>(kp, sizeof(T) == 4 ? 32 * 1024 : 48 * 1024, h, lx, ly)) return cudaErrorNotSupported;
    if (h.vst && sm_bytes<T>(h, 1, kp.Nxa, kp.N1, kp.N2) > (sizeof(T) == 4 ? 113 : 227) * 1024) h.vst = 0;
    h.bpc = L.bpc_set > 0 ? L.bpc_set : pick_bpc<T>(kp, h, lx, ly, nb);
    while (h.bpc > 1 && sm_bytes<T>(h, h.bpc, kp.Nxa, kp.N1, kp.N2) > 227 * 1024) --h.bpc;
    const size_t smem = sm_bytes<T>(h, h.bpc, kp.Nxa, kp.N1, kp.N2);
    if (smem > 227 * 1024) return cudaErrorNotSupported;
    const void *fn = h.vst ? (const void *)ka_plane_vloc<T, true> : (const void *)ka_plane_vloc<T, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    const dim3 grid(kp.N3, (nb + h.bpc - 1) / h.bpc);
    const Cx<T> *twx = (const Cx<T> *)L.twx, *twy = (const Cx<T> *)L.twy;
    if (h.vst)
        ka_plane_vloc<T, true><<<grid, THREADS, smem, st>>>(kp, h, twx, twy, (const T *)Vr, (Cx<T> *)A, nb);
    else
        ka_plane_vloc<T, false><<<grid, THREADS, smem, st>>>(kp, h, twx, twy, (const T *)Vr, (Cx<T> *)A, nb);
    return cudaGetLastError();
}

template <typename T>
cudaError_t plane_rho(const FftLaunch &L, const void *A, int nb, int G, int Bg, const double *w, void *rho_part, cudaStream_t st,
                      int *per_sm) {
    const KPlan &kp = L.kp;
    Shape h;
    Line lx, ly;
    if (!shape_of<T>(kp, sizeof(T) == 4 ? 32 * 1024 : 48 * 1024, h, lx, ly)) return cudaErrorNotSupported;
    if (h.vst && sm_bytes<T>(h, 1, kp.Nxa, kp.N1, kp.N2) > (sizeof(T) == 4 ? 113 : 227) * 1024) h.vst = 0;
    const size_t smem = sm_bytes<T>(h, 1, kp.Nxa, kp.N1, kp.N2);
    if (smem > 227 * 1024) return cudaErrorNotSupported;
    const void *fn = h.vst ? (const void *)ka_plane_rho<T, true> : (const void *)ka_plane_rho<T, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    if (per_sm) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, THREADS, smem);
    const dim3 grid(kp.N3, G);
    const Cx<T> *twx = (const Cx<T> *)L.twx, *twy = (const Cx<T> *)L.twy;
    if (h.vst)
        ka_plane_rho<T, true><<<grid, THREADS, smem, st>>>(kp, h, twx, twy, (const Cx<T> *)A, nb, Bg, w, (T *)rho_part);
    else
        ka_plane_rho<T, false><<<grid, THREADS, smem, st>>>(kp, h, twx, twy, (const Cx<T> *)A, nb, Bg, w, (T *)rho_part);
    return cudaGetLastError();
}

}  // namespace any
}  // namespace pwk
