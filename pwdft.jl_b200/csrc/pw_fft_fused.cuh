// Line FFTs with composite radices held entirely in registers.
//
// Same in-place Stockham stages and warp-group organisation as
// pw_fft_tmpl.cuh, but a stage may use a composite radix R = R1*R2 whose
// R-point DFT runs inside one thread (Cooley-Tukey split: R2 DFTs of size R1,
// twiddles W_R^(n2 k1), R1 DFTs of size R2).  Fewer stages means fewer
// shared-memory round trips per line: 75 = 15*5 and 120 = 15*8 take two
// passes instead of three, 27 takes one.
#pragma once
#include "pw_fft.cuh"
#include <type_traits>

namespace pwf {

template <typename T, int R> struct Dft;

// radices with direct formulas
template <typename T> struct Dft<T, 2> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *, int) { SmallDft<T, 2>::run(v, s); } };
template <typename T> struct Dft<T, 3> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *, int) { SmallDft<T, 3>::run(v, s); } };
template <typename T> struct Dft<T, 4> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *, int) { SmallDft<T, 4>::run(v, s); } };
template <typename T> struct Dft<T, 5> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *, int) { SmallDft<T, 5>::run(v, s); } };
template <typename T> struct Dft<T, 8> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *, int) { SmallDft<T, 8>::run(v, s); } };

// exp(-2 pi i m / R) at compile time, rounded once: the angle is reduced to
// [0, pi/4] as a fraction of a turn, and the Taylor series of sin and cos is summed
// in pairs of doubles (the sum of a pair is exact to about 2^-100).  A series in
// plain doubles on [-pi, pi] was off by up to 4e-16: lines of 36 to 125 points with
// a radix of 9, 16, 25 or 27 lost up to 1.3 times the error of a rounded table.
struct Pair {
    double h, l;
};
__host__ __device__ constexpr Pair two_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
__host__ __device__ constexpr Pair two_prod(double a, double b) {   // Dekker: 26-bit halves
    const double ca = 134217729.0 * a, ah = ca - (ca - a), al = a - ah;
    const double cb = 134217729.0 * b, bh = cb - (cb - b), bl = b - bh, p = a * b;
    return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
__host__ __device__ constexpr Pair operator+(Pair a, Pair b) {
    const Pair s = two_sum(a.h, b.h);
    return two_sum(s.h, s.l + a.l + b.l);
}
__host__ __device__ constexpr Pair operator*(Pair a, Pair b) {
    const Pair p = two_prod(a.h, b.h);
    return two_sum(p.h, p.l + a.h * b.l + a.l * b.h);
}
__host__ __device__ constexpr Pair operator/(Pair a, double d) {
    const double q = a.h / d;
    const Pair p = two_prod(q, -d), r = Pair{a.h, a.l} + p;
    return two_sum(q, r.h / d);
}
// cos or sin of 2 pi p / q for 0 <= p / q <= 1/8
__host__ __device__ constexpr double ce_octant(int p, int q, bool sine) {
    const Pair x = Pair{6.283185307179586, 2.4492935982947064e-16} * Pair{(double)p, 0.0} / (double)q;
    const Pair x2 = x * x;
    Pair term = sine ? x : Pair{1.0, 0.0}, sum = term;
    for (int k = 1; k < 16; ++k) {
        const int a = sine ? 2 * k : 2 * k - 1;
        term = Pair{-x2.h, -x2.l} * term / (double)(a * (a + 1));
        sum = sum + term;
    }
    return sum.h;
}
__host__ __device__ constexpr double ce_trig(int p, int q, bool sine) {   // 0 <= p < q
    double sign = 1.0;
    if (2 * p > q) {   // past half a turn: -p
        p = q - p;
        if (sine) sign = -sign;
    }
    if (4 * p > q) {   // past a quarter: half a turn less
        p = q - 2 * p;
        q *= 2;
        if (!sine) sign = -sign;
    }
    if (8 * p > q) return sign * ce_octant(q - 4 * p, 4 * q, !sine);
    return sign * ce_octant(p, q, sine);
}
template <int M, int R> struct Root {
    static constexpr double c = ce_trig(M % R, R, false), s = -ce_trig(M % R, R, true);
};

// compile-time loop: f(std::integral_constant<int, I>) for I in [I0, I1)
template <int I0, int I1, class F> __host__ __device__ __forceinline__ void sfor(F &&f) {
    if constexpr (I0 < I1) {
        f(std::integral_constant<int, I0>{});
        sfor<I0 + 1, I1>(f);
    }
}

// R = R1*R2 in registers, twiddles W_R^(n2 k1) as compile-time constants
// (no table reads; tw and step pass through to the sub-DFTs, which ignore
// them too).
template <typename T, int R1, int R2> struct CompDft {
    static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int step) {
        constexpr int R = R1 * R2;
        Cx<T> a[R];
        sfor<0, R2>([&](auto n2c) {
            constexpr int n2 = decltype(n2c)::value;
            Cx<T> t[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + n2];
            Dft<T, R1>::run(t, s, tw, step * R2);
            sfor<0, R1>([&](auto k1c) {
                constexpr int k1 = decltype(k1c)::value;
                if constexpr (n2 * k1 != 0) {
                    using W = Root<n2 * k1, R>;
                    const T wy = s > 0 ? (T)-W::s : (T)W::s;
                    t[k1] = cmul(t[k1], cmake((T)W::c, wy));
                }
                a[n2 * R1 + k1] = t[k1];
            });
        });
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            Cx<T> t[R2];
#pragma unroll
            for (int n2 = 0; n2 < R2; ++n2) t[n2] = a[n2 * R1 + k1];
            Dft<T, R2>::run(t, s, tw, step * R1);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k2];
        }
    }
};
// R = R1*R2 with gcd(R1, R2) = 1 (Good-Thomas prime-factor split): input
// n = (R2 n1 + R1 n2) mod R and output k = CRT(k1 mod R1, k2 mod R2) turn
// W_R^(nk) into W_R1^(n1 k1) W_R2^(n2 k2), so no twiddles sit between the
// R2 DFTs of size R1 and the R1 DFTs of size R2 (both index maps are
// compile-time register permutations).
template <int A, int M> __host__ __device__ constexpr int inv_mod() {
    int r = 1;
    while ((A * r) % M != 1) ++r;
    return r;
}
template <typename T, int R1, int R2> struct PfaDft {
    static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int step) {
        constexpr int R = R1 * R2;
        constexpr int E1 = R2 * inv_mod<R2 % R1, R1>(), E2 = R1 * inv_mod<R1 % R2, R2>();   // CRT idempotents
        Cx<T> a[R];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
            Cx<T> t[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[(R2 * n1 + R1 * n2) % R];
            Dft<T, R1>::run(t, s, tw, step);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) a[n2 * R1 + k1] = t[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            Cx<T> t[R2];
#pragma unroll
            for (int n2 = 0; n2 < R2; ++n2) t[n2] = a[n2 * R1 + k1];
            Dft<T, R2>::run(t, s, tw, step);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) v[(E1 * k1 + E2 * k2) % R] = t[k2];
        }
    }
};
template <typename T> struct Dft<T, 10> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { PfaDft<T, 2, 5>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 12> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { PfaDft<T, 3, 4>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 16> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { CompDft<T, 4, 4>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 9> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { CompDft<T, 3, 3>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 15> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { PfaDft<T, 3, 5>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 18> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { PfaDft<T, 2, 9>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 24> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { CompDft<T, 8, 3>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 25> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { CompDft<T, 5, 5>::run(v, s, tw, st); } };
template <typename T> struct Dft<T, 27> { static __host__ __device__ __forceinline__ void run(Cx<T> *v, T s, const Cx<T> *tw, int st) { CompDft<T, 9, 3>::run(v, s, tw, st); } };

// Fused plans: radices per stage (product = N).
template <int N> struct FPlan;
template <> struct FPlan<27> { static constexpr int nst = 1; static __host__ __device__ constexpr int r(int) { return 27; } };
template <> struct FPlan<75> { static constexpr int nst = 2; static __host__ __device__ constexpr int r(int s) { return s == 0 ? 15 : 5; } };
// 120 = 15 * 8: 91-110 registers in the z and plane kernels (24 * 5 needed 128 and spilled
// 72-432 bytes); measured Si216 FFT round trip 7.95 -> 6.52 ms
template <> struct FPlan<120> { static constexpr int nst = 2; static __host__ __device__ constexpr int r(int s) { return s == 0 ? 15 : 8; } };

// The other line lengths of common cutoffs: R0 R1 with R1 <= R0 (a warp's
// first-stage butterflies of its 32 / R1 lines then fill one round) and R0 odd
// where there is a choice (its outputs, R0 apart, fall on different banks;
// the even ones are padded, see fp_pad).
#define PW_FPLAN2(N, R0, R1) \
    template <> struct FPlan<N> { static constexpr int nst = 2; static __host__ __device__ constexpr int r(int s) { return s == 0 ? R0 : R1; } };
PW_FPLAN2(20, 5, 4)
PW_FPLAN2(24, 8, 3)
PW_FPLAN2(25, 5, 5)
PW_FPLAN2(30, 15, 2)
PW_FPLAN2(32, 8, 4)
PW_FPLAN2(36, 9, 4)
PW_FPLAN2(40, 8, 5)
PW_FPLAN2(45, 9, 5)
PW_FPLAN2(48, 12, 4)
PW_FPLAN2(50, 10, 5)
PW_FPLAN2(54, 18, 3)
PW_FPLAN2(60, 15, 4)
PW_FPLAN2(64, 8, 8)
PW_FPLAN2(72, 9, 8)
PW_FPLAN2(80, 16, 5)
PW_FPLAN2(81, 27, 3)
PW_FPLAN2(90, 18, 5)
PW_FPLAN2(96, 12, 8)
PW_FPLAN2(100, 25, 4)
PW_FPLAN2(108, 27, 4)
PW_FPLAN2(125, 25, 5)
PW_FPLAN2(128, 16, 8)
#undef PW_FPLAN2

template <int N> __host__ __device__ constexpr int fp_ns(int s) {
    int p = 1;
    for (int i = 0; i < s; ++i) p *= FPlan<N>::r(i);
    return p;
}
// lines per warp group: the stage with the fewest butterflies per line fills 32 lanes
template <int N> __host__ __device__ constexpr int fp_group() {
    int mn = N;
    for (int s = 0; s < FPlan<N>::nst; ++s) {
        const int nbf = N / FPlan<N>::r(s);
        mn = nbf < mn ? nbf : mn;
    }
    return 32 / mn > 0 ? 32 / mn : 1;
}

// Shared-memory twiddle layout of the fused plans.  One-stage plans keep
// tw[m] = exp(-2 pi i m / N).  Two-stage plans (N = R0 R1) store
//   tw[m]                     = exp(-2 pi i m / R0)   for m < R0 (the
//                               composite DFTs now hold their roots as
//                               compile-time constants and do not read them);
//   tw[R0 + (r - 1) R0 + j]   = exp(-2 pi i r j / N)  for 1 <= r < R1, j < R0,
//                               the stage-1 twiddles, which lanes with
//                               consecutive j read from consecutive words
// (the natural table read at r j puts 2 and 4 lanes of a half-warp on one
// bank for r = 2 and 4).  N entries either way; tw_src(i) is the natural
// index of entry i, for filling the table from tw[m] = exp(-2 pi i m / N).
template <int N> __host__ __device__ constexpr int tw_src(int i) {
    if constexpr (FPlan<N>::nst == 1) {
        return i;
    } else {
        constexpr int R0 = FPlan<N>::r(0);
        return i < R0 ? i * (N / R0) : ((i - R0) / R0 + 1) * ((i - R0) % R0);
    }
}
// step argument of the DFT of stage S: the radix-R0 roots sit at stride 1;
// the stage-1 radix of a two-stage plan reads no table
template <int R> __host__ __device__ constexpr bool direct_radix() { return R == 2 || R == 3 || R == 4 || R == 5 || R == 8; }
template <int N, int S> __host__ __device__ constexpr int tw_step() {
    static_assert(FPlan<N>::nst == 1 || direct_radix<FPlan<N>::r(1)>(), "two-stage plans end on a direct radix");
    return (FPlan<N>::nst == 2 && S == 0) ? 1 : N / FPlan<N>::r(S);
}
// twiddle of element r of stage-S butterfly jm (jm < N_S, the stage's span)
// Padded element positions of a line held in shared memory: pos(x) = x +
// (x / R0) * fp_pad, line stride fp_xs.  Plans with an even R0 would put the
// first stage's outputs (R0 elements apart across lanes) on few banks, so they
// take one spare element per R0; odd ones are unpadded.
template <int N> __host__ __device__ constexpr int fp_pad() { return FPlan<N>::nst == 2 && FPlan<N>::r(0) % 2 == 0 ? 1 : 0; }
template <int N> __host__ __device__ constexpr int fp_pos(int x) {
    if constexpr (fp_pad<N>() == 0)
        return x;
    else
        return x + (x / FPlan<N>::r(0)) * fp_pad<N>();
}
// Line stride = R1 modulo 16: the 16 / R1 lines of a half-warp then start on
// different banks in the first stage (75 = 11 modulo 16 does as well).
template <int N> __host__ __device__ constexpr int fp_xs() {
    if constexpr (FPlan<N>::nst == 1 || N == 75) {
        return N;
    } else {
        constexpr int base = N + N / FPlan<N>::r(0) * fp_pad<N>(), r1 = FPlan<N>::r(1);
        return base + ((r1 - base) % 16 + 16) % 16;
    }
}
static_assert(fp_xs<120>() == 120 && fp_pad<120>() == 0, "the 120-point plan is unpadded");

// twiddle of element r of stage-S butterfly jm (jm < N_S, the stage's span)
template <int N, int S> __host__ __device__ __forceinline__ int tw_at(int r, int jm) {
    if constexpr (FPlan<N>::nst == 2 && S == 1) {
        constexpr int R0 = FPlan<N>::r(0);
        return R0 + (r - 1) * R0 + jm;
    } else {
        constexpr int R = FPlan<N>::r(S);
        return r * jm * (N / (fp_ns<N>(S) * R));
    }
}

// Lane assignment of round t of a stage with NBF butterflies per line and
// G lines per warp group.  Shared memory serves an 8-byte access one
// half-warp at a time, so with NBF <= 16 every half-warp takes whole lines
// (H = 16 / NBF of them, the rest of its lanes idle): its accesses are then H
// runs of NBF consecutive elements, one per line, instead of runs that
// straddle a line boundary onto banks the half-warp already uses (measured
// model of the 75-point plane kernel: 27 % of its shared-memory wavefronts
// were such conflicts).  The number of rounds equals the packed mapping's
// for every plan here (75: 5 and 15 butterflies, 6 lines; 120: 8 and 15, 4;
// 27: 1, 32).
template <int NBF, int G> struct LaneMap {
    static constexpr int H = NBF <= 16 ? 16 / NBF : 0;
    static constexpr int ROUNDS = H ? (G + 2 * H - 1) / (2 * H) : (G * NBF + 31) / 32;
    static __host__ __device__ __forceinline__ bool at(int lane, int t, int nl, int &line, int &j) {
        if constexpr (H > 0) {
            const int sub = lane & 15, li = sub / NBF;
            j = sub - li * NBF;
            line = (2 * t + (lane >> 4)) * H + li;
            return li < H && line < nl;
        } else {
            const int id = lane + 32 * t;
            line = id / NBF;
            j = id - line * NBF;
            return id < nl * NBF;
        }
    }
};

// w[r] = w1^r for r < R, w[r] = w[r / 2] w[r - r / 2] (about log2(r) + 1
// roundings): the stage twiddles of one butterfly from a single table read.
template <typename T, int R> __host__ __device__ __forceinline__ void tw_pow(Cx<T> w1, Cx<T> (&w)[R]) {
    w[0] = cmake((T)1, (T)0);
    if constexpr (R > 1) w[1] = w1;
#pragma unroll
    for (int r = 2; r < R; ++r) w[r] = cmul(w[r / 2], w[r - r / 2]);
}

// Twiddles of butterfly jm of stage S (conjugated for the inverse, sign > 0)
// applied to v[1 .. R).  Only the second stage of a two-stage plan has any;
// its table entry tw_at(1, jm) is exp(-2 pi i jm / N).
// With a whole table (FullTw) every power is read instead: the powers lose up to
// a bit against entries that were rounded once.  FP32 density of 8 bands, 32 / 60
// points: relative error 2.7e-7 / 1.3e-7 against 1.4e-7 / 0.8e-7 (op_H of 8 atoms
// 69.7 against 70.1 us); FP64 density of 4 bands, 40 / 64 / 72 points: 3.3e-16 /
// 4.4e-16 / 4.5e-16 against 2.5e-16 / 3.1e-16 / 2.4e-16 (op_H and density of 40
// bands on 22 boxes at most 3 % longer, 5 % at 72 points; 81 points 3 % shorter).
template <typename T> struct FullTw {
    const Cx<T> *p;
    __host__ __device__ __forceinline__ operator const Cx<T> *() const { return p; }
};
template <typename T, int N, int S, int R>
__host__ __device__ __forceinline__ void apply_tw(Cx<T> (&v)[R], FullTw<T> tw, int jm, int sign) {
#pragma unroll
    for (int r = 1; r < R; ++r) {
        Cx<T> w = tw.p[tw_at<N, S>(r, jm)];
        if (sign > 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
    }
}
template <typename T, int N, int S, int R>
__host__ __device__ __forceinline__ void apply_tw(Cx<T> (&v)[R], const Cx<T> *tw, int jm, int sign) {
    Cx<T> w1 = tw[tw_at<N, S>(1, jm)];
    if (sign > 0) w1.y = -w1.y;
    Cx<T> w[R];
    tw_pow<T, R>(w1, w);
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r]);
}

// PAD: elements at fp_pos(x) (es must be 1, two-stage plans): stage 0 writes
// block j of R0 elements, stage 1 touches element j < R0 of block r
template <typename T, int N, int S, bool JFAST, bool PAD, class TW>
__device__ __forceinline__ void fstage(Cx<T> *buf, int l0, int nl, int es, int ls, TW tw, int sign, int lane) {
    constexpr int R = FPlan<N>::r(S);
    constexpr int NS = fp_ns<N>(S);
    constexpr int NBF = N / R;
    constexpr int G = fp_group<N>();
    using LM = LaneMap<NBF, G>;
    // JFAST lines: whole lines per half-warp; otherwise (z columns, line
    // index fastest) the packed order, whose strides the callers choose
    constexpr int MAXB = JFAST ? LM::ROUNDS : (G * NBF + 31) / 32;
    auto slot = [&](int t, int &line, int &j) -> bool {
        if constexpr (JFAST) {
            const bool ok = LM::at(lane, t, nl, line, j);
            line += l0;
            return ok;
        } else {
            const int id = lane + 32 * t;
            line = l0 + id % nl;
            j = id / nl;
            return id < nl * NBF;
        }
    };
    const T sg = (T)sign;
    Cx<T> v[MAXB][R];
#pragma unroll
    for (int t = 0; t < MAXB; ++t) {
        int line, j;
        if (slot(t, line, j)) {
            const int jm = j % NS;
            const Cx<T> *p = buf + line * ls + j * es;
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[t][r] = PAD ? buf[line * ls + (S == 1 ? j + r * (NBF + fp_pad<N>()) : fp_pos<N>(j + r * NBF))] : p[r * NBF * es];
            if constexpr (NS > 1) apply_tw<T, N, S, R>(v[t], tw, jm, sign);
            Dft<T, R>::run(v[t], sg, tw, tw_step<N, S>());
        }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < MAXB; ++t) {
        int line, j;
        if (slot(t, line, j)) {
            const int jm = j % NS;
            const int x0 = (j / NS) * NS * R + jm;
            Cx<T> *q = buf + line * ls + x0 * es;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (PAD)
                    buf[line * ls + (S == 1 ? x0 + r * (NS + fp_pad<N>()) : x0 + j * fp_pad<N>() + r)] = v[t][r];
                else
                    q[r * NS * es] = v[t][r];
            }
        }
    }
    __syncwarp();
    if constexpr (S + 1 < FPlan<N>::nst) fstage<T, N, S + 1, JFAST, PAD>(buf, l0, nl, es, ls, tw, sign, lane);
}

// All lines [0, nlines) of length N; ends with __syncthreads().
template <typename T, int N, bool JFAST, bool PAD = false, class TW = const Cx<T> *>
__device__ __forceinline__ void lines(Cx<T> *buf, int nlines, int es, int ls, TW tw, int sign) {
    constexpr int G = fp_group<N>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int l0 = warp * G; l0 < nlines; l0 += nw * G) {
        const int nl = min(G, nlines - l0);
        fstage<T, N, 0, JFAST, PAD>(buf, l0, nl, es, ls, tw, sign, lane);
    }
    __syncthreads();
}

}  // namespace pwf

namespace pwf {

// Stage S of the N-point line FFT for lines [0, nl) of one warp group, with
// element access through functors ld(line, x, r) -> Cx<T> and
// st(line, x, r, v) (x the element, r the compile-time slot of the lane's
// butterfly it sits in): the first stage of a line can read its input
// straight from another layout, the last can scale or scatter its output,
// with no extra pass.
template <typename T, int N, int S, class TW, class LD, class ST>
__device__ __forceinline__ void fstage_io(int nl, TW tw, int sign, int lane, LD &ld, ST &st) {
    constexpr int R = FPlan<N>::r(S);
    constexpr int NS = fp_ns<N>(S);
    constexpr int NBF = N / R;
    constexpr int G = fp_group<N>();
    using LM = LaneMap<NBF, G>;
    const T sg = (T)sign;
    Cx<T> v[LM::ROUNDS][R];
#pragma unroll
    for (int t = 0; t < LM::ROUNDS; ++t) {
        int line, j;
        if (LM::at(lane, t, nl, line, j)) {
            const int jm = j % NS;
#pragma unroll
            for (int r = 0; r < R; ++r) v[t][r] = ld(line, j + r * NBF, r);
            if constexpr (NS > 1) apply_tw<T, N, S, R>(v[t], tw, jm, sign);
            Dft<T, R>::run(v[t], sg, tw, tw_step<N, S>());
        }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < LM::ROUNDS; ++t) {
        int line, j;
        if (LM::at(lane, t, nl, line, j)) {
            const int jm = j % NS;
            const int x0 = (j / NS) * NS * R + jm;
#pragma unroll
            for (int r = 0; r < R; ++r) st(line, x0 + r * NS, r, v[t][r]);
        }
    }
    __syncwarp();
}

// Whole N-point FFT of nl <= fp_group<N>() lines held by one warp in buf
// (line stride fp_xs, padded positions): the first stage reads through ld0,
// the last writes through stl, the stages between use buf.
template <typename T, int N, class TW, class LD0, class STL>
__device__ __forceinline__ void group_fft(Cx<T> *buf, int nl, TW tw, int sign, int lane, LD0 &ld0, STL &stl) {
    constexpr int XS = fp_xs<N>();
    // stage 0 writes element r of block (x - r) / R0, stage 1 reads element x - r R0 of block r
    auto bld = [&](int line, int x, int r) { return buf[line * XS + x + r * fp_pad<N>()]; };
    auto bst = [&](int line, int x, int r, Cx<T> v) { buf[line * XS + fp_pos<N>(x - r) + r] = v; };
    constexpr int NST = FPlan<N>::nst;
    static_assert(NST == 1 || NST == 2, "fused plans have one or two stages");
    if constexpr (NST == 1) {
        fstage_io<T, N, 0>(nl, tw, sign, lane, ld0, stl);
    } else {
        fstage_io<T, N, 0>(nl, tw, sign, lane, ld0, bst);
        fstage_io<T, N, 1>(nl, tw, sign, lane, bld, stl);
    }
}

// Inverse N-point FFT, pointwise scale, forward FFT of nl <= fp_group<N>()
// lines held by one warp: the op_V_loc x-pass.  The inverse's last stage
// leaves lane (line, j) holding f[j + R0 r], r < R1 (N = R0 R1), which is
// exactly the input of a decimation-in-frequency forward step,
//   F[k2 + R1 k1] = sum_j w_R0^(j k1) [w_N^(j k2) sum_r f[j + R0 r] w_R1^(r k2)],
// so the scale (vsc(line, x)), the forward radix-R1 DFT and its twiddles
// stay in registers and one shared-memory exchange (buf) precedes the
// radix-R0 DFTs, whose outputs go out through st(line, x, r, v).  One-stage
// plans (one line per lane) never touch buf.
template <typename T, int N, class TW, class LD0, class VS, class ST>
__device__ __forceinline__ void group_fft_vpair(Cx<T> *buf, int nl, TW tw, int lane, LD0 &ld0, VS &vsc,
                                                ST &st) {
    constexpr int NST = FPlan<N>::nst;
    static_assert(NST == 1 || NST == 2, "fused plans have one or two stages");
    if constexpr (NST == 1) {
        if (lane < nl) {
            Cx<T> v[N];
#pragma unroll
            for (int r = 0; r < N; ++r) v[r] = ld0(lane, r, r);
            Dft<T, N>::run(v, (T)1, tw, 1);
#pragma unroll
            for (int r = 0; r < N; ++r) v[r] = cscale(v[r], vsc(lane, r));
            Dft<T, N>::run(v, (T)-1, tw, 1);
#pragma unroll
            for (int k = 0; k < N; ++k) st(lane, k, k, v[k]);
        }
        __syncwarp();
    } else {
        constexpr int R0 = FPlan<N>::r(0), R1 = FPlan<N>::r(1);
        constexpr int G = fp_group<N>();
        constexpr int XS = fp_xs<N>(), RP = R0 + fp_pad<N>();   // fp_pos(j + R0 r) = j + RP r for j < R0
        auto bst = [&](int line, int x, int r, Cx<T> v) { buf[line * XS + fp_pos<N>(x - r) + r] = v; };
        fstage_io<T, N, 0>(nl, tw, 1, lane, ld0, bst);   // inverse stage 0 into buf
        using L1 = LaneMap<R0, G>;                         // stage-1 butterflies: R0 per line
        Cx<T> v[L1::ROUNDS][R1];
#pragma unroll
        for (int t = 0; t < L1::ROUNDS; ++t) {
            int line, j;
            if (L1::at(lane, t, nl, line, j)) {
#pragma unroll
                for (int r = 0; r < R1; ++r) v[t][r] = buf[line * XS + j + r * RP];
                apply_tw<T, N, 1, R1>(v[t], tw, j, +1);
                Dft<T, R1>::run(v[t], (T)1, tw, N / R1);      // v[r] = f[j + R0 r]
#pragma unroll
                for (int r = 0; r < R1; ++r) v[t][r] = cscale(v[t][r], vsc(line, j + R0 * r));
                Dft<T, R1>::run(v[t], (T)-1, tw, N / R1);     // sum_r f[j + R0 r] w_R1^(r k2)
                apply_tw<T, N, 1, R1>(v[t], tw, j, -1);
            }
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < L1::ROUNDS; ++t) {
            int line, j;
            if (L1::at(lane, t, nl, line, j)) {
#pragma unroll
                for (int k2 = 0; k2 < R1; ++k2) buf[line * XS + k2 * RP + j] = v[t][k2];
            }
        }
        __syncwarp();
        using L2 = LaneMap<R1, G>;                         // radix-R0 butterflies: R1 per line
#pragma unroll
        for (int t = 0; t < L2::ROUNDS; ++t) {
            int line, k2;
            if (L2::at(lane, t, nl, line, k2)) {
                Cx<T> u[R0];
#pragma unroll
                for (int j = 0; j < R0; ++j) u[j] = buf[line * XS + k2 * RP + j];
                Dft<T, R0>::run(u, (T)-1, tw, tw_step<N, 0>());
#pragma unroll
                for (int k1 = 0; k1 < R0; ++k1) st(line, k2 + R1 * k1, k1, u[k1]);
            }
        }
        __syncwarp();
    }
}

}  // namespace pwf
