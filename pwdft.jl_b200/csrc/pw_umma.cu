// Complex GEMMs of the mixed-precision path on the 5th-generation tensor
// cores (tcgen05.mma, kind::f16 with BF16 operands, FP32 accumulation in
// TMEM, operands staged by TMA into 128B-swizzled shared memory).
//
// Every product is brought to one form, C (m x n complex) = Z^H W with
// Z (K x m) and W (K x n):
//   betaNL' psi        (PsPotNL.jl:252)              Z = betaNL,  W = psi
//   X'HX, Q'HQ, Q'Q    (diag_LOBPCG.jl:85,183-184)   Z = Q,       W = HQ / Q
//   A*U                (diag_LOBPCG.jl:188-194,
//                       op_V_Ps_nloc.jl:59-76)       Z = A^H,     W = U
// and formed as two real products over the real and imaginary parts,
//   Re C = Zr' Wr + Zi' Wi,   Im C = Zr' Wi - Zi' Wr.
// An operand row (one column of Z or W) holds its values along K in blocks of
// 32: 32 real parts, then 32 imaginary parts, one 128-byte swizzle row of BF16
// a block.  A k-block of Z and W in shared memory then serves both
// accumulators: Re C takes the parts as they lie, Im C pairs each half with
// the other half of W (the Zi half with a negated A operand), so each byte
// loaded feeds two products.  (Rows [Re, Im] and [-Im, Re] of one real GEMM of
// twice the rows, the form before this, load and store every Z value twice:
// betaNL P of 216 atoms and 480 bands ran at 75 loaded bytes a clock and SM,
// 0.91 of 1.38 PFLOP/s; this form loads 43.)  Measured: Q'HQ, Q'Q and Q U of
// 480 bands over 80,797 plane waves 11.0 -> 9.6 ms, op_H of 64 atoms (160 bands)
// 720 -> 694 us, of 216 atoms (480 bands) 8.86 -> 8.55 ms.
//
// Precision: split BF16 x 3.  Each FP32 operand x = hi + lo with
// hi = bf16(x), lo = bf16(x - hi); Z'W ~ hi*hi + hi*lo + lo*hi, all three
// accumulated in the same FP32 TMEM accumulator (relative error ~2^-17 per
// product, then FP32 accumulation).  The "prep" kernels below write the
// K-major BF16 pieces (transposing where Z = A^H) so that the MMA kernel only
// ever sees K-major operands.
//
// MMA kernel: 128 x BN complex output tile per CTA, k-blocks of 32 complex
// values, 2-3 stage TMA -> MMA pipeline on mbarriers, split-K over gridDim.z
// into an FP32 workspace, then a finalize kernel that sums the splits and
// writes the complex result (FP32 or FP64, overwrite or add); a single split
// goes through shared memory straight into C.  Persistent CTAs, one an SM.
// Warp roles: warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer,
// warps 2..5 = epilogue of Re C, warps 6..9 of Im C (TMEM -> registers ->
// global).  Every mbarrier wait is bounded; on expiry the CTA records an error
// code and returns after releasing its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>

#include "pw_launch.h"
#include "pw_umma.h"

namespace pwk {
namespace umma {

constexpr int BM = 128, BK = 64;            // complex rows of a tile; BF16 values of a k-block row (32 Re, 32 Im)
constexpr int TILE_A_BYTES = BM * BK * 2;   // 16 KB per A operand tile
constexpr int THREADS = 320;
constexpr long long WAIT_LIMIT = 1ll << 26;
constexpr int MAX_STAGES = 3;
constexpr int EC = 32;                      // output columns that the epilogue writes at a time

// NS = number of BF16 pieces per FP32 value: 2 (hi, lo: 3 products, ~2^-17)
// or 3 (hi, mid, lo: 6 products, ~2^-24, for products with heavy
// cancellation such as betaNL' psi).  BN = output tile width (complex
// columns).  Stages: as many as fit in 225 KB.
template <int NS, int BN> struct Cfg {
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 128, "tcgen05 N for M = 128; four accumulators in 512 TMEM columns");
    static constexpr int TILE_B_BYTES = BN * BK * 2;
    static constexpr int STAGE_BYTES = NS * (TILE_A_BYTES + TILE_B_BYTES);
    static constexpr int STAGES = (225 * 1024) / STAGE_BYTES < MAX_STAGES ? (225 * 1024) / STAGE_BYTES : MAX_STAGES;
    static_assert(STAGES >= 2, "at least a double-buffered pipeline");
    // the epilogue's copy of EC columns (of BM + 1 complex values) has its own
    // place where it fits beside the stages; else a CTA runs one tile and
    // reuses them
    static constexpr bool OWN_E = 1024 + STAGES * STAGE_BYTES + EC * (BM + 1) * 8 + 256 <= 227 * 1024;
    static constexpr int E_BYTES = OWN_E ? EC * (BM + 1) * 8 : 0;
    // Re and Im accumulators, double-buffered, each from a multiple of 32
    // columns on; allocation a power of two >= 32
    static constexpr int ACC = (BN + 31) / 32 * 32;
    static constexpr uint32_t TMEM_COLS = 4 * ACC <= 128 ? 128u : 4 * ACC <= 256 ? 256u : 512u;
    // kind::f16, A = B = BF16, D = F32, both K-major, M = 128, N = BN; NEG: A negated
    static constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    static constexpr uint32_t NEG = 1u << 13;
};

struct __align__(8) Bars {
    uint64_t full[MAX_STAGES];
    uint64_t empty[MAX_STAGES];
    uint64_t tfull[2];    // accumulator pair b holds a finished k-block
    uint64_t tempty[2];   // the epilogue has drained accumulator pair b
    uint32_t tmem_base;
    int failed;
};
template <int NS, int BN> constexpr size_t smem_bytes() {
    return 1024 + (size_t)Cfg<NS, BN>::STAGES * Cfg<NS, BN>::STAGE_BYTES + Cfg<NS, BN>::E_BYTES + sizeof(Bars);
}

__device__ __forceinline__ uint32_t su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity) {
    for (long long i = 0; i < WAIT_LIMIT; ++i)
        if (mbar_try(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            su32(dst)),
        "l"((uint64_t)map), "r"(su32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
    // K-major, 128B swizzle: LBO = 16 B (unused), SBO = 1024 B (8 rows x 128 B), version 1
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accum));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
                 : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive TMEM columns of this thread's lane (wait before use)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// EC columns of a tile from shared memory (T2, columns of BM + 1) to C: thread
// (r, h) writes row r of every other column, UB old values loaded together.
template <typename E>
__device__ __forceinline__ void store_columns(E *C, int64_t ld, const float2 *T2, int m0, int n0, int M, int N, int cols,
                                              bool add, bool up) {
    constexpr int UB = sizeof(E) == 16 ? 4 : 8;
    const int t = threadIdx.x - 64, r = t & (BM - 1), h = t >> 7, i = m0 + r;
#pragma unroll 1
    for (int c = h; c < cols; c += 2 * UB) {
        E o[UB];
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int n = n0 + c + 2 * u;
            o[u].x = o[u].y = 0;
            if (add && i < M && n < N && !(up && i > n)) o[u] = C[(size_t)n * ld + i];
        }
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int n = n0 + c + 2 * u;
            if (i < M && n < N && !(up && i > n)) {
                const float2 v = T2[(c + 2 * u) * (BM + 1) + r];
                o[u].x += v.x;
                o[u].y += v.y;
                C[(size_t)n * ld + i] = o[u];
            }
        }
    }
}

// The same columns' conjugates to the other triangle of C (one split of Z^H Z,
// complex128; the widest tile has no registers for it: 24 -> 40 bytes spilled).
template <int BN> constexpr bool MIRROR_BN = BN < 128;
__device__ __noinline__ void mirror_columns(double2 *C, int64_t ld, const float2 *T2, int m0, int n0, int N, int cols, bool add) {
    for (int e = threadIdx.x - 64; e < cols * BM; e += 256) {
        const int c = e / BM, r = e % BM, i = m0 + r, n = n0 + c;
        if (i < n && n < N) {
            double2 *h = C + (size_t)i * ld + n;
            const float2 v = T2[c * (BM + 1) + r];
            *h = make_double2((add ? h->x : 0.0) + v.x, (add ? h->y : 0.0) - v.y);
        }
    }
}

// C (m x n complex) = sum over the split's k-blocks of the piece products
//   NS = 2:  A0 B0 + A0 B1 + A1 B0
//   NS = 3:  A0 B0 + A0 B1 + A1 B0 + A0 B2 + A1 B1 + A2 B0
// written to W[z][n][m] (float2, column-major, ld = m), or, with a single
// split (S == 1) and C given, into the result C (element (i, j) at
// C[j ldc + i]; cdouble: C is complex128; accumulate: C += D; upper: only
// i <= j formed, 2: the other triangle filled with its conjugate).
// A CTA runs the tiles blockIdx.x, + gridDim.x, ... of the (split, row block,
// column block) list, the column block fastest: the CTAs that share a row block
// of a tall A run together, so that A comes from DRAM once, and the products of
// a CTA's next tile run while its epilogue writes the last one.  (betaNL D P of 64
// atoms, 160 bands 118 -> 63 us against one tile a CTA, row blocks fastest, of
// 216 atoms, 480 bands 1.51 -> 1.07 ms, there bound by the tensor pipe at 57 % of
// its rate; Q U of 480 bands 1.36 -> 1.27 ms.)
template <int NS, int BN>
__global__ void __launch_bounds__(THREADS, 1)
k_umma_gemm(const __grid_constant__ CUtensorMap tA0, const __grid_constant__ CUtensorMap tA1,
            const __grid_constant__ CUtensorMap tA2, const __grid_constant__ CUtensorMap tB0,
            const __grid_constant__ CUtensorMap tB1, const __grid_constant__ CUtensorMap tB2, int M, int N, int KB,
            int kb_per, float2 *__restrict__ W, int *__restrict__ err, int upper, int lolo, void *__restrict__ C,
            int64_t ldc, int cdouble, int accumulate, int S) {
    using CF = Cfg<NS, BN>;
    constexpr int STAGES = CF::STAGES;
    constexpr int STAGE_BYTES = CF::STAGE_BYTES;
    constexpr int TB = CF::TILE_B_BYTES;
    constexpr int TA = TILE_A_BYTES;
    const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN, tiles = mt * nt * S;
    // upper: C = Z^H W is Hermitian and only its upper triangle is read; a
    // tile whose rows all lie below its columns is skipped (with one tile a CTA
    // before any barrier or TMEM allocation)
    auto skipped = [&](int t) { return upper && (t / nt % mt) * BM > (t % nt) * BN + BN - 1; };
    if ((int)gridDim.x >= tiles && skipped(blockIdx.x)) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars *bars = reinterpret_cast<Bars *>(smem + (size_t)STAGES * STAGE_BYTES + CF::E_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the tile's k-blocks [kb0, kb0 + count)
    auto first_kb = [&](int t) { return t / (nt * mt) * kb_per; };
    auto count_kb = [&](int t) { return max(0, min(KB - first_kb(t), kb_per)); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&bars->full[s], 1);
            mbar_init(&bars->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bars->tfull[b], 1);
            mbar_init(&bars->tempty[b], 8);   // one arrival per epilogue warp
        }
        bars->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&bars->tmem_base)),
                     "r"(CF::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = bars->tmem_base;   // columns: [pair 0: Re, Im][pair 1: Re, Im], ACC each

    if (warp == 0 && lane == 0) {
        // ---------------- TMA producer
        int i = 0;   // k-blocks of all tiles so far
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            if (skipped(t)) continue;
            const int m0 = (t / nt % mt) * BM, n0 = (t % nt) * BN, kb0 = first_kb(t), nkb = count_kb(t);
            for (int k = 0; k < nkb; ++k, ++i) {
                const int s = i % STAGES;
                const uint32_t ph = (uint32_t)((i / STAGES) & 1);
                if (!mbar_wait(&bars->empty[s], ph ^ 1)) {
                    bars->failed = 1;
                    ok = false;
                    break;
                }
                unsigned char *st = smem + (size_t)s * STAGE_BYTES;
                mbar_expect_tx(&bars->full[s], STAGE_BYTES);
                const int kc = (kb0 + k) * BK;
                // stage layout: A pieces 0..NS-1, then B pieces 0..NS-1
                tma_load_2d(st, &tA0, &bars->full[s], kc, m0);
                tma_load_2d(st + TA, &tA1, &bars->full[s], kc, m0);
                if constexpr (NS == 3) tma_load_2d(st + 2 * TA, &tA2, &bars->full[s], kc, m0);
                tma_load_2d(st + NS * TA, &tB0, &bars->full[s], kc, n0);
                tma_load_2d(st + NS * TA + TB, &tB1, &bars->full[s], kc, n0);
                if constexpr (NS == 3) tma_load_2d(st + NS * TA + 2 * TB, &tB2, &bars->full[s], kc, n0);
            }
        }
        // wait (bounded) for the loads still in flight before leaving
        for (int j = max(0, i - STAGES); j < i; ++j) {
            const int s = j % STAGES;
            if (!mbar_wait(&bars->full[s], (uint32_t)((j / STAGES) & 1))) bars->failed = 1;
        }
    } else if (warp == 1 && lane == 0) {
        // ---------------- MMA issuer: every k-block accumulates into a fresh
        // pair of TMEM tiles, the correction products first and the main
        // product last, so that the tensor core's truncating FP32 accumulation
        // touches each value only a few times; the epilogue sums the tiles
        // with round-to-nearest adds (chains of 2 to 8 k-blocks gain at most
        // 6 % and bias the Gram diagonal by -6e-7 to -3e-6, one by -1e-7)
        int nkb = 0;   // of all tiles
        for (int t = blockIdx.x; t < tiles; t += gridDim.x)
            if (!skipped(t)) nkb += count_kb(t);
        for (int i = 0; i < nkb; ++i) {
            const int s = i % STAGES;
            const uint32_t ph = (uint32_t)((i / STAGES) & 1);
            const int b = i & 1;
            const uint32_t tu = (uint32_t)((i >> 1) & 1);
            if (!mbar_wait(&bars->tempty[b], tu ^ 1) || !mbar_wait(&bars->full[s], ph)) {
                bars->failed = 1;
                break;
            }
            fence_after();
            const uint32_t base = su32(smem + (size_t)s * STAGE_BYTES);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const uint32_t d = tmem + (uint32_t)((2 * b + part) * CF::ACC);
                // 16-value step kk of A (0, 1: Re, 2, 3: Im) against kk of B for
                // Re C, against the other half for Im C (Zi Wr negated)
                auto da = [&](int q, int kk) { return sdesc(base + q * TA + kk * 32); };
                auto db = [&](int q, int kk) { return sdesc(base + NS * TA + q * TB + (part ? kk ^ 2 : kk) * 32); };
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) {
                    const uint32_t ID = CF::IDESC | (part && kk >= 2 ? CF::NEG : 0u);
                    // lolo (two pieces, A and B the same block): the lo*lo term
                    // too, whose omission would bias every |z|^2 on the diagonal low
                    if (NS == 2 && lolo) mma_bf16(d, da(1, kk), db(1, kk), ID, kk > 0 ? 1u : 0u);
                    mma_bf16(d, da(0, kk), db(1, kk), ID, (kk > 0 || (NS == 2 && lolo)) ? 1u : 0u);
                    mma_bf16(d, da(1, kk), db(0, kk), ID, 1u);
                    if constexpr (NS == 3) {
                        mma_bf16(d, da(0, kk), db(2, kk), ID, 1u);
                        mma_bf16(d, da(1, kk), db(1, kk), ID, 1u);
                        mma_bf16(d, da(2, kk), db(0, kk), ID, 1u);
                    }
                }
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                    mma_bf16(d, da(0, kk), db(0, kk), CF::IDESC | (part && kk >= 2 ? CF::NEG : 0u), 1u);
            }
            mma_commit(&bars->empty[s]);
            mma_commit(&bars->tfull[b]);
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: warps 2..5 Re C, 6..9 Im C; TMEM lanes
        // [32q, 32q+32) (q = warp mod 4) -> rows m0 + 32q + lane, the k-blocks'
        // tiles summed in registers
        const int q = warp & 3, part = warp >= 6 ? 1 : 0;
        const int ml = 32 * q + lane;
        const bool direct = S == 1 && C;
        bool ok = true;
        int it = 0;   // k-blocks of all tiles so far
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            if (skipped(t)) continue;
            const int m0 = (t / nt % mt) * BM, n0 = (t % nt) * BN, nkb = count_kb(t);
            // the values to add to, on their way to L2 while the products run
            // (betaNL P of 216 atoms took 1.51 ms with plain loads at the end)
            if (direct && accumulate) {
                const int es = cdouble ? 16 : 8, rows = 128 / es, lines = BM / rows;
                for (int e = threadIdx.x - 64; e < BN * lines; e += 256) {
                    const int n = n0 + e / lines, i = m0 + (e % lines) * rows;
                    if (n < N && i < M)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)C + ((size_t)n * ldc + i) * es));
                }
            }
            float acc[BN];
#pragma unroll
            for (int c = 0; c < BN; ++c) acc[c] = 0.f;
            for (int k = 0; k < nkb; ++k, ++it) {
                const int b = it & 1;
                const uint32_t tu = (uint32_t)((it >> 1) & 1);
                // (after a wait ran out: no more waits, but every barrier below)
                ok = ok && mbar_wait(&bars->tfull[b], tu);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                fence_after();
                const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)((2 * b + part) * CF::ACC);
                // two 16-column loads in flight
#pragma unroll
                for (int c = 0; c < BN / 16; c += 2) {
                    uint32_t r0[16], r1[16];
                    tmem_ld16(ta + 16 * c, r0);
                    if (c + 1 < BN / 16) tmem_ld16(ta + 16 * (c + 1), r1);
                    tmem_wait_ld();
#pragma unroll
                    for (int u = 0; u < 16; ++u) acc[16 * c + u] += __uint_as_float(r0[u]);
                    if (c + 1 < BN / 16) {
#pragma unroll
                        for (int u = 0; u < 16; ++u) acc[16 * (c + 1) + u] += __uint_as_float(r1[u]);
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->tempty[b]);
            }
            // through shared memory (with one tile a CTA maybe the stages: every
            // MMA has completed), so that complex values leave in runs along the rows
            float *T = reinterpret_cast<float *>(smem + (CF::OWN_E ? (size_t)STAGES * STAGE_BYTES : 0));
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += EC) {
                constexpr int LAST = BN % EC ? BN % EC : EC;
                const int cols = c0 + EC <= BN ? EC : LAST;
#pragma unroll
                for (int c = 0; c < EC; ++c)
                    if (c0 + c < BN) T[2 * (c * (BM + 1) + ml) + part] = acc[c0 + c];
                asm volatile("bar.sync 1, 256;" ::: "memory");   // the eight epilogue warps
                const float2 *T2 = reinterpret_cast<const float2 *>(T);
                if (!direct)
                    store_columns(W + (size_t)(t / (nt * mt)) * M * (size_t)N, M, T2, m0, n0 + c0, M, N, cols, false, false);
                else if (cdouble) {
                    store_columns((double2 *)C, ldc, T2, m0, n0 + c0, M, N, cols, accumulate != 0, upper != 0);
                    if constexpr (MIRROR_BN<BN>)
                        if (upper == 2) mirror_columns((double2 *)C, ldc, T2, m0, n0 + c0, N, cols, accumulate != 0);
                } else
                    store_columns((float2 *)C, ldc, T2, m0, n0 + c0, M, N, cols, accumulate != 0, upper != 0);
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
        }
        if (!ok) atomicExch(err, 2);
    }
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && bars->failed) atomicExch(err, 1);
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CF::TMEM_COLS));
    }
}

// ------------------------------------------------------------ prep kernels
__device__ __forceinline__ void split2(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}
// x = p[0] + p[1] (+ p[2]): successive BF16 roundings of the remainder
template <int NS> __device__ __forceinline__ void splitn(float x, __nv_bfloat16 *p) {
    p[0] = __float2bfloat16_rn(x);
    const float r = x - __bfloat162float(p[0]);
    p[1] = __float2bfloat16_rn(r);
    if constexpr (NS == 3) p[2] = __float2bfloat16_rn(r - __bfloat162float(p[1]));
}

// position of the real part of value k in an operand row (its imaginary part
// 32 further on)
__host__ __device__ constexpr int64_t kpos(int64_t k) { return (k >> 5) * 64 + (k & 31); }

// Operand rows from the columns of Z (K x m, complex, column-major, ld), one
// array of m rows per BF16 piece (pc[0..NS-1]); two values a thread.
template <typename CT, int NS>
__global__ void k_prep_tn(const CT *__restrict__ Z, int64_t ld, int64_t K, int m, int Kp, __nv_bfloat16 *__restrict__ p0,
                          __nv_bfloat16 *__restrict__ p1, __nv_bfloat16 *__restrict__ p2) {
    __nv_bfloat16 *pc[3] = {p0, p1, p2};
    for (int i = blockIdx.y; i < m; i += gridDim.y) {
        const CT *z = Z + (size_t)i * ld;
        for (int64_t k = 2 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); k < Kp / 2;
             k += 2 * (int64_t)gridDim.x * blockDim.x) {
            float re[2], im[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const bool in = k + u < K;
                re[u] = in ? (float)z[k + u].x : 0.f;
                im[u] = in ? (float)z[k + u].y : 0.f;
            }
            __nv_bfloat16 a[2][3], c[2][3];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                splitn<NS>(re[u], a[u]);
                splitn<NS>(im[u], c[u]);
            }
            const size_t o = (size_t)i * Kp + kpos(k);
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                *reinterpret_cast<__nv_bfloat162 *>(pc[q] + o) = __nv_bfloat162(a[0][q], a[1][q]);
                *reinterpret_cast<__nv_bfloat162 *>(pc[q] + o + 32) = __nv_bfloat162(c[0][q], c[1][q]);
            }
        }
    }
}

// Operand rows for Z = A^H, A (M x k complex, column-major, lda): row g = [Re,
// Im] of conj(A[g, :]) = [Ar, -Ai], zero past k.  A 32 x 32 tile is transposed
// through shared memory: A is read along g, and a warp writes the 128-byte
// block of one row.
template <typename CT>
__global__ void k_prep_nn_a(const CT *__restrict__ A, int64_t lda, int64_t M, int k, int Kp, __nv_bfloat16 *__restrict__ hi,
                            __nv_bfloat16 *__restrict__ lo) {
    __shared__ float2 tile[32][33];
    const int64_t g0 = (int64_t)blockIdx.x * 32;
    const int l0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const int l = l0 + r;
        const int64_t g = g0 + tx;
        float2 v = make_float2(0.f, 0.f);
        if (l < k && g < M) v = make_float2((float)A[(size_t)l * lda + g].x, (float)A[(size_t)l * lda + g].y);
        tile[r][tx] = v;  // tile[l][g]
    }
    __syncthreads();
    // lanes 0..15: real parts of l0 + 2 lane, + 1; lanes 16..31: minus the imaginary parts
    const int l2 = 2 * (tx & 15);
    for (int r = ty; r < 32; r += 8) {
        const int64_t g = g0 + r;
        if (g >= M) continue;
        const float2 u = tile[l2][r], v = tile[l2 + 1][r];
        __nv_bfloat16 a, b, c, d;
        split2(tx < 16 ? u.x : -u.y, a, b);
        split2(tx < 16 ? v.x : -v.y, c, d);
        const size_t o = (size_t)g * Kp + (size_t)l0 * 2 + 2 * tx;
        *reinterpret_cast<__nv_bfloat162 *>(hi + o) = __nv_bfloat162(a, c);
        *reinterpret_cast<__nv_bfloat162 *>(lo + o) = __nv_bfloat162(b, d);
    }
}

// C (m x n complex, ldc) (+)= sum_z W[z][j][i].  upper: 1 = only i <= j is
// formed and written, 2 = only i <= j was formed (Z^H Z) and the other
// triangle gets its conjugate.
template <typename CT>
__device__ __forceinline__ void put_sum(CT *C, int64_t ldc, size_t i, size_t j, double re, double im, int accumulate, int upper) {
    auto put = [&](CT *p, double y) {
        p->x = accumulate ? re + (double)p->x : re;
        p->y = accumulate ? y + (double)p->y : y;
    };
    put(C + j * ldc + i, im);
    if (upper == 2 && i < j) put(C + i * ldc + j, -im);
}
template <typename CT>
__global__ void k_finalize(const float2 *__restrict__ W, int S, int m, int n, CT *__restrict__ C, int64_t ldc, int accumulate,
                           int upper) {
    const size_t total = (size_t)m * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t j = t / m, i = t - j * m;
        if (upper && i > j) continue;
        double re = 0.0, im = 0.0;
#pragma unroll 4
        for (int z = 0; z < S; ++z) {
            const float2 w = W[(size_t)z * total + t];
            re += (double)w.x;
            im += (double)w.y;
        }
        put_sum(C, ldc, i, j, re, im, accumulate, upper);
    }
}
// The same with eight lanes to an element, for many parts and few elements: 8 x 8
// values in 64 parts 17 us with one thread an element, 240 x 240 (one triangle) in
// 47 parts 16 us against 10; 480 x 480 in 9 parts 6.5, here slower.
template <typename CT>
__global__ void k_finalize8(const float2 *__restrict__ W, int S, int m, int n, CT *__restrict__ C, int64_t ldc, int accumulate,
                            int upper) {
    const size_t total = (size_t)m * n;
    const int l8 = threadIdx.x & 7;
    for (size_t t0 = (blockIdx.x * (size_t)blockDim.x + (threadIdx.x & ~31)) >> 3; t0 < total;
         t0 += ((size_t)gridDim.x * blockDim.x) >> 3) {
        const size_t t = t0 + ((threadIdx.x & 31) >> 3), j = t / m, i = t - j * m;
        const bool in = t < total && !(upper && i > j);
        double re = 0.0, im = 0.0;
        if (in) {
#pragma unroll 4
            for (int z = l8; z < S; z += 8) {
                const float2 w = W[(size_t)z * total + t];
                re += (double)w.x;
                im += (double)w.y;
            }
        }
        for (int o = 4; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (in && l8 == 0) put_sum(C, ldc, i, j, re, im, accumulate, upper);
    }
}

// The operand of betaNL (D P) straight from the split sums W of
// P = betaNL' psi: row b = [Re, Im] of sum_j D[i][j] sum_z W[z][b][j] along i,
// two BF16 pieces, zero past nbeta.  One pass where finalize, D P and the
// operand's own prep pass were three launches (about 4 us each).
__global__ void k_dcsr_prep(const float2 *__restrict__ W, int S, int nbeta, int nb, const int *__restrict__ rowptr,
                            const int *__restrict__ col, const double *__restrict__ val, int Kp,
                            __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo) {
    const int kp2 = Kp / 2, l8 = threadIdx.x & 7;   // eight lanes share an element's splits
    const size_t total = (size_t)kp2 * nb, wz = (size_t)nbeta * nb;
    for (size_t t0 = (blockIdx.x * (size_t)blockDim.x + (threadIdx.x & ~31)) >> 3; t0 < total;
         t0 += ((size_t)gridDim.x * blockDim.x) >> 3) {
        const size_t t = t0 + ((threadIdx.x & 31) >> 3);
        const int b = (int)(t / kp2), i = (int)(t - (size_t)b * kp2);
        double re = 0.0, im = 0.0;
        if (t < total && i < nbeta)
            for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
                const float2 *w = W + (size_t)b * nbeta + col[e];
                double pr = 0.0, pi = 0.0;
#pragma unroll 4
                for (int z = l8; z < S; z += 8) {
                    const float2 v = w[z * wz];
                    pr += (double)v.x;
                    pi += (double)v.y;
                }
                re += val[e] * pr;
                im += val[e] * pi;
            }
        for (int o = 4; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (t >= total || l8) continue;
        __nv_bfloat16 a[2], c[2];
        splitn<2>((float)re, a);
        splitn<2>((float)im, c);
        const size_t o = (size_t)b * Kp + kpos(i);
        hi[o] = a[0];
        hi[o + 32] = c[0];
        lo[o] = a[1];
        lo[o + 32] = c[1];
    }
}

// ------------------------------------------------------------- host side
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

cudaError_t get_encoder() {
    if (g_encode) return cudaSuccess;
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    return cudaSuccess;
}

// rows of Kp BF16 values
cudaError_t make_map(CUtensorMap *map, const void *base, int64_t rows, int Kp, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)Kp * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

int blocks_for(size_t total) {
    size_t b = (total + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    return b < 1 ? 1 : (int)b;
}

}  // namespace umma

using namespace umma;

int umma_kpad(int64_t K) { return (int)(((2 * K + BK - 1) / BK) * BK); }

size_t umma_operand_bytes(int64_t rows, int64_t K) { return (size_t)rows * umma_kpad(K) * 2 * 2; }

template <typename CT>
cudaError_t umma_prep_tn(const void *Z, int64_t ld, int64_t K, int m, UmmaOperand &op, cudaStream_t st) {
    op.rows = m;
    op.Kp = umma_kpad(K);
    dim3 grid((unsigned)std::min<int64_t>((op.Kp / 4 + 255) / 256, 64), (unsigned)std::min(m, 65535));
    if (op.lo2)
        k_prep_tn<CT, 3><<<grid, 256, 0, st>>>((const CT *)Z, ld, K, m, op.Kp, op.hi, op.lo, op.lo2);
    else
        k_prep_tn<CT, 2><<<grid, 256, 0, st>>>((const CT *)Z, ld, K, m, op.Kp, op.hi, op.lo, nullptr);
    return cudaGetLastError();
}

template <typename CT>
cudaError_t umma_prep_nn_a(const void *A, int64_t lda, int64_t M, int k, UmmaOperand &op, cudaStream_t st) {
    op.rows = M;
    op.Kp = umma_kpad(k);
    dim3 grid((unsigned)((M + 31) / 32), (k + 31) / 32);
    k_prep_nn_a<CT><<<grid, 256, 0, st>>>((const CT *)A, lda, M, k, op.Kp, op.hi, op.lo);
    return cudaGetLastError();
}

// Tile width and split-K count of a product of M x N complex values: the pair with
// the shortest modelled time, in units of about 1.2 us.  One CTA fits on an SM (222 KB
// of shared memory), so the active tiles (those on or above the diagonal for a
// Hermitian product) x splits run in waves of 148; a k-block takes 0.73 to 0.83
// whatever the tile's width (the chain TMA, MMA, TMEM read), a tile 1.8 for its
// pipeline and 0.23 for each 32 columns of its epilogue; split sums take a launch and
// their trip through memory.  Splits: as many as fill whole waves, or as the split
// sums' cost allows.  The numbers are a fit to 176 products (1 to 1440 columns, K =
// 62 to 80,000) with each width and 5 to 15 split counts measured: the choice is 0.6 %
// from the best of a product on average.  The width with the least padding and at
// most 64 splits was up to 65 % off (8 x 8 values over 80,000: 68 us in 64 parts, 41
// in 148; 100 x 100 over 200: 28.8 us in one tile, 19.2 in four narrow ones x 7).
// Accuracy does not depend on either: every k-block is its own accumulation chain in
// TMEM.
UmmaPlan umma_plan(int64_t M, int N, int Kp, int splits, int upper) {
    const int KB = Kp / BK, mt = (int)((M + BM - 1) / BM);
    UmmaPlan best{128, 1, 1, 0};
    double tbest = 1e300;
    for (int bn : {128, 96, 80, 64, 32}) {
        if (bn > 32 && N <= (bn > 96 ? 96 : bn > 64 ? 64 : 32)) continue;   // a narrower tile holds all columns
        const int nt = (N + bn - 1) / bn;
        int active = mt * nt;
        if (upper) {
            active = 0;
            for (int c = 0; c < nt; ++c) active += std::min(mt, (c * bn + bn - 1) / BM + 1);
        }
        const double sum = 2.9e-6 * (double)M * (double)N;   // a split's values
        const int smax = splits > 0 ? std::min(splits, KB) : std::max(1, std::min(KB, std::max(64, 148 / active)));
        const int even = smax > 1 ? (int)std::sqrt(KB / sum) : 1;
        const int wmax = active > 64 ? 12 : 4;   // waves that the parts may fill
        for (int w = 0, last = 0; w <= wmax + 1; ++w) {
            int S = splits > 0 ? smax : w == 0 ? 1 : w > wmax ? even : (int)std::min<int64_t>((int64_t)148 * w / active, KB);
            S = std::max(1, std::min(S, smax));
            if (S == last) continue;
            last = S;
            const int per = (KB + S - 1) / S;
            if (splits <= 0) S = (KB + per - 1) / per;
            const double waves = (double)(((int64_t)active * S + 147) / 148);
            double t = waves * (per * (0.73 + 0.0008 * bn) + 1.8 + 0.23 * bn / 32.0);
            const bool two = S > 1 || (upper == 2 && bn == 128);   // passes
            if (two) t += 0.9 + S * sum;
            if (t < tbest * (1.0 - 1e-9)) {
                tbest = t;
                best = UmmaPlan{bn, S, two ? 2 : 1, (size_t)S * M * N * sizeof(float2)};
            }
            if (splits > 0) break;
        }
    }
    return best;
}

template <int NS, int BN>
static cudaError_t launch_umma(const CUtensorMap *mA, const CUtensorMap *mB, int tiles, int M, int n, int KB, int kb_per,
                               float *ws, int *err, int upper, int lolo, void *C, int64_t ldc, int cdouble, int accumulate,
                               int S, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_umma_gemm<NS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem_bytes<NS, BN>());
    if (e != cudaSuccess) return e;
    // one CTA fits on an SM; a Hermitian product's tiles, half of them skipped,
    // go out one a CTA
    const int grid = !Cfg<NS, BN>::OWN_E || upper ? tiles : std::min(tiles, 148);
    k_umma_gemm<NS, BN><<<grid, THREADS, smem_bytes<NS, BN>(), st>>>(mA[0], mA[1], mA[2], mB[0], mB[1], mB[2], M, n, KB,
                                                                      kb_per, (float2 *)ws, err, upper, lolo, C, ldc, cdouble,
                                                                      accumulate, S);
    return cudaGetLastError();
}

cudaError_t umma_dcsr_prep(const float *ws, int S, int nbeta, int nb, const int *rowptr, const int *col, const double *val,
                           UmmaOperand &op, cudaStream_t st) {
    op.rows = nb;
    op.Kp = umma_kpad(nbeta);
    k_dcsr_prep<<<blocks_for((size_t)op.Kp / 2 * nb * 8), 256, 0, st>>>((const float2 *)ws, S, nbeta, nb, rowptr, col, val, op.Kp, op.hi,
                                                                   op.lo);
    return cudaGetLastError();
}

template <typename CT>
cudaError_t umma_gemm(const UmmaPlan &plan, const UmmaOperand &A, const UmmaOperand &B, int m, int n, void *C, int64_t ldc,
                      int accumulate, float *ws, int *err, cudaStream_t st, int upper, int lolo) {
    cudaError_t e = get_encoder();
    if (e != cudaSuccess) return e;
    if (A.Kp != B.Kp || A.rows != m || B.rows != n) return cudaErrorInvalidValue;
    // three BF16 pieces only when both operands carry them
    const int ns = (A.lo2 && B.lo2) ? 3 : 2;
    const int bn = plan.bn;
    CUtensorMap mA[3], mB[3];
    const __nv_bfloat16 *pa[3] = {A.hi, A.lo, ns == 3 ? A.lo2 : A.lo};
    const __nv_bfloat16 *pb[3] = {B.hi, B.lo, ns == 3 ? B.lo2 : B.lo};
    for (int q = 0; q < 3; ++q) {
        if ((e = make_map(&mA[q], pa[q], A.rows, A.Kp, BM)) != cudaSuccess) return e;
        if ((e = make_map(&mB[q], pb[q], B.rows, B.Kp, bn)) != cudaSuccess) return e;
    }
    const int KB = A.Kp / BK;
    const int S = plan.S;
    const int kb_per = (KB + S - 1) / S;
    const int tiles = (int)((A.rows + BM - 1) / BM) * ((n + bn - 1) / bn) * S;
    // one split: the epilogue writes or adds into C itself, no workspace pass
    const int cd = sizeof(CT) == 16 ? 1 : 0;
    void *Cd = plan.passes == 1 ? C : nullptr;
    e = cudaErrorInvalidValue;
#define PW_U(BN)                                                                                                     \
    if (bn == BN)                                                                                                    \
        e = ns == 3 ? launch_umma<3, BN>(mA, mB, tiles, m, n, KB, kb_per, ws, err, upper, 0, Cd, ldc, cd, accumulate, S, st) \
                    : launch_umma<2, BN>(mA, mB, tiles, m, n, KB, kb_per, ws, err, upper, lolo, Cd, ldc, cd, accumulate, S, st);
    PW_U(128)
    PW_U(96)
    PW_U(80)
    PW_U(64)
    PW_U(32)
#undef PW_U
    if (e != cudaSuccess || Cd || !C) return e;
    const size_t total = (size_t)m * n;
    if (S >= 16 && total <= 65536)
        k_finalize8<CT><<<blocks_for(total * 8), 256, 0, st>>>((const float2 *)ws, S, m, n, (CT *)C, ldc, accumulate, upper);
    else
        k_finalize<CT><<<blocks_for(total), 256, 0, st>>>((const float2 *)ws, S, m, n, (CT *)C, ldc, accumulate, upper);
    return cudaGetLastError();
}

template cudaError_t umma_prep_tn<float2>(const void *, int64_t, int64_t, int, UmmaOperand &, cudaStream_t);
template cudaError_t umma_prep_tn<double2>(const void *, int64_t, int64_t, int, UmmaOperand &, cudaStream_t);
template cudaError_t umma_prep_nn_a<float2>(const void *, int64_t, int64_t, int, UmmaOperand &, cudaStream_t);
template cudaError_t umma_gemm<float2>(const UmmaPlan &, const UmmaOperand &, const UmmaOperand &, int, int, void *, int64_t,
                                       int, float *, int *, cudaStream_t, int, int);
template cudaError_t umma_gemm<double2>(const UmmaPlan &, const UmmaOperand &, const UmmaOperand &, int, int, void *, int64_t,
                                        int, float *, int *, cudaStream_t, int, int);

}  // namespace pwk
