// The tridiagonalisation's host and protocol arithmetic (kernels in pw_eig.cu).
//
// Who takes part in which step of the cluster kernel (k_tridiag_c): columns 1 .. n-1 of an n x n matrix go round-robin to the
// TRC CTAs of the cluster, column i to rank (i - 1) mod TRC.
//
// In step j the owners of the columns i > j exchange one pair a column.  A rank
// takes part in the steps j < tri_steps(n, rank), its last column: it publishes
// in each of them, and it is sent to in these and no others.  Every rank that is
// sent to in step j + 2 therefore published in step j + 1, after it had read
// step j, and nobody publishes step j + 2 before having everyone's step j + 1:
// two exchange buffers and two mbarriers are enough.  (A rank that went on
// receiving after its last column would hold nobody back: two steps late, it would
// find step j + 2 in step j's buffer, and the bytes of both in one phase.)
#pragma once

#ifdef __CUDACC__
#define PW_TRI_HD __host__ __device__ __forceinline__
#else
#define PW_TRI_HD inline
#endif

namespace pwk {
namespace eig {

constexpr int TRC = 16;   // CTAs of the cluster

// steps that `rank` takes part in: its last column, 0 if it owns none
PW_TRI_HD int tri_steps(int n, int rank) { return rank > n - 2 ? 0 : 1 + rank + (n - 2 - rank) / TRC * TRC; }
// the owner of column n - 1: takes part in every step
PW_TRI_HD int tri_last_rank(int n) { return n < 2 ? 0 : (n - 2) % TRC; }
// the rank that stores v_j: it owns column j + 1, so it takes part in step j
PW_TRI_HD int tri_writer(int j) { return j % TRC; }
// bytes that a participant of step j receives in it
PW_TRI_HD unsigned tri_bytes(int n, int j) { return (unsigned)(n - 1 - j) * 32u; }

// Columns of an order-n matrix that the grid's kernels take before the cluster
// (n - 1: all of them), and whether the register kernel k_tridiag_r does: up to n =
// 1024 if its CTAs are all resident at once, which its exchange and its cooperative
// launch need; the kernel with a grid barrier runs on as many CTAs as there are.
// r_ctas: CTAs of k_tridiag_r, r_resident: how many fit on the device; clusters:
// how many clusters of TRC CTAs do (0 on a device without TRC neighbouring SMs).
constexpr int TRI_NC = 256;   // columns that one cluster holds in registers
struct TriRoute {
    int jend;
    bool registers, cluster;
};
inline int tri_r_warps(int n) { return n > 512 ? 8 : 4; }
inline int tri_r_ctas(int n) { return n < 2 ? 1 : (n - 1 + tri_r_warps(n) - 1) / tri_r_warps(n); }
inline TriRoute tri_route(int n, int r_resident, int clusters) {
    TriRoute t;
    t.cluster = clusters > 0;
    t.jend = !t.cluster ? n - 1 : n > TRI_NC ? n - TRI_NC : 0;
    t.registers = n <= 1024 && tri_r_ctas(n) <= r_resident;
    return t;
}

}  // namespace eig
}  // namespace pwk
#undef PW_TRI_HD
