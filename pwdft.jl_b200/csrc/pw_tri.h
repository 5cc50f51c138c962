// Who takes part in which step of the cluster tridiagonalisation (k_tridiag_c
// in pw_eig.cu): columns 1 .. n-1 of an n x n matrix go round-robin to the
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

}  // namespace eig
}  // namespace pwk
#undef PW_TRI_HD
