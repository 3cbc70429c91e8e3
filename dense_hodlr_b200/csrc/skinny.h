// Kernels of the direct solve for a few right-hand sides (skinny.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "lu.h"

// Rows of the diagonal blocks whose triangles' inverses are kept.
constexpr int TRI_NB = 64;
// Doubles behind an n x n packed LU for them: the inverses of block after block
// (column-major, leading dimension the block's rows), then an int2 a block, how
// its lower and its upper triangle are solved.
__host__ __device__ inline int64_t tri_elems(int n) {
  const int nb = (n + TRI_NB - 1) / TRI_NB, last = n - (nb - 1) * TRI_NB;
  return n > 0 ? (int64_t)(nb - 1) * TRI_NB * TRI_NB + last * last + nb : 0;
}
// Right-hand sides the row-major path takes (two tiles of 8).
constexpr int SKINNY_MAX = 16;
// Rows of V^T X that go through shared memory at a time; a panel's start may be
// odd, the rows are read in aligned pairs.
constexpr int TN_ROWS = 504;
constexpr int TN_COLS = 128;  // most columns of a V^T X item

// V^T X over rows [row0, row0 + rows): out = M x ncp row-major sums, V the
// item's first column at matrix row 0 (leading dimension ldp).
struct TnItem {
  const double* V;
  int row0, rows, M, pad;
  int64_t out;
};

// X[row0 .. row0 + rows) -= Y y, at most 128 rows; y = K x ncp row-major at z.
struct NnItem {
  const double* Y;
  int row0, rows, K, pad;
  int64_t z;
};

// One capacitance system: its two halves' V^T X sums by chunk, and where its
// solution goes.
struct CapNode {
  int n, pad;
  int64_t s_off, p_off;  // LU (and tri_elems), permutation
  int off[2], m[2], chunks[2];
  int64_t part[2];
  int64_t z;  // row-major result / column-major right-hand sides and result
};

// Most shared memory of a CTA: rows that a cluster of 8 cannot hold in so much of
// it are kept in device memory.
constexpr size_t CAP_SMEM = 227 * 1024;

struct CapLaunch {
  const CapNode* nodes = nullptr;
  const double* S = nullptr;
  const int* perm = nullptr;
  const double* part = nullptr;
  double* z = nullptr;
  double* big = nullptr;  // cap_big_elems doubles, or null when that is 0
  size_t smem_limit = CAP_SMEM;
};

// Column tiles of 8 a launch carries per CTA: 1 or 2.
inline int skinny_tiles(int nrhs) { return nrhs <= 8 ? 1 : 2; }

// Memory a launch needs for systems whose rows do not fit the shared memory of
// a cluster (doubles; 0: they fit).
int64_t cap_big_elems(int nnodes, int nrhs, int max_sd, size_t limit);

// The inverses of the triangles of every TRI_NB diagonal block of the packed LUs
// (n x n at off, column-major, tri_elems(n) doubles behind each).
int tri_invert_leaves_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s);
// The same for the nodes' capacitance LUs, and their interchanges as
// permutations: perm[i] = row of the right-hand side that becomes row i.
int tri_invert_nodes_launch(const SchurLaunch& L, int* perm, int nnodes, int max_sd,
                            cudaStream_t s);
// X[leaf rows] <- U^-1 L^-1 P X.
int leaf_apply_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s);
int skinny_tn_launch(const TnItem* items, int count, const double* X, int64_t ldx, int nrhs,
                     int64_t ldv, double* part, cudaStream_t s);
int skinny_nn_launch(const NnItem* items, int count, double* X, int64_t ldx, int nrhs, int64_t ldy,
                     const double* z, cudaStream_t s);
// y = S^-1 r per node: r summed from the chunks' partials, y row-major
// (parts), or both column-major in z, n x nrhs at the node's z.
int cap_solve_launch(const CapLaunch& L, int nnodes, int nrhs, int max_sd, bool parts,
                     unsigned* err, cudaStream_t s);
