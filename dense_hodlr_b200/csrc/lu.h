// Batched LU interfaces (lu.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hodlr_internal.h"

struct LeafLULaunch {
  const int* leaf_min;
  const int* leaf_size;
  const int64_t* lu_off;  // offset of each leaf's s x s LU (and tri_elems) in `lu`
  double* lu;
  int* perm;              // length N: row permutation of each leaf, local indices
  EntrySrc src;
  unsigned* err;
  // optional: the assembled leaf blocks before factoring, leaf (r0, s) at
  // a_copy[r0 + i + j * lda_copy] (i, j < s)
  double* a_copy;
  int64_t lda_copy;
};

struct LeafSolveLaunch {
  const int* leaf_min;
  const int* leaf_size;
  const int64_t* lu_off;
  const double* lu;
  const int* perm;
  double* X;     // N x ncols panel, column-major
  int64_t ldx;
  int ncols;
  unsigned* err;  // DEV_ERR_INDEX: a permutation entry outside its leaf
};

struct SchurNode {
  int kb, kt;       // ranks of the bottom / top off-diagonal blocks
  int coff;         // number of ancestor columns (Schur right-hand sides)
  // unknown order of the capacitance system: 0 [bottom rank; top rank], the
  // Schur matrix of recLU (src/HODLR_Matrix.cpp:663-670); 1 [top; bottom],
  // the perturbI matrix I + VT U of recSM (src/perturbI.cpp:28-38)
  int order;
  int64_t s_off;    // S (sd x sd) offset
  int64_t z_off;    // Z (sd x zcols) offset
  int64_t r_off;    // right-hand sides (sd x cols) offset for the solve
  int64_t p_off;    // pivots offset
};

struct SchurLaunch {
  const SchurNode* nodes;
  double* S;
  const double* Z;
  double* R;
  int* piv;
  unsigned* err;
};

int leaf_lu_launch(const LeafLULaunch& L, int nleaves, int smax, cudaStream_t s);
int leaf_solve_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s);
// Capacitance matrices of at least this size are factored by the multi-CTA
// blocked LU (panel, swap + triangular solve, tiled trailing update per 32
// columns); smaller ones by one CTA each.  Factorization with the line at 192,
// 256, 384 and 416: N = 20011 2D 13.1, 13.1, 13.7, 13.7 ms, forest of 40 systems
// 21.5, 21.9, 22.0, 22.0 ms; more nodes than SMs favour one CTA each.
constexpr int SCHUR_BIG_SD = 256;
// sd: host array of the nodes' capacitance sizes (kb + kt), in node order.
int schur_factor_launch(const SchurLaunch& L, int nnodes, const int* sd, cudaStream_t s);
// Kernel launches schur_factor_launch makes for these sizes.
int schur_factor_launches(const int* sd, int nnodes);
// The factorization's solves y = S^-1 Z of the `coff` ancestor columns of every
// node (R at r_off, ld sd), in 32-row diagonal blocks: the LU is read once per 64
// columns and every SM is busy.  Nodes of less than 32 rows too: one register
// substitution each way instead of 16-column tiles in shared memory (factorization
// of 1D N = 1024 1.00 -> 0.89 ms, N = 4096 1.40 -> 1.35).  sd: host array of the nodes' sizes.  *launches:
// kernels launched.
int schur_solve_factor_launch(const SchurLaunch& L, int nnodes, const int* sd, int coff,
                              cudaStream_t s, int* launches);
