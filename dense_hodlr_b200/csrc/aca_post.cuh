// Post-processing of one compressed block (src/lowRank.cpp:250-277), shared
// by the ACA kernels: zero blocks, and blocks whose loop ran to full rank,
// which are stored exactly (W = block, V = I or W = I, V = block^T).
#pragma once

#include "common.cuh"

// Every thread of the block's CTAs; this CTA owns rows [i_lo, i_hi) of W and
// rows [j_lo, j_hi) of V, and `nt` threads share them.  status must be
// ACA_POST on entry; *rank and the returned status are those of the block.
template <typename T>
__device__ int aca_post_process(const AcaBlock& B, const EntrySrc& S, T* BW, T* BV, int64_t ld,
                                int k, int i_lo, int i_hi, int j_lo, int j_hi, int nt,
                                int* rank) {
  const int tid = threadIdx.x, m = B.m, n = B.n, ub = min(m, n);
  *rank = k;
  if (k == 0) {
    for (int i = i_lo + tid; i < i_hi; i += nt) BW[i] = (T)0;
    for (int j = j_lo + tid; j < j_hi; j += nt) BV[j] = (T)0;
    *rank = 1;
    return ACA_DONE;
  }
  if (k < ub - 1) return ACA_DONE;
  const int full = (n <= m) ? n : m;
  *rank = full;
  if (B.kcap < full) return ACA_NEED_CAP_POST;  // the full representation needs more columns
  if (n <= m) {                                 // W = block (m x n), V = I_n
    for (int l = 0; l < n; ++l) {
      double xc[3] = {0.0, 0.0, 0.0};
      if (!S.dense) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (d < S.kp.dim) xc[d] = __ldg(S.pts + d * S.ld + B.c0 + l);
      }
      for (int i = i_lo + tid; i < i_hi; i += nt)
        BW[i + (int64_t)l * ld] = (T)src_entry_xj(S, xc, B.r0 + i, B.c0 + l);
      for (int j = j_lo + tid; j < j_hi; j += nt)
        BV[j + (int64_t)l * ld] = (T)((j == l) ? 1.0 : 0.0);
    }
  } else {  // W = I_m, V = block^T (n x m)
    for (int l = 0; l < m; ++l) {
      double xr[3] = {0.0, 0.0, 0.0};
      if (!S.dense) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (d < S.kp.dim) xr[d] = __ldg(S.pts + d * S.ld + B.r0 + l);
      }
      for (int j = j_lo + tid; j < j_hi; j += nt)
        BV[j + (int64_t)l * ld] = (T)src_entry_xi(S, xr, B.r0 + l, B.c0 + j);
      for (int i = i_lo + tid; i < i_hi; i += nt)
        BW[i + (int64_t)l * ld] = (T)((i == l) ? 1.0 : 0.0);
    }
  }
  return ACA_DONE;
}
