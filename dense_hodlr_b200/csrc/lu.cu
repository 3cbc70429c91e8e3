// Batched LU kernels of the recLU factorization and solve.
//
//  leaf_lu_kernel     assembles every leaf block from the kernel (or the dense
//                     input) and factors it with row partial pivoting, one CTA
//                     per leaf, all in shared memory.  Replaces the leaf path
//                     of storeLRinTree (src/HODLR_Matrix.cpp:303-312) and
//                     PartialPivLU(leafMatrix) (src/HODLR_Matrix.cpp:625).
//  leaf_solve_kernel  applies the leaf LU to a tile of a wide panel: the
//                     leafLU.solve of recLU_Factorize (src/HODLR_Matrix.cpp:626).
//  schur_form_kernel  builds S = [[I, V_b^T K_t^-1 U_t], [V_t^T K_b^-1 U_b, I]]
//                     (src/HODLR_Matrix.cpp:663-673) from the level product Z.
//  schur_lu_kernel    blocked partial-pivot LU of each node's S in place
//                     (SchurLU = PartialPivLU(S), src/HODLR_Matrix.cpp:675).
//  big_rhs_* kernels  y = S^-1 Z by the stored LU (src/HODLR_Matrix.cpp:682).
// The right-hand sides of a solve go through skinny.cu.
// Pivoting takes the first maximum |a| of the column, as PartialPivLU does.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "lu.h"

namespace cg = cooperative_groups;

namespace {

constexpr int LNT = 256;

// ------------------------------------------------------------- leaf LU
__global__ void __launch_bounds__(LNT) leaf_lu_kernel(LeafLULaunch L) {
  extern __shared__ double a[];  // s x s, leading dimension s | 1
  __shared__ int s_piv;
  const int leaf = blockIdx.x;
  const int r0 = L.leaf_min[leaf], s = L.leaf_size[leaf];
  const int lda = s | 1;
  const int tid = threadIdx.x;
  int* perm = L.perm + r0;  // final row permutation, local indices
  const EntrySrc S = src_for(L.src, r0);  // the kernel of this leaf's system
  // assemble
  for (int e = tid; e < s * s; e += LNT) {
    int i = e % s, j = e / s;
    a[j * lda + i] = src_entry(S, r0 + i, r0 + j);
  }
  for (int i = tid; i < s; i += LNT) perm[i] = i;
  __syncthreads();
  if (L.a_copy)
    for (int e = tid; e < s * s; e += LNT) {
      int i = e % s, j = e / s;
      L.a_copy[r0 + i + (int64_t)j * L.lda_copy] = a[j * lda + i];
    }
  bool singular = false, nonfinite = false;
  for (int p = 0; p < s; ++p) {
    // pivot search in column p, rows p..s-1, first maximum
    if (tid < 32) {
      double bv = -1.0;
      int bi = INT_MAX;
      for (int i = p + tid; i < s; i += 32) {
        double v = fabs(a[p * lda + i]);
        if (v > bv) {
          bv = v;
          bi = i;
        }
      }
      warp_argmax(bv, bi);
      if (tid == 0) s_piv = (bi == INT_MAX) ? p : bi;
    }
    __syncthreads();
    const int q = s_piv;
    if (q != p) {
      for (int j = tid; j < s; j += LNT) {
        double t = a[j * lda + p];
        a[j * lda + p] = a[j * lda + q];
        a[j * lda + q] = t;
      }
      if (tid == 0) {
        int t = perm[p];
        perm[p] = perm[q];
        perm[q] = t;
      }
    }
    __syncthreads();
    const double d = a[p * lda + p];
    if (d == 0.0) {
      singular = true;
      __syncthreads();
      continue;
    }
    if (!isfinite(d)) nonfinite = true;
    for (int i = p + 1 + tid; i < s; i += LNT) a[p * lda + i] = a[p * lda + i] / d;
    __syncthreads();
    // rank-1 update of the trailing block
    const int rem = s - p - 1;
    for (int e = tid; e < rem * rem; e += LNT) {
      int i = p + 1 + e % rem, j = p + 1 + e / rem;
      a[j * lda + i] = fma(-a[p * lda + i], a[j * lda + p], a[j * lda + i]);
    }
    __syncthreads();
  }
  double* out = L.lu + L.lu_off[leaf];
  for (int e = tid; e < s * s; e += LNT) {
    int i = e % s, j = e / s;
    out[(int64_t)j * s + i] = a[j * lda + i];
  }
  if (tid == 0) {
    if (singular) atomicOr(L.err, DEV_ERR_SINGULAR);
    if (nonfinite) atomicOr(L.err, DEV_ERR_NONFINITE);
  }
}

// ------------------------------------------------ blocked tile solves
// x <- U^-1 L^-1 x for `ncol` columns of a tile in shared memory (x[c*ldx+i]),
// where the unit-lower L and the upper U are read through `A(i, j)` (the
// packed LU of an n x n matrix).  Diagonal blocks of BS rows are solved by one
// thread per column; the rows below / above are updated by all threads.
constexpr int BS = 16;

struct SmemLU {
  const double* a;
  int lda;
  __device__ double operator()(int i, int j) const { return a[j * lda + i]; }
};

__device__ void lu_solve_tile(const SmemLU& A, int n, double* x, int ldx, int ncol) {
  const int tid = threadIdx.x, NT = blockDim.x;
  for (int b0 = 0; b0 < n; b0 += BS) {  // forward, unit lower
    const int be = min(n, b0 + BS);
    for (int c = tid; c < ncol; c += NT) {
      double* xc = x + c * ldx;
      for (int i = b0 + 1; i < be; ++i) {
        double t = xc[i];
        for (int p = b0; p < i; ++p) t = fma(-A(i, p), xc[p], t);
        xc[i] = t;
      }
    }
    __syncthreads();
    const int rem = n - be;
    for (int e = tid; e < rem * ncol; e += NT) {
      const int r = be + e % rem, c = e / rem;
      double* xc = x + c * ldx;
      double t = xc[r];
      for (int p = b0; p < be; ++p) t = fma(-A(r, p), xc[p], t);
      xc[r] = t;
    }
    __syncthreads();
  }
  for (int be = n; be > 0; be -= BS) {  // backward, upper
    const int b0 = max(0, be - BS);
    for (int c = tid; c < ncol; c += NT) {
      double* xc = x + c * ldx;
      for (int i = be - 1; i >= b0; --i) {
        double t = xc[i];
        for (int p = i + 1; p < be; ++p) t = fma(-A(i, p), xc[p], t);
        xc[i] = t / A(i, i);
      }
    }
    __syncthreads();
    for (int e = tid; e < b0 * ncol; e += NT) {
      const int r = e % b0, c = e / b0;
      double* xc = x + c * ldx;
      double t = xc[r];
      for (int p = b0; p < be; ++p) t = fma(-A(r, p), xc[p], t);
      xc[r] = t;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------- leaf solve
// X[leaf rows, c0 : c0+TC] <- U^-1 L^-1 P X.  One CTA per (leaf, column tile).
template <int TC>
__global__ void __launch_bounds__(LNT) leaf_solve_kernel(LeafSolveLaunch L) {
  extern __shared__ double sm[];
  const int leaf = blockIdx.y;
  const int c0 = blockIdx.x * TC;
  const int ncol = min(TC, L.ncols - c0);
  if (ncol <= 0) return;
  const int r0 = L.leaf_min[leaf], s = L.leaf_size[leaf];
  const int lda = s | 1;
  double* lu = sm;                    // s x s
  double* x = sm + (size_t)s * lda;   // s x TC, x[c * (s|1) + i]
  const int ldx = s | 1;
  const int tid = threadIdx.x;
  const double* g = L.lu + L.lu_off[leaf];
  for (int e = tid; e < s * s; e += LNT) {
    int i = e % s, j = e / s;
    lu[j * lda + i] = g[(int64_t)j * s + i];
  }
  const int* perm = L.perm + r0;
  for (int e = tid; e < s * ncol; e += LNT) {
    int i = e % s, c = e / s;
    const int pi = perm[i];
    if (pi < 0 || pi >= s) {  // never written by a valid leaf LU: skip and report
      if (L.err) atomicOr(L.err, DEV_ERR_INDEX | DEV_ERR_AT_LEAF_PERM);
      x[c * ldx + i] = 0.0;
      continue;
    }
    x[c * ldx + i] = L.X[(int64_t)(c0 + c) * L.ldx + r0 + pi];
  }
  __syncthreads();
  lu_solve_tile(SmemLU{lu, lda}, s, x, ldx, ncol);
  for (int e = tid; e < s * ncol; e += LNT) {
    int i = e % s, cc = e / s;
    L.X[(int64_t)(c0 + cc) * L.ldx + r0 + i] = x[cc * ldx + i];
  }
}

// ---------------------------------------------------------- Schur form
// S[node] (sd x sd, sd = kb + kt): identity blocks on the diagonal, the level
// products of Z on the off-diagonal blocks.  With n1 the size of the first
// unknown block (kb in recLU order, kt in recSM order), Z's rows follow the
// same order and its own-level columns start at coff: the upper-right block
// is Z[:n1, coff + (j - n1)], the lower-left Z[n1:, coff + j].
// CTA (node, y) fills every gridDim.y-th slice of the node's entries, so a
// large S is written by many CTAs.
__global__ void schur_form_kernel(SchurLaunch L) {
  const int node = blockIdx.x;
  const SchurNode N = L.nodes[node];
  const int sd = N.kb + N.kt;
  double* S = L.S + N.s_off;
  const double* Z = L.Z + N.z_off;  // sd x zcols, ld sd
  const int n1 = N.order ? N.kt : N.kb;
  for (int64_t e = threadIdx.x + (int64_t)blockIdx.y * blockDim.x; e < (int64_t)sd * sd;
       e += (int64_t)blockDim.x * gridDim.y) {
    int i = (int)(e % sd), j = (int)(e / sd);
    double v;
    if ((i < n1) == (j < n1))
      v = (i == j) ? 1.0 : 0.0;
    else if (i < n1)  // recLU: V_b^T K_t^-1 U_t; recSM: V_t^T K_b^-1 U_b
      v = Z[(int64_t)(N.coff + j - n1) * sd + i];
    else  // recLU: V_t^T K_b^-1 U_b; recSM: V_b^T K_t^-1 U_t
      v = Z[(int64_t)(N.coff + j) * sd + i];
    S[(int64_t)j * sd + i] = v;
  }
}

// ------------------------------------------------------ dense batched LU
// Blocked right-looking LU with row partial pivoting, S in global memory (L2
// resident).  The row interchanges of a panel are applied to the whole row, so the
// packed result and `piv` are those of an unblocked partial-pivot LU with the same
// pivot choices (LAPACK getrf convention).
constexpr int SNT = 512;

// One CTA factors columns [jlo, jhi) of the n x n matrix a (columns < jlo
// final, their interchanges already applied to columns >= jlo) in inner panels of
// pnb columns in shared memory: the pivots of those columns go to piv, their
// interchanges are applied to the columns of [jlo, jhi) only, and the columns
// >= jhi are not touched.  For panels of too many rows to be held in registers.
__device__ bool lu_columns(double* a, int n, int* piv, int jlo, int jhi, int pnb, double* pan,
                           double* red_v, int* red_i, int* lpiv) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  bool singular = false;
  for (int j0 = jlo; j0 < jhi; j0 += pnb) {
    const int nb = min(pnb, jhi - j0), rows = n - j0;
    for (int e = tid; e < rows * nb; e += SNT) {
      int r = e % rows, c = e / rows;
      pan[c * rows + r] = a[(int64_t)(j0 + c) * n + j0 + r];
    }
    __syncthreads();
    for (int c = 0; c < nb; ++c) {
      // pivot: first maximum |.| of panel column c, rows c..rows-1
      double bv = -1.0;
      int bi = INT_MAX;
      for (int r = c + tid; r < rows; r += SNT) {
        double v = fabs(pan[c * rows + r]);
        if (v > bv) {
          bv = v;
          bi = r;
        }
      }
      warp_argmax(bv, bi);
      if (lane == 0) {
        red_v[w] = bv;
        red_i[w] = bi;
      }
      __syncthreads();
      if (w == 0) {
        bv = lane < SNT / 32 ? red_v[lane] : -1.0;
        bi = lane < SNT / 32 ? red_i[lane] : INT_MAX;
        warp_argmax(bv, bi);
        if (lane == 0) lpiv[c] = (bi == INT_MAX) ? c : bi;
      }
      __syncthreads();
      const int q = lpiv[c];
      if (q != c)
        for (int cc = tid; cc < nb; cc += SNT) {
          double t = pan[cc * rows + c];
          pan[cc * rows + c] = pan[cc * rows + q];
          pan[cc * rows + q] = t;
        }
      __syncthreads();
      const double d = pan[c * rows + c];
      if (d == 0.0) {
        singular = true;
        continue;
      }
      for (int r = c + 1 + tid; r < rows; r += SNT) pan[c * rows + r] /= d;
      __syncthreads();
      const int rr = rows - c - 1, cols = nb - c - 1;
      for (int e = tid; e < rr * cols; e += SNT) {
        int r = c + 1 + e % rr, cc = c + 1 + e / rr;
        pan[cc * rows + r] = fma(-pan[c * rows + r], pan[cc * rows + c], pan[cc * rows + r]);
      }
      __syncthreads();
    }
    // panel back to global, pivots, interchanges in the other columns of the range
    for (int e = tid; e < rows * nb; e += SNT) {
      int r = e % rows, c = e / rows;
      a[(int64_t)(j0 + c) * n + j0 + r] = pan[c * rows + r];
    }
    if (tid < nb) piv[j0 + tid] = j0 + lpiv[tid];
    for (int col = jlo + tid; col < jhi; col += SNT) {
      if (col >= j0 && col < j0 + nb) continue;
      double* ac = a + (int64_t)col * n;
      for (int c = 0; c < nb; ++c) {
        const int q = lpiv[c];
        if (q != c) {
          double t = ac[j0 + c];
          ac[j0 + c] = ac[j0 + q];
          ac[j0 + q] = t;
        }
      }
    }
    __syncthreads();
    const int rest = n - j0 - nb;      // trailing rows
    const int crest = jhi - j0 - nb;   // trailing columns inside the range
    if (rest > 0 && crest > 0) {
      // U12 = L11^-1 A12, one thread per column
      for (int col = j0 + nb + tid; col < jhi; col += SNT) {
        double* ac = a + (int64_t)col * n + j0;
        for (int i = 1; i < nb; ++i) {
          double t = ac[i];
          for (int p = 0; p < i; ++p) t = fma(-pan[p * rows + i], ac[p], t);
          ac[i] = t;
        }
      }
      __syncthreads();
      // A22 -= L21 U12 with 4x4 register tiles
      const int tr = (rest + 3) / 4, tc = (crest + 3) / 4;
      for (int tt = tid; tt < tr * tc; tt += SNT) {
        const int ti = (tt % tr) * 4, tj = (tt / tr) * 4;
        double acc[4][4];
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[x][y] = 0.0;
        for (int p = 0; p < nb; ++p) {
          double l[4], u[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) l[x] = (ti + x < rest) ? pan[p * rows + nb + ti + x] : 0.0;
#pragma unroll
          for (int y = 0; y < 4; ++y)
            u[y] = (tj + y < crest) ? a[(int64_t)(j0 + nb + tj + y) * n + j0 + p] : 0.0;
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) acc[x][y] = fma(l[x], u[y], acc[x][y]);
        }
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          if (tj + y >= crest) continue;
          double* ac = a + (int64_t)(j0 + nb + tj + y) * n + j0 + nb + ti;
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (ti + x < rest) ac[x] -= acc[x][y];
        }
      }
      __syncthreads();
    }
  }
  return singular;
}

// ------------------------------------------------- panels in registers
// Columns [j0, j0 + nb), nb <= PW, of an n x n matrix, rows j0..: a row in each
// thread's registers, one CTA or a cluster (CL) of up to 8 for more than SNT rows.
// A column costs one barrier (and one of the cluster): every warp finds its first
// maximum with warp reductions on the bits of |a|, its owner puts the value, its
// position and the whole row into shared memory, and after the barrier all threads
// pick the best of the warps' candidates and read that row.  Rows do not move:
// each thread tracks the position its row would have after the interchanges and
// writes it back there.  The same pivots, interchanges and eliminations as with
// moved rows.
//
// Bound by that chain of PW reductions.  The panel in shared memory (three barriers
// more, divisions and the rank-1 update through shared memory) took about 3 us a
// column, in registers about 0.4 us:
// factorization of N = 20011 2D 18.5 -> 13.1 ms, of 16384 points on a sphere
// 62.8 -> 45.2 ms, of a forest of 40 systems 26.3 -> 21.9 ms.
constexpr int PW = 32;
struct PanelSmem {
  unsigned hi[2][SNT / 32], lo[2][SNT / 32];
  int pos[2][SNT / 32];
  double row[2][SNT / 32][PW];
  unsigned chi[2][8], clo[2][8];  // the cluster's candidates
  int cpos[2][8];
  double crow[2][8][PW];
};

// Index of the best candidate (largest |a| bits, then smallest position) among
// `count` slots, in every lane.
__device__ __forceinline__ int best_slot(const unsigned* hi, const unsigned* lo, const int* pos,
                                         int count, int* q) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned h = lane < count ? hi[lane] : 0u, l = lane < count ? lo[lane] : 0u;
  const int p = lane < count ? pos[lane] : INT_MAX;
  const unsigned mh = __reduce_max_sync(all, h);
  const unsigned ml = __reduce_max_sync(all, h == mh ? l : 0u);
  const bool c = lane < count && h == mh && l == ml;
  *q = __reduce_min_sync(all, c ? p : INT_MAX);
  return __ffs(__ballot_sync(all, c && p == *q)) - 1;
}

template <bool CL>
__device__ bool panel_in_registers(double* a, int n, int* piv, int j0, int nb, PanelSmem& sm) {
  const unsigned all = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int rank = 0, size = 1;
  if (CL) {
    rank = (int)cg::this_cluster().block_rank();
    size = (int)cg::this_cluster().num_blocks();
    // a CTA's shared memory may be written once it has started: waited for
    // before the first column's stores, behind the panel's loads
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  const int r = rank * SNT + tid;
  const bool live = r < n - j0;
  int pos = r;
  bool done = !live, singular = false;
  double x[PW];
#pragma unroll
  for (int c = 0; c < PW; ++c) x[c] = live && c < nb ? a[(int64_t)(j0 + c) * n + j0 + r] : 0.0;
#pragma unroll
  for (int c = 0; c < PW; ++c) {
    if (c < nb) {  // uniform
      const int buf = c & 1;  // read until the next column's barrier
      // a NaN is never larger than another value; rows in play have the top bit
      const double v = fabs(x[c]);
      const unsigned hi = done ? 0u : (v == v ? (unsigned)__double2hiint(v) : 0u) | 0x80000000u;
      const unsigned lo = !done && v == v ? (unsigned)__double2loint(v) : 0u;
      const unsigned mh = __reduce_max_sync(all, hi);
      const unsigned ml = __reduce_max_sync(all, hi == mh ? lo : 0u);
      const bool cand = !done && hi == mh && lo == ml;
      const int mp = __reduce_min_sync(all, cand ? pos : INT_MAX);
      if (mh == 0u) {
        if (lane == 0) {
          sm.hi[buf][w] = sm.lo[buf][w] = 0u;
          sm.pos[buf][w] = INT_MAX;
        }
      } else if (cand && pos == mp) {
        sm.hi[buf][w] = mh;
        sm.lo[buf][w] = ml;
        sm.pos[buf][w] = pos;
#pragma unroll
        for (int k = c & ~1; k < PW; k += 2)
          *reinterpret_cast<double2*>(&sm.row[buf][w][k]) = make_double2(x[k], x[k + 1]);
      }
      __syncthreads();
      int q;
      int b = best_slot(sm.hi[buf], sm.lo[buf], sm.pos[buf], SNT / 32, &q);
      const double* pr = sm.row[buf][b];
      if (CL) {
        if (c == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (w == 0)
          for (int o = 0; o < size; ++o) {
            PanelSmem* to = cg::this_cluster().map_shared_rank(&sm, o);
            to->crow[buf][rank][lane] = pr[lane];
            if (lane == 0) {
              to->chi[buf][rank] = sm.hi[buf][b];
              to->clo[buf][rank] = sm.lo[buf][b];
              to->cpos[buf][rank] = q;
            }
          }
        cg::this_cluster().sync();
        b = best_slot(sm.chi[buf], sm.clo[buf], sm.cpos[buf], size, &q);
        pr = sm.crow[buf][b];
      }
      if (r == 0) piv[j0 + c] = j0 + q;
      if (pos == q) {
        pos = c;
        done = true;
      } else if (pos == c) {
        pos = q;
      }
      const double d = pr[c];
      if (d == 0.0) {
        singular = true;
      } else if (!done) {
        const double l = x[c] / d;
        x[c] = l;
#pragma unroll
        for (int k = c + 1; k < PW; ++k) x[k] = fma(-l, pr[k], x[k]);
      }
    }
  }
  if (live) {
#pragma unroll
    for (int c = 0; c < PW; ++c)
      if (c < nb) a[(int64_t)(j0 + c) * n + j0 + pos] = x[c];
  }
  return singular;
}

// The interchanges piv[0..nb) (relative positions p <-> piv[p], p = 0, 1, ..) as
// moves: position i < nb receives row from[i], and position to[i] >= nb (or
// to[i] < nb: none) row i.  Run by one warp; false: not LU interchanges.
__device__ bool panel_moves(const int* piv, int j0, int nb, int rows, int* from, int* to) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int q = lane < nb ? piv[j0 + lane] - j0 : lane;
  const bool ok = __all_sync(all, q >= lane && (lane >= nb || q < rows));
  int t = lane, f = lane;
  for (int c = 0; c < nb; ++c) {
    const int qc = __shfl_sync(all, q, c);
    t = t == c ? qc : t == qc ? c : t;
  }
  for (int c = nb - 1; c >= 0; --c) {
    const int qc = __shfl_sync(all, q, c);
    f = f == c ? qc : f == qc ? c : f;
  }
  from[lane] = ok ? f : lane;
  to[lane] = ok ? t : lane;
  return ok;
}

// A column's part of a panel's interchanges: u[i] <- its rows at positions < nb,
// the displaced rows written below.  The caller writes u back.
__device__ __forceinline__ void gather_moved(double* ac, int nb, const int* from, const int* to,
                                             double (&u)[PW]) {
#pragma unroll
  for (int i = 0; i < PW; ++i) u[i] = i < nb ? ac[from[i]] : 0.0;
#pragma unroll 8
  for (int i = 0; i < nb; ++i)
    if (to[i] >= nb) ac[to[i]] = ac[i];
}

// u <- L11^-1 u, unit lower, rows in order
__device__ __forceinline__ void unit_lower_solve(const double (*l11)[PW], double (&u)[PW]) {
#pragma unroll
  for (int p = 0; p < PW - 1; ++p)
#pragma unroll
    for (int i = p + 1; i < PW; ++i) u[i] = fma(-l11[p][i], u[p], u[i]);
}

// D = A B for a warp: A 32 x 32 at as[p * lda + row], B 32 x 16 at bs[p * ldb + col],
// leading dimensions 4 mod 16 (no bank conflicts).  D[m][v] of lane (g, t): rows
// 8 m + g, columns 8 v + 2 t, + 1.
__device__ __forceinline__ void warp_tile(const double* as, int lda, const double* bs, int ldb,
                                          double (&acc)[4][2][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int v = 0; v < 2; ++v) acc[m][v][0] = acc[m][v][1] = 0.0;
#pragma unroll
  for (int k = 0; k < PW; k += 4) {
    double av[4], bv[2];
#pragma unroll
    for (int m = 0; m < 4; ++m) av[m] = as[(k + t) * lda + 8 * m + g];
#pragma unroll
    for (int v = 0; v < 2; ++v) bv[v] = bs[(k + t) * ldb + 8 * v + g];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int v = 0; v < 2; ++v)
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
            : "+d"(acc[m][v][0]), "+d"(acc[m][v][1])
            : "d"(av[m]), "d"(bv[v]));
  }
}

// rows or columns of a trailing block, padded for warp_tile
__host__ __device__ constexpr int tile_pitch(int m) { return (m + 31) / 32 * 32 + 4; }

// Whole LU of every node with sd < big_sd, one CTA per node (larger nodes are
// left to the multi-CTA path below): panels in registers, a column a thread for
// the interchanges and U12 = L11^-1 A12, A22 -= L21 U12 on the matrix
// instructions from shared memory.
__global__ void __launch_bounds__(SNT) schur_lu_kernel(SchurLaunch L, int big_sd) {
  extern __shared__ __align__(16) double dyn[];
  __shared__ __align__(16) PanelSmem sm;
  __shared__ __align__(16) double l11[PW][PW];
  __shared__ int from[PW], to[PW];
  const SchurNode N = L.nodes[blockIdx.x];
  const int n = N.kb + N.kt;
  if (n >= big_sd) return;
  double* a = L.S + N.s_off;
  int* piv = L.piv + N.p_off;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  bool singular = false;
  for (int j0 = 0; j0 < n; j0 += PW) {
    const int nb = min(PW, n - j0), rest = n - j0 - nb;
    singular |= panel_in_registers<false>(a, n, piv, j0, nb, sm);
    __syncthreads();  // the panel and its pivots, by this CTA
    if (w == 0) panel_moves(piv, j0, nb, n - j0, from, to);
    const int ld = tile_pitch(rest);
    double* ls = dyn;            // [PW][ld] L21
    double* us = dyn + PW * ld;  // [PW][ld] U12
    for (int e = tid; e < PW * PW; e += SNT) {
      const int i = e % PW, p = e / PW;
      l11[p][i] = i < nb && p < nb ? a[(int64_t)(j0 + p) * n + j0 + i] : 0.0;
    }
    if (rest > 0)
      for (int e = tid; e < PW * (ld - 4); e += SNT) {
        const int i = e % (ld - 4), p = e / (ld - 4);
        ls[p * ld + i] = i < rest && p < nb ? a[(int64_t)(j0 + p) * n + j0 + nb + i] : 0.0;
      }
    __syncthreads();
    for (int col = tid; col < n + (ld - 4 - rest); col += SNT) {
      if (col >= j0 && col < j0 + nb) continue;
      const int right = col - j0 - nb;  // column of U12; from n on: padding
      double u[PW];
      if (col < n) {
        double* ac = a + (int64_t)col * n + j0;
        gather_moved(ac, nb, from, to, u);
        if (right >= 0) unit_lower_solve(l11, u);
#pragma unroll
        for (int i = 0; i < PW; ++i)
          if (i < nb) ac[i] = u[i];
      }
      if (right >= 0 && rest > 0)
#pragma unroll
        for (int i = 0; i < PW; ++i) us[i * ld + right] = col < n ? u[i] : 0.0;
    }
    __syncthreads();
    if (rest <= 0) break;
    const int tr = (rest + 31) / 32, tc = (rest + 15) / 16;
    for (int tt = w; tt < tr * tc; tt += SNT / 32) {
      const int r0 = 32 * (tt % tr), c0 = 16 * (tt / tr);
      double acc[4][2][2];
      warp_tile(ls + r0, ld, us + c0, ld, acc);
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = c0 + 8 * v + 2 * t + e;
          double* ac = a + (int64_t)(j0 + nb + c) * n + j0 + nb;
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const int rr = r0 + 8 * m + g;
            if (c < rest && rr < rest) ac[rr] -= acc[m][v][e];
          }
        }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && singular) atomicOr(L.err, DEV_ERR_SINGULAR);
}

// ------------------------------------------- multi-CTA LU of large nodes
// Right-looking, outer panels of BNB columns.  Per panel j0, for every large
// node (its index in BigNodes): (1) the panel columns [j0, j0+BNB), in the
// registers of one CTA or of a cluster of up to 8 (512 rows each), above 4096 rows
// by one CTA through shared memory (lu_columns); (2) many CTAs apply the panel's
// interchanges to every other column and form U12 = L11^-1 A12 right of the panel;
// (3) A22 -= L21 U12 in 64 x 64 tiles over all SMs.  The pivot choices are the
// column-wise first maxima, as in the one-CTA kernel.
constexpr int BNB = PW;
constexpr int BIG_MAX = 1024;  // nodes per launch (kernel parameter: 4 KB)
struct BigNodes {
  int idx[BIG_MAX];
  int count;
};

template <bool CL>
__global__ void __launch_bounds__(SNT) panel_kernel(SchurLaunch L, BigNodes B, int j0) {
  __shared__ __align__(16) PanelSmem sm;
  const SchurNode N = L.nodes[B.idx[blockIdx.y]];
  const int n = N.kb + N.kt;
  if (j0 >= n) return;  // the whole cluster
  const bool singular = panel_in_registers<CL>(L.S + N.s_off, n, L.piv + N.p_off, j0,
                                               min(BNB, n - j0), sm);
  if (threadIdx.x == 0 && singular) atomicOr(L.err, DEV_ERR_SINGULAR);
}

// Panels of more rows than 8 CTAs' threads: through shared memory, one CTA.
__global__ void __launch_bounds__(SNT) big_panel_kernel(SchurLaunch L, BigNodes B, int j0, int pnb) {
  extern __shared__ double pan[];
  __shared__ double red_v[SNT / 32];
  __shared__ int red_i[SNT / 32];
  __shared__ int lpiv[64];
  const SchurNode N = L.nodes[B.idx[blockIdx.x]];
  const int n = N.kb + N.kt;
  if (j0 >= n) return;
  const bool singular = lu_columns(L.S + N.s_off, n, L.piv + N.p_off, j0, min(n, j0 + BNB), pnb,
                                   pan, red_v, red_i, lpiv);
  if (threadIdx.x == 0 && singular) atomicOr(L.err, DEV_ERR_SINGULAR);
}

// One thread per column outside the panel: the panel's interchanges as moves (32
// independent loads instead of a chain of swaps), then (right of the panel) the
// unit-lower solve with L11.
__global__ void __launch_bounds__(128) big_swap_trsm_kernel(SchurLaunch L, BigNodes B, int j0) {
  __shared__ __align__(16) double l11[PW][PW];
  __shared__ int from[PW], to[PW];
  const SchurNode N = L.nodes[B.idx[blockIdx.y]];
  const int n = N.kb + N.kt;
  if (j0 >= n) return;
  const int nb = min(BNB, n - j0);
  double* a = L.S + N.s_off;
  if (threadIdx.x < 32 && !panel_moves(L.piv + N.p_off, j0, nb, n - j0, from, to) &&
      threadIdx.x == 0)  // not LU interchanges: skipped and reported
    atomicOr(L.err, DEV_ERR_INDEX | DEV_ERR_AT_LU_SWAP);
  for (int e = threadIdx.x; e < PW * PW; e += blockDim.x) {
    const int i = e % PW, p = e / PW;
    l11[p][i] = (i < nb && p < nb) ? a[(int64_t)(j0 + p) * n + j0 + i] : 0.0;
  }
  __syncthreads();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n || (col >= j0 && col < j0 + nb)) return;
  double* ac = a + (int64_t)col * n + j0;
  double u[PW];
  gather_moved(ac, nb, from, to, u);
  if (col > j0) unit_lower_solve(l11, u);
#pragma unroll
  for (int i = 0; i < PW; ++i)
    if (i < nb) ac[i] = u[i];
}

// A22 -= L21 U12: CTA (ti, tj, node) owns a 64 x 64 tile, 256 threads with
// 4 x 4 outputs each; L21 and U12 tiles staged in shared memory.
constexpr int BT = 64;
__global__ void __launch_bounds__(256) big_update_kernel(SchurLaunch L, BigNodes B, int j0) {
  __shared__ double ls[BNB][BT + 1];  // L21 tile, [p][row]
  __shared__ double us[BNB][BT + 1];  // U12 tile, [p][col]
  const SchurNode N = L.nodes[B.idx[blockIdx.z]];
  const int n = N.kb + N.kt;
  const int r0 = j0 + BNB + blockIdx.x * BT, c0 = j0 + BNB + blockIdx.y * BT;
  if (r0 >= n || c0 >= n) return;
  double* a = L.S + N.s_off;
  for (int e = threadIdx.x; e < BNB * BT; e += blockDim.x) {
    const int i = e % BT, p = e / BT;
    ls[p][i] = r0 + i < n ? a[(int64_t)(j0 + p) * n + r0 + i] : 0.0;
    us[p][i] = c0 + i < n ? a[(int64_t)(c0 + i) * n + j0 + p] : 0.0;
  }
  __syncthreads();
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // rows tx + 16x, cols ty + 16y
  double acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = 0.0;
#pragma unroll 8
  for (int p = 0; p < BNB; ++p) {
    double l[4], u[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) l[x] = ls[p][tx + 16 * x];
#pragma unroll
    for (int y = 0; y < 4; ++y) u[y] = us[p][ty + 16 * y];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[x][y] = fma(l[x], u[y], acc[x][y]);
  }
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const int c = c0 + ty + 16 * y;
    if (c >= n) continue;
    double* ac = a + (int64_t)c * n;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int r = r0 + tx + 16 * x;
      if (r < n) ac[r] -= acc[x][y];
    }
  }
}

// ---------------------------------- blocked solve of the nodes' ancestor columns
// y = S^-1 Z for the N.coff ancestor columns of a node (the factorization's
// schur solve, src/HODLR_Matrix.cpp:682): the LU's row interchanges, then the
// unit-lower and the upper solves by 32-row diagonal blocks, each a
// register-resident triangular solve (one thread per column) followed by a
// 64 x 64-tiled update of the remaining rows over all SMs: each block of the LU is
// read once per 64 columns.
__global__ void __launch_bounds__(256) big_rhs_perm_kernel(SchurLaunch L, BigNodes B) {
  const SchurNode N = L.nodes[B.idx[blockIdx.y]];
  const int n = N.kb + N.kt;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N.coff) return;
  double* x = L.R + N.r_off + (int64_t)c * n;
  const int* piv = L.piv + N.p_off;
  for (int p = 0; p < n; ++p) {
    const int q = __ldg(piv + p);
    if (q < p || q >= n) {  // not an LU interchange: skip and report
      atomicOr(L.err, DEV_ERR_INDEX | DEV_ERR_AT_BLOCKED_PIV);
      continue;
    }
    if (q != p) {
      const double t = x[p];
      x[p] = x[q];
      x[q] = t;
    }
  }
}

template <bool LOWER>
__global__ void __launch_bounds__(256) big_rhs_diag_kernel(SchurLaunch L, BigNodes B, int j0) {
  __shared__ double t11[BNB][BNB + 1];
  const SchurNode N = L.nodes[B.idx[blockIdx.y]];
  const int n = N.kb + N.kt;
  if (j0 >= n) return;
  const int nb = min(BNB, n - j0);
  const double* a = L.S + N.s_off;
  for (int e = threadIdx.x; e < BNB * BNB; e += blockDim.x) {
    const int i = e % BNB, p = e / BNB;
    t11[i][p] = (i < nb && p < nb) ? a[(int64_t)(j0 + p) * n + j0 + i] : (i == p ? 1.0 : 0.0);
  }
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N.coff) return;
  double* x = L.R + N.r_off + (int64_t)c * n + j0;
  double u[BNB];
#pragma unroll
  for (int i = 0; i < BNB; ++i) u[i] = i < nb ? x[i] : 0.0;
  if (LOWER) {  // unit lower, rows in order
#pragma unroll
    for (int i = 1; i < BNB; ++i)
#pragma unroll
      for (int p = 0; p < i; ++p) u[i] = fma(-t11[i][p], u[p], u[i]);
  } else {  // upper, rows in reverse order
#pragma unroll
    for (int i = BNB - 1; i >= 0; --i) {
      u[i] = u[i] / t11[i][i];
#pragma unroll
      for (int p = 0; p < i; ++p) u[p] = fma(-t11[p][i], u[i], u[p]);
    }
  }
#pragma unroll
  for (int i = 0; i < BNB; ++i)
    if (i < nb) x[i] = u[i];
}

// Rows below the block (LOWER) or above it (!LOWER) of the node's ancestor
// columns -= S[those rows, block columns] * the block's solved rows.
template <bool LOWER>
__global__ void __launch_bounds__(256) big_rhs_update_kernel(SchurLaunch L, BigNodes B, int j0) {
  __shared__ double ls[BNB][BT + 1];  // S tile, [p][row]
  __shared__ double us[BNB][BT + 1];  // solved block rows, [p][col]
  const SchurNode N = L.nodes[B.idx[blockIdx.z]];
  const int n = N.kb + N.kt;
  if (j0 >= n) return;
  const int nb = min(BNB, n - j0);
  const int rlo = LOWER ? j0 + nb : 0, rhi = LOWER ? n : j0;
  const int r0 = rlo + blockIdx.x * BT, c0 = blockIdx.y * BT;
  if (r0 >= rhi || c0 >= N.coff) return;
  const double* a = L.S + N.s_off;
  double* x = L.R + N.r_off;
  for (int e = threadIdx.x; e < BNB * BT; e += blockDim.x) {
    const int i = e % BT, p = e / BT;
    ls[p][i] = (p < nb && r0 + i < rhi) ? a[(int64_t)(j0 + p) * n + r0 + i] : 0.0;
    us[p][i] = (p < nb && c0 + i < N.coff) ? x[(int64_t)(c0 + i) * n + j0 + p] : 0.0;
  }
  __syncthreads();
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double acc[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[q][y] = 0.0;
#pragma unroll 8
  for (int p = 0; p < BNB; ++p) {
    double l[4], u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) l[q] = ls[p][tx + 16 * q];
#pragma unroll
    for (int y = 0; y < 4; ++y) u[y] = us[p][ty + 16 * y];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[q][y] = fma(l[q], u[y], acc[q][y]);
  }
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const int c = c0 + ty + 16 * y;
    if (c >= N.coff) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + tx + 16 * q;
      if (r < rhi) x[(int64_t)c * n + r] -= acc[q][y];
    }
  }
}

// Launch helpers return the first CUDA error at once.
#define LCK(call)                             \
  do {                                        \
    cudaError_t e__ = (call);                 \
    if (e__ != cudaSuccess) return (int)e__;  \
  } while (0)

}  // namespace

int leaf_lu_launch(const LeafLULaunch& L, int nleaves, int smax, cudaStream_t s) {
  size_t smem = sizeof(double) * (size_t)smax * (smax | 1);
  LCK(smem_opt_in((const void*)leaf_lu_kernel, smem));
  leaf_lu_kernel<<<nleaves, LNT, smem, s>>>(L);
  return (int)cudaGetLastError();
}

int leaf_solve_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s) {
  if (L.ncols <= 0) return 0;
  if (L.ncols <= 16) {
    constexpr int TC = 16;
    size_t smem = sizeof(double) * (size_t)(smax | 1) * (smax + TC);
    LCK(smem_opt_in((const void*)leaf_solve_kernel<TC>, smem));
    leaf_solve_kernel<TC><<<dim3((L.ncols + TC - 1) / TC, nleaves), LNT, smem, s>>>(L);
  } else {
    constexpr int TC = 64;
    size_t smem = sizeof(double) * (size_t)(smax | 1) * (smax + TC);
    LCK(smem_opt_in((const void*)leaf_solve_kernel<TC>, smem));
    leaf_solve_kernel<TC><<<dim3((L.ncols + TC - 1) / TC, nleaves), LNT, smem, s>>>(L);
  }
  return (int)cudaGetLastError();
}

// Inner panel width for rows x pnb doubles of shared memory (<= 200 KB).
static int panel_width(int rows) {
  int pnb = 16;
  while (pnb > 1 && (size_t)rows * pnb * sizeof(double) > 200 * 1024) pnb >>= 1;
  return pnb;
}

int schur_factor_launch(const SchurLaunch& L, int nnodes, const int* sd, cudaStream_t s) {
  if (nnodes == 0) return 0;
  int form_y = 1;  // CTAs per node for forming S: about 64K entries each
  for (int i = 0; i < nnodes; ++i)
    form_y = std::max(form_y, (int)std::min<int64_t>(256, (int64_t)sd[i] * sd[i] / 65536 + 1));
  schur_form_kernel<<<dim3(nnodes, form_y), 256, 0, s>>>(L);
  LCK(cudaGetLastError());
  int small_max = 0, big_max = 0;
  std::vector<int> big;
  for (int i = 0; i < nnodes; ++i) {
    if (sd[i] >= SCHUR_BIG_SD) {
      big.push_back(i);
      big_max = std::max(big_max, sd[i]);
    } else {
      small_max = std::max(small_max, sd[i]);
    }
  }
  if (small_max > 0) {
    // L21 and U12 of the first panel
    const size_t smem = sizeof(double) * 2 * PW * tile_pitch(std::max(0, small_max - PW));
    LCK(smem_opt_in((const void*)schur_lu_kernel, smem));
    schur_lu_kernel<<<nnodes, SNT, smem, s>>>(L, SCHUR_BIG_SD);
    LCK(cudaGetLastError());
  }
  for (size_t b0 = 0; b0 < big.size(); b0 += BIG_MAX) {
    BigNodes B;
    B.count = (int)std::min<size_t>(BIG_MAX, big.size() - b0);
    int mx = 0;
    for (int i = 0; i < B.count; ++i) {
      B.idx[i] = big[b0 + i];
      mx = std::max(mx, sd[big[b0 + i]]);
    }
    const int pnb = std::min(BNB, panel_width(mx));
    const size_t smem = (size_t)mx * pnb * sizeof(double);
    LCK(smem_opt_in((const void*)big_panel_kernel, smem));
    for (int j0 = 0; j0 < mx; j0 += BNB) {
      const int ctas = (mx - j0 + SNT - 1) / SNT;  // of a cluster, SNT rows each
      if (ctas == 1) {
        panel_kernel<false><<<dim3(1, B.count), SNT, 0, s>>>(L, B, j0);
      } else if (ctas <= 8) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas, B.count);
        cfg.blockDim = dim3(SNT);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = ctas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        LCK(cudaLaunchKernelEx(&cfg, panel_kernel<true>, L, B, j0));
      } else {
        big_panel_kernel<<<B.count, SNT, smem, s>>>(L, B, j0, pnb);
      }
      LCK(cudaGetLastError());
      big_swap_trsm_kernel<<<dim3((mx + 127) / 128, B.count), 128, 0, s>>>(L, B, j0);
      LCK(cudaGetLastError());
      const int rest = mx - j0 - BNB;
      if (rest > 0) {
        const int t = (rest + BT - 1) / BT;
        big_update_kernel<<<dim3(t, t, B.count), 256, 0, s>>>(L, B, j0);
        LCK(cudaGetLastError());
      }
    }
  }
  return (int)cudaGetLastError();
}

int schur_factor_launches(const int* sd, int nnodes) {
  int n = 1, small = 0, mx = 0, big = 0;
  for (int i = 0; i < nnodes; ++i) {
    if (sd[i] >= SCHUR_BIG_SD) {
      ++big;
      mx = std::max(mx, sd[i]);
    } else {
      small = 1;
    }
  }
  n += small;
  if (big) {
    const int batches = (big + BIG_MAX - 1) / BIG_MAX;
    for (int j0 = 0; j0 < mx; j0 += BNB) n += batches * (mx - j0 - BNB > 0 ? 3 : 2);
  }
  return n;
}

int schur_solve_factor_launch(const SchurLaunch& L, int nnodes, const int* sd, int coff,
                              cudaStream_t s, int* launches) {
  *launches = 0;
  if (nnodes == 0 || coff <= 0) return 0;
  std::vector<int> big;
  for (int i = 0; i < nnodes; ++i)
    if (sd[i] > 0) big.push_back(i);
  const int ctiles = (coff + BT - 1) / BT, cblocks = (coff + 255) / 256;
  for (size_t b0 = 0; b0 < big.size(); b0 += BIG_MAX) {
    BigNodes B;
    B.count = (int)std::min<size_t>(BIG_MAX, big.size() - b0);
    int mx = 0;
    for (int i = 0; i < B.count; ++i) {
      B.idx[i] = big[b0 + i];
      mx = std::max(mx, sd[big[b0 + i]]);
    }
    big_rhs_perm_kernel<<<dim3(cblocks, B.count), 256, 0, s>>>(L, B);
    LCK(cudaGetLastError());
    ++*launches;
    for (int j0 = 0; j0 < mx; j0 += BNB) {
      big_rhs_diag_kernel<true><<<dim3(cblocks, B.count), 256, 0, s>>>(L, B, j0);
      LCK(cudaGetLastError());
      const int rows = mx - j0 - BNB;
      if (rows > 0) {
        big_rhs_update_kernel<true><<<dim3((rows + BT - 1) / BT, ctiles, B.count), 256, 0, s>>>(
            L, B, j0);
        LCK(cudaGetLastError());
      }
      *launches += 1 + (rows > 0);
    }
    for (int j0 = (mx - 1) / BNB * BNB; j0 >= 0; j0 -= BNB) {
      big_rhs_diag_kernel<false><<<dim3(cblocks, B.count), 256, 0, s>>>(L, B, j0);
      LCK(cudaGetLastError());
      if (j0 > 0) {
        big_rhs_update_kernel<false><<<dim3((j0 + BT - 1) / BT, ctiles, B.count), 256, 0, s>>>(
            L, B, j0);
        LCK(cudaGetLastError());
      }
      *launches += 1 + (j0 > 0);
    }
  }
  return (int)cudaGetLastError();
}
