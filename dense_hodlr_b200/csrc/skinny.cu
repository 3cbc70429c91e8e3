// The direct solve for a few right-hand sides: every kernel reads its matrix
// once, as operand fragments of mma.m8n8k4.f64 loaded straight from global
// memory, with the right-hand sides as the 8 columns of the other operand.
//
// What bounds them: the bytes of V, K^-1 U and the LUs (each entry is used
// once per solve), and at the top of the tree the chain of block steps of a
// triangular solve.  The 64-wide GEMM tiles these products ran through before
// did 8 to 64 times the work of 8 or 1 columns, and the substitutions ran a
// 32-step chain of shuffles per 32 rows in one CTA.
//
//  * Triangular solves multiply by inverted 64 x 64 diagonal triangles (formed
//    once per factorization, behind the LU), so a block step is two small products
//    instead of a substitution: n / 64 steps each way.  A product with an inverse
//    alone is not backward stable; blocks that need it are refined (tri_mode).
//  * Large capacitance systems run on a cluster of up to 8 CTAs: block rows
//    dealt out cyclically, a solved block written to every CTA's shared memory.
//  * V^T X is split over rows into items; their sums are added by the
//    capacitance solve that reads them, in a fixed order.
//
// Measured on B200, a repeated direct solve end to end, 64-wide tiles and
// one-CTA substitutions -> these kernels: N = 262144 2D, 8 columns 7.59 -> 2.31
// ms (its panels' 3.2 GB at the copy rate: 0.49 ms); N = 30001 2D, 1 column 1.81
// -> 0.68.  Unrefined, and with the sums of V^T X that a capacitance solve starts
// with read one at a time, they took 2.48 and 0.88; unrefined, 1.99 and 0.59.
// What is left of 0.68 is the capacitance solves' 0.43 (the top one, 704 rows: 0.03
// for its sums, 22 block steps of 4 us), the panel kernels' 0.19 and 25 launches.
#include "skinny.h"

#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int NB = TRI_NB;
constexpr int SK_NT = 256;  // 8 warps
constexpr int TRI_BUFS = 4;  // block buffers of tri_solve; the triangle behind them

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// ------------------------------------------- inverted diagonal triangles
// How a block step uses an inverse D of a triangle T.  The residual of y = D x is at
// most u |T| |D| |T| |y|, a substitution's u |T| |y|: in the norm of the weights
// w = |T| z, z_j = 1 / max_i |T_ij| (rows and columns of a capacitance matrix differ
// by up to 1e43, so the measure must not depend on their scales), an excess of
// c = max_i (|T| |D| w)_i / w_i, and each y += D (x - T y) multiplies the excess by
// c u.  So k of them while c (c u)^k is below 0.01, k <= 3, none up to c = 4, and a
// substitution beyond (or where D overflows).  numpy, leaves of 64 and 128 points,
// five kernels in 1D to 3D, shifts 1 to 1e-8, residuals over a substitution's: at
// most 1.37, mean 1.04, as with a refinement everywhere; with none up to c = 8 2.1,
// 64 3.7, 512 22; with none at all 1e1 (shift 1e-2) to 1e6 (1e-8).
constexpr int TRI_SUBST = 4;
__device__ __forceinline__ int tri_mode(double c) {
  return c <= 4.0 ? 0 : c <= 1e7 ? 1 : c <= 1e10 ? 2 : c <= 3e11 ? 3 : TRI_SUBST;  // NaN: the last
}

// sum of at(p) over lo <= p < hi, eight loads in flight
template <class F>
__device__ __forceinline__ double sum_in_row(int lo, int hi, const F& at) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int p0 = lo & ~7; p0 < hi; p0 += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = p0 + u >= lo && p0 + u < hi ? at(p0 + u) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s[u & 3] += v[u];
  }
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// One CTA per diagonal block T of `m` rows (the rest of 64 is the identity):
// threads 0..63 invert the unit lower triangle (a column each), threads 64..127 the
// upper one, both by substitution in registers over a copy in shared memory.
__device__ void invert_block(const double* a, int ld, int m, double* inv, int2* mode,
                             double (*t)[NB + 1]) {
  __shared__ double z[2][NB], wt[2][NB];
  __shared__ int worst[2];
  const int tid = threadIdx.x, h = tid >= NB, j = tid & (NB - 1);
  const int lo = h ? j : 0, hi = h ? NB : j;  // stored columns of row j
  for (int e = tid; e < NB * NB; e += blockDim.x) {
    const int i = e % NB, q = e / NB;
    t[i][q] = i < m && q < m ? a[(int64_t)q * ld + i] : i == q ? 1.0 : 0.0;
  }
  if (tid < 2) worst[tid] = 0;
  __syncthreads();
  bool range = true;  // no inverse of a pivot is subnormal, or overflows
  double big = h ? 0.0 : 1.0;
#pragma unroll 16
  for (int i = 0; i < NB; ++i)
    if (h ? i <= j : i > j) big = fmax(big, fabs(t[i][j]));
  z[h][j] = 1.0 / big;
  if (tid < NB) {
    const double r = 1.0 / t[tid][tid];
    t[tid][NB] = r;
    range = fabs(r) > 0x1p-1000 && fabs(r) < 0x1p1000;
  }
  __syncthreads();
  const double w = (h ? 0.0 : z[0][j]) +
                   sum_in_row(lo, hi, [&](int p) { return fabs(t[j][p]) * z[h][p]; });
  wt[h][j] = w;
  double x[NB];
  if (tid < NB) {
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      double v = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int p = 0; p < i; ++p) v = fma(-t[i][p], x[p], v);
      x[i] = v;
    }
  } else {
#pragma unroll
    for (int i = NB - 1; i >= 0; --i) {
      double v = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int p = NB - 1; p > i; --p) v = fma(-t[i][p], x[p], v);
      x[i] = v * t[i][NB];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (tid < NB ? i > j : i <= j) t[i][j] = x[i];
  __syncthreads();
  const double v = (h ? 0.0 : wt[0][j]) +  // |D| w
                   sum_in_row(lo, hi, [&](int p) { return fabs(t[j][p]) * wt[h][p]; });
  z[h][j] = v;
  __syncthreads();
  const double c =  // |T| |D| w
      j >= m ? w : (h ? 0.0 : v) + sum_in_row(lo, min(hi, m), [&](int p) {
        return fabs(a[(int64_t)p * ld + j]) * z[h][p];
      });
  atomicMax(&worst[h], tri_mode(c / w));
  if (!range) atomicMax(&worst[1], TRI_SUBST);
  for (int e = tid; e < NB * NB; e += blockDim.x) {
    const int i = e % NB, q = e / NB;
    if (i < m && q < m) inv[q * m + i] = t[i][q];
  }
  __syncthreads();
  if (tid == 0) *mode = make_int2(worst[0], worst[1]);
}

// Where block b of a packed n x n LU has its inverse, and the modes of its
// lower and upper triangle (tri_elems doubles behind the LU).
__device__ __forceinline__ const double* tri_inverse(const double* a, int n, int b) {
  return a + (int64_t)n * n + (int64_t)b * NB * NB;
}
__device__ __forceinline__ const int2* tri_modes(const double* a, int n) {
  return reinterpret_cast<const int2*>(a + (int64_t)n * n + tri_elems(n)) - (n + NB - 1) / NB;
}

__global__ void __launch_bounds__(2 * NB) invert_leaves_kernel(LeafSolveLaunch L) {
  __shared__ double t[NB][NB + 1];
  const int s = L.leaf_size[blockIdx.x], b0 = blockIdx.y * NB;
  if (b0 >= s) return;
  double* a = const_cast<double*>(L.lu) + L.lu_off[blockIdx.x];
  invert_block(a + (int64_t)b0 * s + b0, s, min(NB, s - b0),
               const_cast<double*>(tri_inverse(a, s, blockIdx.y)),
               const_cast<int2*>(tri_modes(a, s)) + blockIdx.y, t);
}

__global__ void __launch_bounds__(2 * NB) invert_nodes_kernel(SchurLaunch L, int* perm) {
  __shared__ double t[NB][NB + 1];
  const SchurNode N = L.nodes[blockIdx.x];
  const int n = N.kb + N.kt, b0 = (int)(blockIdx.y - 1) * NB;
  if (blockIdx.y == 0) {  // the interchanges, in order, as a permutation
    int* p = perm + N.p_off;
    const int* piv = L.piv + N.p_off;
    // a chain of swaps: in shared memory where both arrays fit
    constexpr int FIT = (int)(sizeof(t) / sizeof(int) / 2);
    int* sp = reinterpret_cast<int*>(&t[0][0]);
    const bool fit = n <= FIT;
    int* q = fit ? sp : p;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      q[i] = i;
      if (fit) sp[FIT + i] = piv[i];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < n; ++i) {
        const int r = fit ? sp[FIT + i] : piv[i];
        if (r < i || r >= n) {  // not an LU interchange: skip and report
          atomicOr(L.err, DEV_ERR_INDEX | DEV_ERR_AT_SOLVE_PIV);
          continue;
        }
        const int v = q[i];
        q[i] = q[r];
        q[r] = v;
      }
    __syncthreads();
    if (fit)
      for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = sp[i];
    return;
  }
  if (b0 >= n) return;
  double* a = L.S + N.s_off;
  invert_block(a + (int64_t)b0 * n + b0, n, min(NB, n - b0),
               const_cast<double*>(tri_inverse(a, n, blockIdx.y - 1)),
               const_cast<int2*>(tri_modes(a, n)) + blockIdx.y - 1, t);
}

// --------------------------------------------------- blocked triangular solve
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// D (8 x 8 NT tile) = A (8 x 64, fragments av) times a 64-row block of x, the
// 16 MMAs of a tile in independent chains of 4.
template <int NT>
__device__ __forceinline__ void block_product(const double (&av)[NB / 4],
                                              const double* const (&x)[NT],
                                              double (&out)[NT][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    double acc[4][2];
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c][0] = acc[c][1] = 0.0;
#pragma unroll
    for (int k = 0; k < NB / 4; ++k) dmma(acc[k & 3], av[k], x[u][(4 * k + t) * 8 + g]);
#pragma unroll
    for (int e = 0; e < 2; ++e) out[u][e] = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
  }
}

// A triangle itself, for blocks that are refined or substituted: element (i, j) at
// ts[j * TRI_PITCH + i], no bank conflicts between the lanes of a fragment.
constexpr int TRI_PITCH = NB + 4;

// The 8 rows of a triangular block that a warp multiplies: a scheduler's two warps
// (w and w + 4) together have 9 of the 16 8 x 8 tiles that are not zero.
__device__ __forceinline__ int tri_rows(int w) { return 8 * (w < 4 ? w : 11 - w); }

// A triangle's (dir 0: unit lower, 1: upper) element in that warp's fragment k:
// stored(col, row), or what the format implies.
template <class F>
__device__ __forceinline__ void load_tri(int dir, int m, const F& stored, double (&v)[NB / 4]) {
  const int lane = threadIdx.x & 31, row = tri_rows(threadIdx.x >> 5) + (lane >> 2), t = lane & 3;
#pragma unroll
  for (int k = 0; k < NB / 4; ++k) {
    const int col = 4 * k + t;
    const bool in = (dir == 0 ? col < row : col >= row) && row < m && col < m;
    v[k] = in ? stored(col, row) : dir == 0 && col == row ? 1.0 : 0.0;
  }
}

// block_product for a triangle's fragments, without its zero tiles.
template <int NT>
__device__ __forceinline__ void tri_product(int dir, const double (&av)[NB / 4],
                                            const double* const (&x)[NT], double (&out)[NT][2]) {
  const int lane = threadIdx.x & 31, r8 = tri_rows(threadIdx.x >> 5) / 8, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    double acc[4][2];
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c][0] = acc[c][1] = 0.0;
#pragma unroll
    for (int k = 0; k < NB / 4; ++k)
      if (dir == 0 ? k / 2 <= r8 : k / 2 >= r8)  // the same for the warp
        dmma(acc[k & 3], av[k], x[u][(4 * k + t) * 8 + g]);
#pragma unroll
    for (int e = 0; e < 2; ++e) out[u][e] = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
  }
}

// Columns of a 64-row block (row i, column c at x[u][i * 8 + c]) by substitution:
// a warp takes column w of each tile, lane l rows l and l + 32.
template <int NT>
__device__ __noinline__ void substitute_block(const double* ts, int dir, int m,
                                              double* const (&x)[NT]) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r1 = lane + 32;
  // the reciprocal pivots, before the chain (a division inside it: 8 us a block)
  const double q0 = 1.0 / (lane < m ? ts[lane * TRI_PITCH + lane] : 1.0);
  const double q1 = 1.0 / (r1 < m ? ts[r1 * TRI_PITCH + r1] : 1.0);
  for (int u = 0; u < NT; ++u) {
    double v0 = x[u][lane * 8 + w], v1 = x[u][r1 * 8 + w];
    // the next column is on its way while this one's chain runs
    auto column = [&](int s, double& t0, double& t1) {
      const double* tp = ts + (dir == 0 ? s : m - 1 - s) * TRI_PITCH;
      t0 = tp[lane];
      t1 = tp[r1];
    };
    double t0, t1, n0 = 0.0, n1 = 0.0;
    column(0, t0, t1);
    for (int s = 0; s < m; ++s) {
      const int p = dir == 0 ? s : m - 1 - s;
      if (s + 1 < m) column(s + 1, n0, n1);
      double xp = p < 32 ? v0 : v1;
      if (dir == 1 && lane == (p & 31)) {
        const double r = p < 32 ? q0 : q1;
        xp = fabs(r) > 0x1p-1000 && fabs(r) < 0x1p1000 ? xp * r : xp / ts[p * TRI_PITCH + p];
        (p < 32 ? v0 : v1) = xp;
      }
      xp = __shfl_sync(all, xp, p & 31);
      if (dir == 0 ? lane > p && lane < m : lane < p) v0 = fma(-t0, xp, v0);
      if (dir == 0 ? r1 > p && r1 < m : r1 < p) v1 = fma(-t1, xp, v1);
      t0 = n0;
      t1 = n1;
    }
    x[u][lane * 8 + w] = v0;
    x[u][r1 * 8 + w] = v1;
  }
}

// x <- U^-1 L^-1 x with the packed LU `a` (n x n, its triangles' inverses behind it)
// in global memory.  The CTAs of a cluster (CL; otherwise one CTA) own block
// rows rank, rank + size, ...: own[u][q][r][c] is column c of column tile u,
// row r of owned block q.  Step b: its owner forms D_b x_b, one 8-row tile a
// warp, refines it where the triangle asks for that, and writes it to every CTA's
// xb[b mod 3]; all subtract A(b', b) x_b from their blocks still to be solved.
// xb[3] and the triangle at `ts` are the refinement's, and xb[b mod 3] before x_b is
// there; the triangle is copied into shared memory a step ahead, not held in
// registers, which doubled (120 -> 255).
//
// The chain is wait, update of the next block, its product, write: the owner
// of the next step does those first and everybody else's updates overlap it.
// A CTA arrives for step b + 1 once its updates of step b - 1 are done, so the
// buffer of step b - 1 is free when step b + 2 is written: three buffers.  The
// matrix fragments of both products are loaded before the wait.
template <int NT, bool CL>
__device__ void tri_solve(const double* __restrict__ a, int n, double* own, int own_blocks,
                          double (*xb)[NT][NB][8]) {
  double* ts = &xb[TRI_BUFS][0][0][0];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  int rank = 0, size = 1;
  if (CL) {
    rank = (int)cg::this_cluster().block_rank();
    size = (int)cg::this_cluster().num_blocks();
  }
  const int nb = (n + NB - 1) / NB;
  auto ox = [&](int u, int q) { return own + ((int64_t)u * own_blocks + q) * NB * 8; };
  double dv[NB / 4];
  int mode = 0;
  auto load_diag = [&](int dir, int b) {
    const int m = min(NB, n - b * NB);
    const int2 md = __ldg(tri_modes(a, n) + b);
    mode = dir == 0 ? md.x : md.y;
    const double* inv = tri_inverse(a, n, b);
    load_tri(dir, m, [&](int c, int r) { return __ldg(inv + c * m + r); }, dv);
    if (mode > 0) {
      const double* tri = a + (int64_t)b * NB * n + b * NB;
      for (int e = threadIdx.x; e < NB * m; e += SK_NT) {
        const int i = e % NB, j = e / NB;
        if (i < m)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                           (unsigned)__cvta_generic_to_shared(ts + j * TRI_PITCH + i)),
                       "l"(tri + (int64_t)j * n + i)
                       : "memory");
      }
    }
  };
  double av[NB / 4];
  auto load_tile = [&](int q, int r8, int b) {
    const int gr = (q * size + rank) * NB + 8 * r8 + g;
#pragma unroll
    for (int k = 0; k < NB / 4; ++k) {
      const int col = b * NB + 4 * k + t;
      av[k] = gr < n && col < n ? __ldg(a + (int64_t)col * n + gr) : 0.0;
    }
  };
  // x_b = D_b x_b of this CTA's block b, to all CTAs' buffers
  auto solve_block = [&](int dir, int b, int buf) {
    const int q = CL ? b / size : b;
    const int m = min(NB, n - b * NB), at = (tri_rows(w) + g) * 8 + 2 * t;  // this lane's
    if (mode > 0) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the block's updates, by all warps; its triangle
    const double* x[NT];
    double y[NT][2];
#pragma unroll
    for (int u = 0; u < NT; ++u) x[u] = ox(u, q);
    if (mode == TRI_SUBST) {
      double* xs[NT];
#pragma unroll
      for (int u = 0; u < NT; ++u) xs[u] = ox(u, q);
      substitute_block<NT>(ts, dir, m, xs);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        y[u][0] = x[u][at];
        y[u][1] = x[u][at + 1];
      }
    } else {
      tri_product<NT>(dir, dv, x, y);
    }
    const double *yp[NT], *rp[NT];
#pragma unroll
    for (int u = 0; u < NT; ++u) {
      yp[u] = &xb[buf][u][0][0];
      rp[u] = &xb[3][u][0][0];
    }
#pragma unroll 1
    for (int it = 0; it < (mode == TRI_SUBST ? 0 : mode); ++it) {  // y += D (x - T y)
      double v[NT][2];
#pragma unroll
      for (int u = 0; u < NT; ++u)
        *reinterpret_cast<double2*>(&xb[buf][u][0][0] + at) = make_double2(y[u][0], y[u][1]);
      __syncthreads();
      double tv[NB / 4];
      load_tri(dir, m, [&](int c, int r) { return ts[c * TRI_PITCH + r]; }, tv);
      tri_product<NT>(dir, tv, yp, v);
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        const double2 r = *reinterpret_cast<const double2*>(x[u] + at);
        *reinterpret_cast<double2*>(&xb[3][u][0][0] + at) =
            make_double2(r.x - v[u][0], r.y - v[u][1]);
      }
      __syncthreads();
      tri_product<NT>(dir, dv, rp, v);
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        y[u][0] += v[u][0];
        y[u][1] += v[u][1];
      }
    }
    if (mode == 0) __syncthreads();  // everybody has read x
#pragma unroll
    for (int u = 0; u < NT; ++u) {
      const double2 v = make_double2(y[u][0], y[u][1]);
      *reinterpret_cast<double2*>(ox(u, q) + at) = v;
      double* to = &xb[buf][u][0][0] + at;
      if (CL)
        for (int r = 0; r < size; ++r)
          *reinterpret_cast<double2*>(cg::this_cluster().map_shared_rank(to, r)) = v;
      else
        *reinterpret_cast<double2*>(to) = v;
    }
  };
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir) {  // forward with L, backward with U
    auto block_of = [&](int step) { return dir == 0 ? step : nb - 1 - step; };
    auto mine = [&](int step) { return step < nb && (!CL || block_of(step) % size == rank); };
    if (mine(0)) {
      load_diag(dir, block_of(0));
      solve_block(dir, block_of(0), 0);
    }
    if (CL) cluster_arrive();
#pragma unroll 1
    for (int step = 0; step < nb; ++step) {
      const int b = block_of(step), buf = step % 3;
      // the owned blocks behind step b (nearest first), in 8-row tiles over warps
      int q0, q1;
      if (dir == 0) {
        q0 = (b + 1 - rank + size - 1) / size;
        q1 = (nb - rank + size - 1) / size;
      } else {
        q0 = 0;
        q1 = b > rank ? (b - rank + size - 1) / size : 0;
      }
      q0 = max(q0, 0);
      const bool next = mine(step + 1);
      if (q0 < q1) load_tile(dir == 0 ? q0 : q1 - 1, w, b);
      if (next) load_diag(dir, block_of(step + 1));
      if (CL) {
        cluster_wait();
        if (!next && step + 1 < nb) cluster_arrive();
      } else {
        __syncthreads();
      }
      const double* xs[NT];
#pragma unroll
      for (int u = 0; u < NT; ++u) xs[u] = &xb[buf][u][0][0];
#pragma unroll 1
      for (int i = 0; i < q1 - q0; ++i) {  // a warp takes tile w of every block
        const int q = dir == 0 ? q0 + i : q1 - 1 - i;
        double y[NT][2];
        block_product<NT>(av, xs, y);
        if (i + 1 < q1 - q0) load_tile(dir == 0 ? q + 1 : q - 1, w, b);
#pragma unroll
        for (int u = 0; u < NT; ++u) {
          double2* x = reinterpret_cast<double2*>(ox(u, q) + (8 * w + g) * 8 + 2 * t);
          double2 v = *x;
          v.x -= y[u][0];
          v.y -= y[u][1];
          *x = v;
        }
        if (i == 0 && next) {
          solve_block(dir, block_of(step + 1), (step + 1) % 3);
          if (CL) cluster_arrive();
        }
      }
    }
    // everybody's updates before the other direction's first block
    if (CL)
      cg::this_cluster().sync();
    else
      __syncthreads();
  }
}

// ------------------------------------------------------------------ leaves
// One CTA per leaf and 8 NT columns, the leaf's rows in shared memory.
template <int NT>
__global__ void __launch_bounds__(SK_NT, 2) leaf_apply_kernel(LeafSolveLaunch L) {
  extern __shared__ __align__(16) double dyn[];
  const int leaf = blockIdx.x, c0 = blockIdx.y * 8 * NT;
  const int r0 = L.leaf_min[leaf], s = L.leaf_size[leaf], nb = (s + NB - 1) / NB;
  double* own = dyn;
  auto xb = reinterpret_cast<double(*)[NT][NB][8]>(dyn + (size_t)NT * nb * NB * 8);  // TRI_BUFS
  const int* perm = L.perm + r0;
  for (int e = threadIdx.x; e < 8 * NT * nb * NB; e += SK_NT) {
    const int i = e % (nb * NB), c = e / (nb * NB);
    double v = 0.0;
    if (i < s && c0 + c < L.ncols) {
      const int pi = perm[i];
      if (pi < 0 || pi >= s) {  // never written by a valid leaf LU: skip and report
        if (L.err) atomicOr(L.err, DEV_ERR_INDEX | DEV_ERR_AT_LEAF_PERM);
      } else {
        v = L.X[(int64_t)(c0 + c) * L.ldx + r0 + pi];
      }
    }
    own[((int64_t)(c >> 3) * nb * NB + i) * 8 + (c & 7)] = v;
  }
  __syncthreads();
  tri_solve<NT, false>(L.lu + L.lu_off[leaf], s, own, nb, xb);
  for (int e = threadIdx.x; e < 8 * NT * nb * NB; e += SK_NT) {
    const int i = e % (nb * NB), c = e / (nb * NB);
    if (i < s && c0 + c < L.ncols)
      L.X[(int64_t)(c0 + c) * L.ldx + r0 + i] = own[((int64_t)(c >> 3) * nb * NB + i) * 8 + (c & 7)];
  }
}

// ------------------------------------------------------------ capacitances
// PARTS: r row-summed from the V^T X chunks, y row-major; otherwise r and y
// column-major (n x nrhs at the node's z).  Cluster `size` CTAs per (node,
// column tile); grid.x = node * size + rank.
// Two CTAs an SM for one column tile (128 registers; N = 262144, 8 columns 2.24 ms
// against 2.38 unbounded); two tiles spill inside the chain then (40000-point cube, 16
// columns, the capacitance solves of 5 passes 6.3 ms against 3.9).
template <int NT, bool PARTS, bool CL>
__global__ void __launch_bounds__(SK_NT, NT == 1 ? 2 : 1) cap_solve_kernel(CapLaunch L, int nrhs, int own_max,
                                                          int ncp, unsigned* err) {
  extern __shared__ __align__(16) double dyn[];
  int rank = 0, size = 1;
  if (CL) {
    rank = (int)cg::this_cluster().block_rank();
    size = (int)cg::this_cluster().num_blocks();
  }
  const CapNode N = L.nodes[blockIdx.x / size];
  const int n = N.n, nb = (n + NB - 1) / NB, c0 = blockIdx.y * 8 * NT;
  constexpr int NCP = 8 * NT;
  const int ob = (nb - rank + size - 1) / size;  // owned blocks
  // the owned rows: in shared memory, or (one CTA, more rows than fit) in L.big
  const size_t mine = (size_t)NT * own_max * NB * 8;
  double* own = L.big ? L.big + (blockIdx.y * gridDim.x + blockIdx.x) * mine : dyn;
  auto xb = reinterpret_cast<double(*)[NT][NB][8]>(L.big ? dyn : dyn + mine);
  const int* perm = L.perm + N.p_off;
  for (int e = threadIdx.x; e < NCP * ob * NB; e += SK_NT) {
    const int c = PARTS ? e % NCP : e / (ob * NB), lr = PARTS ? e / NCP : e % (ob * NB);
    const int i = ((lr / NB) * size + rank) * NB + lr % NB;
    double v = 0.0;
    if (i < n) {
      const int q = __ldg(perm + i);
      if (q < 0 || q >= n) {
        atomicOr(err, DEV_ERR_INDEX | DEV_ERR_AT_SOLVE_PIV);
      } else if (PARTS) {
        const bool h = !(q >= N.off[0] && q < N.off[0] + N.m[0]);
        const double* p = L.part + (h ? N.part[1] : N.part[0]) +
                          (int64_t)(q - (h ? N.off[1] : N.off[0])) * ncp + c0 + c;
        const int64_t st = (int64_t)(h ? N.m[1] : N.m[0]) * ncp;
        const int count = h ? N.chunks[1] : N.chunks[0];
        constexpr int U = 16;  // loads in flight, added in order
        for (int k = 0; k < count; k += U) {
          double s[U];
#pragma unroll
          for (int i = 0; i < U; ++i) s[i] = k + i < count ? __ldg(p + (k + i) * st) : 0.0;
#pragma unroll
          for (int i = 0; i < U; ++i)
            if (k + i < count) v += s[i];
        }
      } else if (c0 + c < nrhs) {
        v = L.z[N.z + (int64_t)(c0 + c) * n + q];
      }
    }
    own[((int64_t)(c >> 3) * own_max * NB + lr) * 8 + (c & 7)] = v;
  }
  // column-major right-hand sides are overwritten by other CTAs of the cluster
  if (CL)
    cg::this_cluster().sync();
  else
    __syncthreads();
  tri_solve<NT, CL>(L.S + N.s_off, n, own, own_max, xb);
  for (int e = threadIdx.x; e < NCP * ob * NB; e += SK_NT) {
    const int c = PARTS ? e % NCP : e / (ob * NB), lr = PARTS ? e / NCP : e % (ob * NB);
    const int i = ((lr / NB) * size + rank) * NB + lr % NB;
    if (i >= n) continue;
    const double v = own[((int64_t)(c >> 3) * own_max * NB + lr) * 8 + (c & 7)];
    if (PARTS)
      L.z[N.z + (int64_t)i * ncp + c0 + c] = v;
    else if (c0 + c < nrhs)
      L.z[N.z + (int64_t)(c0 + c) * n + i] = v;
  }
}

// ------------------------------------------------------------------ V^T X
// One CTA per item: at most 128 columns of V, any number of rows, TN_ROWS at a
// time.  A fragments are 8 columns of V by 4 row pairs: a lane loads rows 2t,
// 2t + 1 of column g (16 bytes) and feeds them to two MMAs, the right-hand
// sides with the same rows from shared memory.  Warps share the columns (16
// each), or, when there are few, the rows, added in warp order.  Few, long
// items keep the sums short that the capacitance solve adds up (a 504-row item
// of all 357 columns left it 293 of them at N = 262144).
constexpr int TN_PITCH = TN_ROWS + 8 + 8;  // a multiple of 8, odd in units of 64 bytes
static_assert((TN_PITCH / 8) % 2 == 1, "column tiles must not share banks");

template <int NT>
__global__ void __launch_bounds__(SK_NT) skinny_tn_kernel(const TnItem* __restrict__ items,
                                                          const double* __restrict__ X,
                                                          int64_t ldx, int nrhs, int64_t ldv,
                                                          double* __restrict__ part) {
  extern __shared__ __align__(16) double dyn[];
  constexpr int NCP = 8 * NT;
  double* xs = dyn;                        // [NCP][TN_PITCH]
  double* red = dyn + NCP * TN_PITCH;      // [8 warps][2][NT][32][2]
  const TnItem it = items[blockIdx.x];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int cw = (it.M + 15) / 16;                             // 16-column groups, at most 8
  const int mw = cw > 4 ? 8 : cw > 2 ? 4 : cw, rw = 8 / mw;    // warps over columns, over rows
  const int wm = w % mw, wr = w / mw, m0 = 16 * wm;
  const bool ok0 = m0 + g < it.M, ok1 = m0 + 8 + g < it.M;
  double acc[2][NT][2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[q][u][0] = acc[q][u][1] = 0.0;
  for (int r0 = it.row0; r0 < it.row0 + it.rows;) {
    const int base = r0 & ~1, end = min(it.row0 + it.rows, base + TN_ROWS);
    const int lo = r0 - base, hi = end - base, span = (hi + 7) & ~7;
    r0 = end;
    __syncthreads();  // the last piece has been read
    for (int e = threadIdx.x; e < NCP * span; e += SK_NT) {
      const int c = e / span, i = e - c * span;
      xs[c * TN_PITCH + i] =
          c < nrhs && i >= lo && i < hi ? X[(int64_t)c * ldx + base + i] : 0.0;
    }
    __syncthreads();
    if (m0 >= it.M) continue;
    const double* v0 = it.V + (int64_t)(ok0 ? m0 + g : 0) * ldv + base + 2 * t;
    const double* v1 = it.V + (int64_t)(ok1 ? m0 + 8 + g : 0) * ldv + base + 2 * t;
    constexpr int U = 4;
    for (int i0 = 8 * U * wr; i0 < span; i0 += 8 * U * rw) {
      double2 a[2][U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 8 * u, r = i + 2 * t;
        double2 x = make_double2(0.0, 0.0), y = x;
        if (r < hi) {  // the pair's second row may be padding: in the panel's storage
          x = *reinterpret_cast<const double2*>(v0 + i);
          y = *reinterpret_cast<const double2*>(v1 + i);
        }
        // rows outside the item may hold anything
        const bool in0 = r >= lo && r < hi, in1 = r + 1 < hi;
        a[0][u] = make_double2(ok0 && in0 ? x.x : 0.0, ok0 && in1 ? x.y : 0.0);
        a[1][u] = make_double2(ok1 && in0 ? y.x : 0.0, ok1 && in1 ? y.y : 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 8 * u;
        if (i >= span) break;
#pragma unroll
        for (int v = 0; v < NT; ++v) {
          const double2 b =
              *reinterpret_cast<const double2*>(xs + (8 * v + g) * TN_PITCH + i + 2 * t);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            dmma(acc[q][v], a[q][u].x, b.x);
            dmma(acc[q][v], a[q][u].y, b.y);
          }
        }
      }
    }
  }
  if (rw > 1) {  // the rows' shares, warps in order
    auto slot = [&](int ww, int q, int v) {
      return reinterpret_cast<double2*>(red + ((((ww * 2 + q) * NT + v) * 32) + lane) * 2);
    };
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int v = 0; v < NT; ++v) *slot(w, q, v) = make_double2(acc[q][v][0], acc[q][v][1]);
    __syncthreads();
    if (wr == 0)
      for (int r = 1; r < rw; ++r)
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int v = 0; v < NT; ++v) {
            const double2 o = *slot(wm + r * mw, q, v);
            acc[q][v][0] += o.x;
            acc[q][v][1] += o.y;
          }
  }
  if (wr == 0)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int m = m0 + 8 * q + g;
      if (m < it.M)
#pragma unroll
        for (int v = 0; v < NT; ++v)
          *reinterpret_cast<double2*>(part + it.out + (int64_t)m * NCP + 8 * v + 2 * t) =
              make_double2(acc[q][v][0], acc[q][v][1]);
    }
}

// --------------------------------------------------------------- X -= Y y
// One CTA per 128 rows (8 warps of 16).  A fragments are 8 row pairs by 4
// columns: a lane loads rows 2g, 2g + 1 of column t (16 bytes; a column's
// piece is a full 128-byte line) for two MMAs; y in shared memory, NN_K rows
// at a time.
constexpr int NN_K = 256;

template <int NT>
__global__ void __launch_bounds__(SK_NT) skinny_nn_kernel(const NnItem* __restrict__ items,
                                                          double* __restrict__ X, int64_t ldx,
                                                          int nrhs, int64_t ldy,
                                                          const double* __restrict__ z) {
  __shared__ __align__(16) double ys[NT][NN_K][8];
  constexpr int NCP = 8 * NT;
  const NnItem it = items[blockIdx.x];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int base = it.row0 & ~1;
  const int r = base + 16 * w + 2 * g;  // this lane's row pair
  const bool in0 = r >= it.row0 && r < it.row0 + it.rows, in1 = r + 1 < it.row0 + it.rows;
  const bool load = r < it.row0 + it.rows;
  double acc[2][NT][2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int v = 0; v < NT; ++v) acc[q][v][0] = acc[q][v][1] = 0.0;
  for (int kb = 0; kb < it.K; kb += NN_K) {
    const int kn = min(NN_K, it.K - kb), k4 = (kn + 3) & ~3;
    __syncthreads();
    for (int e = threadIdx.x; e < k4 * NCP; e += SK_NT) {
      const int k = e / NCP, c = e % NCP;
      ys[c >> 3][k][c & 7] = k < kn ? z[it.z + (int64_t)(kb + k) * NCP + c] : 0.0;
    }
    __syncthreads();
    constexpr int U = 8;
    for (int k0 = 0; k0 < k4; k0 += 4 * U) {
      double2 a[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + 4 * u + t;
        a[u] = load && k < kn
                   ? *reinterpret_cast<const double2*>(it.Y + (int64_t)(kb + k) * ldy + r)
                   : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + 4 * u >= k4) break;
#pragma unroll
        for (int v = 0; v < NT; ++v) {
          const double b = ys[v][k0 + 4 * u + t][g];
          dmma(acc[0][v], a[u].x, b);
          dmma(acc[1][v], a[u].y, b);
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NT; ++v)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = 8 * v + 2 * t + q;
      if (c >= nrhs) continue;
      double* x = X + (int64_t)c * ldx + r;
      if (in0) x[0] -= acc[0][v][q];
      if (in1) x[1] -= acc[1][v][q];
    }
}

#define LCK(call)                             \
  do {                                        \
    cudaError_t e__ = (call);                 \
    if (e__ != cudaSuccess) return (int)e__;  \
  } while (0)

// Shared memory of tri_solve beside the owned rows.
constexpr size_t tri_smem(int nt) {
  return sizeof(double) * (size_t)(TRI_BUFS * nt * NB * 8 + NB * TRI_PITCH);
}
// ... and with them, of the largest of the CTAs that share nb block rows.
size_t cap_smem(int nt, int nb, int ctas) {
  return sizeof(double) * 8 * NB * nt * (size_t)((nb + ctas - 1) / ctas) + tri_smem(nt);
}
// Column tiles a CTA takes: both of 9 to 16 columns where a cluster holds them
// (7000 rows), else one (22528 rows; beyond, L.big).
int cap_tiles(int nrhs, int max_sd, size_t limit) {
  const int nt = skinny_tiles(nrhs);
  return nt == 2 && cap_smem(2, (max_sd + NB - 1) / NB, 8) > limit ? 1 : nt;
}

template <int NT, bool PARTS>
int cap_launch(const CapLaunch& L, int nnodes, int nrhs, int max_sd, unsigned* err,
               cudaStream_t s) {
  const int nb = (max_sd + NB - 1) / NB;
  // CTAs of a cluster: at least two block rows each, and as few nodes as leave
  // SMs over; more where the rows would not fit
  int size = 1;
  while (size < 8 && (cap_smem(NT, nb, size) > std::min<size_t>(200 * 1024, L.smem_limit) ||
                      (nb >= 4 * size && nnodes * size < 148)))
    size *= 2;
  if (L.big) size = 1;
  const size_t smem = L.big ? tri_smem(NT) : cap_smem(NT, nb, size);
  if (smem > CAP_SMEM) return (int)cudaErrorInvalidValue;
  const dim3 grid(nnodes * size, (nrhs + 8 * NT - 1) / (8 * NT));
  const int own = (nb + size - 1) / size, ncp = 8 * skinny_tiles(nrhs);
  if (size == 1) {
    LCK(smem_opt_in((const void*)cap_solve_kernel<NT, PARTS, false>, smem));
    cap_solve_kernel<NT, PARTS, false><<<grid, SK_NT, smem, s>>>(L, nrhs, own, ncp, err);
    return (int)cudaGetLastError();
  }
  LCK(smem_opt_in((const void*)cap_solve_kernel<NT, PARTS, true>, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(SK_NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, cap_solve_kernel<NT, PARTS, true>, L, nrhs, own, ncp, err);
}

}  // namespace

int64_t cap_big_elems(int nnodes, int nrhs, int max_sd, size_t limit) {
  const int nt = cap_tiles(nrhs, max_sd, limit), nb = (max_sd + NB - 1) / NB;
  if (cap_smem(nt, nb, 8) <= limit) return 0;
  return (int64_t)nnodes * ((nrhs + 8 * nt - 1) / (8 * nt)) * nt * nb * NB * 8;
}

int tri_invert_leaves_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s) {
  if (nleaves == 0) return 0;
  invert_leaves_kernel<<<dim3(nleaves, (smax + NB - 1) / NB), 2 * NB, 0, s>>>(L);
  return (int)cudaGetLastError();
}

int tri_invert_nodes_launch(const SchurLaunch& L, int* perm, int nnodes, int max_sd,
                            cudaStream_t s) {
  if (nnodes == 0) return 0;
  invert_nodes_kernel<<<dim3(nnodes, 1 + (max_sd + NB - 1) / NB), 2 * NB, 0, s>>>(L, perm);
  return (int)cudaGetLastError();
}

int leaf_apply_launch(const LeafSolveLaunch& L, int nleaves, int smax, cudaStream_t s) {
  if (L.ncols <= 0 || nleaves == 0) return 0;
  const int nt = skinny_tiles(L.ncols), nb = (smax + NB - 1) / NB;
  const size_t smem = sizeof(double) * 8 * NB * nt * (size_t)nb + tri_smem(nt);
  const dim3 grid(nleaves, (L.ncols + 8 * nt - 1) / (8 * nt));
  if (nt == 1) {
    LCK(smem_opt_in((const void*)leaf_apply_kernel<1>, smem));
    leaf_apply_kernel<1><<<grid, SK_NT, smem, s>>>(L);
  } else {
    LCK(smem_opt_in((const void*)leaf_apply_kernel<2>, smem));
    leaf_apply_kernel<2><<<grid, SK_NT, smem, s>>>(L);
  }
  return (int)cudaGetLastError();
}

int skinny_tn_launch(const TnItem* items, int count, const double* X, int64_t ldx, int nrhs,
                     int64_t ldv, double* part, cudaStream_t s) {
  if (count == 0) return 0;
  const int nt = skinny_tiles(nrhs);
  const size_t smem = sizeof(double) * ((size_t)8 * nt * TN_PITCH + 8 * 2 * nt * 64);
  if (nt == 1) {
    LCK(smem_opt_in((const void*)skinny_tn_kernel<1>, smem));
    skinny_tn_kernel<1><<<count, SK_NT, smem, s>>>(items, X, ldx, nrhs, ldv, part);
  } else {
    LCK(smem_opt_in((const void*)skinny_tn_kernel<2>, smem));
    skinny_tn_kernel<2><<<count, SK_NT, smem, s>>>(items, X, ldx, nrhs, ldv, part);
  }
  return (int)cudaGetLastError();
}

int skinny_nn_launch(const NnItem* items, int count, double* X, int64_t ldx, int nrhs, int64_t ldy,
                     const double* z, cudaStream_t s) {
  if (count == 0) return 0;
  if (skinny_tiles(nrhs) == 1)
    skinny_nn_kernel<1><<<count, SK_NT, 0, s>>>(items, X, ldx, nrhs, ldy, z);
  else
    skinny_nn_kernel<2><<<count, SK_NT, 0, s>>>(items, X, ldx, nrhs, ldy, z);
  return (int)cudaGetLastError();
}

int cap_solve_launch(const CapLaunch& L, int nnodes, int nrhs, int max_sd, bool parts,
                     unsigned* err, cudaStream_t s) {
  if (nnodes == 0 || nrhs <= 0) return 0;
  if (cap_tiles(nrhs, max_sd, L.smem_limit) == 1)
    return parts ? cap_launch<1, true>(L, nnodes, nrhs, max_sd, err, s)
                 : cap_launch<1, false>(L, nnodes, nrhs, max_sd, err, s);
  return parts ? cap_launch<2, true>(L, nnodes, nrhs, max_sd, err, s)
               : cap_launch<2, false>(L, nnodes, nrhs, max_sd, err, s);
}
