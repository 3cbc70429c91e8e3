// Batched partial-pivot ACA: every off-diagonal block of a tree level (or of
// several levels) is compressed in one launch.
//
// Restates partialPivACA_LowRankApprox (src/lowRank.cpp:117-279) and
// chooseNextRowCol (src/lowRank.cpp:291-298).  The values that decide pivots
// are bit-identical to the CPU oracle: entries come from kfun.h, the residual
// row/column are accumulated in l order with separately rounded products and
// sums (src/lowRank.cpp:164-168, 211-215), the pivot is 1/r then multiplied
// (src/lowRank.cpp:208,230), and every argmax returns the first maximum.
// Only the Frobenius-norm dots of the stopping test (src/lowRank.cpp:234-241)
// are summed in a GPU order; they change epsilon in its last bits and thus
// the rank only when epsilon sits within rounding of the tolerance.  Each
// block records its smallest |eps - tol| / tol so such near ties are visible.
//
// Work decomposition.  A block is processed by a group of G CTAs.  CTA g owns
// a contiguous slice of the block's rows (for W, the column pass) and of its
// columns (for V, the row pass).  One ACA step is two group phases:
//   A  row residual on the column slice, slice argmax   -> barrier
//   B  pick pivot column, column residual on the row slice, slice argmax
//                                                        -> barrier
//   C  (redundant in every CTA) combine partials, next row.
// Each step streams the W and V panels once.  The stopping test of step k-1
// needs dots of its new columns with all earlier ones; they are accumulated
// while step k streams the same panels for its residuals, and step k is run
// speculatively: if epsilon_{k-1} <= tol it is discarded, so pivots and ranks
// are those of the reference's loop.  Where step k cannot stream the panels
// (a zero residual row, the capacity limit) the dots take a pass of their own.
// G = 1 for levels with many blocks (barriers are __syncthreads); G > 1 runs
// under a cooperative launch so that a group's CTAs are co-resident, and its
// barrier is a counter in global memory polled with a bounded spin.  Groups
// are either all of size L.G (CTA c works on block c / G) or, with a CTA
// table, of per-block size B.G starting at CTA B.g0 (sized from predicted
// ranks so that a level's blocks finish together).
#include "aca_post.cuh"
#include "common.cuh"
#include "hodlr_internal.h"

namespace {

// The block's W or V panel in the launch's element type (FP64 panels).
template <typename T>
__device__ __forceinline__ T* panel_of(double* d) { return d; }

struct Shared {
  double red_v[32];
  int red_i[32];
  int red_c[32];
  double bcast_d[8];
  int bcast_i[8];
};

// Group barrier.  gen counts the barriers this CTA has passed.  It gives up
// after L.spin_limit polls (or once another CTA has raised the error word).
__device__ bool group_sync(const AcaLaunch& L, unsigned* bar, int G, unsigned& gen,
                           unsigned* err) {
  __syncthreads();
  if (G == 1) return true;
  __shared__ int s_fail;
  if (threadIdx.x == 0) {
    s_fail = 0;
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned target = (gen + 1) * (unsigned)G + L.bar_extra;
    unsigned polls = 0;
    while (ld_acquire_u32(bar) < target) {
      if (++polls > L.spin_limit || *(volatile unsigned*)err) {
        atomicOr(err, DEV_ERR_TIMEOUT);
        s_fail = 1;
        break;
      }
      __nanosleep(128);
    }
    __threadfence();
  }
  ++gen;
  __syncthreads();
  return s_fail == 0;
}

template <int NT>
__device__ void block_argmax(Shared& sh, double& v, int& i) {
  warp_argmax(v, i);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    sh.red_v[w] = v;
    sh.red_i[w] = i;
  }
  __syncthreads();
  if (w == 0) {
    v = lane < NT / 32 ? sh.red_v[lane] : -1.0;
    i = lane < NT / 32 ? sh.red_i[lane] : INT_MAX;
    warp_argmax(v, i);
  }
  __syncthreads();
}

template <int NT>
__device__ int block_min_int(Shared& sh, int x) {
  x = warp_min_int(x);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh.red_c[w] = x;
  __syncthreads();
  int r = INT_MAX;
  if (w == 0) {
    r = lane < NT / 32 ? sh.red_c[lane] : INT_MAX;
    r = warp_min_int(r);
    if (lane == 0) sh.bcast_i[7] = r;
  }
  __syncthreads();
  r = sh.bcast_i[7];
  __syncthreads();
  return r;
}

// Deterministic block sum (fixed tree); result valid in every thread.
template <int NT>
__device__ double block_sum(Shared& sh, double x) {
  x = warp_sum(x);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh.red_v[w] = x;
  __syncthreads();
  if (w == 0) {
    double y = lane < NT / 32 ? sh.red_v[lane] : 0.0;
    y = warp_sum(y);
    if (lane == 0) sh.bcast_d[7] = y;
  }
  __syncthreads();
  double r = sh.bcast_d[7];
  __syncthreads();
  return r;
}

// Combine the G slice partials (value, index, chosen-flag, candidate) stored
// at part[g * stride + off .. off+3].  Slices are in index order, so the
// lowest index among equal maxima is the first maximum of the block.
__device__ void reduce_partials(Shared& sh, const double* part, int64_t stride, int G,
                                int off, double& v, int& idx, int& flag, int& cand) {
  if (threadIdx.x < 32) {
    double bv = -1.0;
    int bi = INT_MAX, bf = 0, bc = INT_MAX;
    for (int g = threadIdx.x; g < G; g += 32) {
      const double* p = part + g * stride + off;
      double pv = __ldcg(p);
      int pi = (int)__ldcg(p + 1);
      int pf = (int)__ldcg(p + 2);
      int pc = (int)__ldcg(p + 3);
      if (pv > bv || (pv == bv && pi < bi)) {
        bv = pv;
        bi = pi;
        bf = pf;
      }
      bc = min(bc, pc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      double v2 = __shfl_down_sync(0xffffffffu, bv, o);
      int i2 = __shfl_down_sync(0xffffffffu, bi, o);
      int f2 = __shfl_down_sync(0xffffffffu, bf, o);
      int c2 = __shfl_down_sync(0xffffffffu, bc, o);
      if (v2 > bv || (v2 == bv && i2 < bi)) {
        bv = v2;
        bi = i2;
        bf = f2;
      }
      bc = min(bc, c2);
    }
    if (threadIdx.x == 0) {
      sh.bcast_d[0] = bv;
      sh.bcast_i[0] = bi;
      sh.bcast_i[1] = bf;
      sh.bcast_i[2] = bc;
    }
  }
  __syncthreads();
  v = sh.bcast_d[0];
  idx = sh.bcast_i[0];
  flag = sh.bcast_i[1];
  cand = sh.bcast_i[2];
  __syncthreads();
}

// One residual pass over a slice [lo, hi) of a panel P (column l at P + l*ld):
//   r[j] = entry(j) - sum_{l<k} coef[l] * P(j, l)     (l order, unfused: bit-exact)
//   written to P(j, k) * scale (scale = 1 for V, the pivot reciprocal for W),
// and, if `dots`, the per-warp partial dots  sum_j P(j, l) * P(j, k-1)  for
// l < k-1 accumulated into dotw[warp * ldd + l] (the norm update of step k-1,
// computed while the panel streams through for step k).  Returns the slice
// argmax of |r| (first maximum), the first admissible candidate (unchosen,
// |r| > minPiv) and the partial sum of squares of the stored column.
template <int NT, int E, bool ROW, typename T>
__device__ void residual_pass(const AcaLaunch& L, const AcaBlock& B, T* P, int lo, int hi,
                              int k, const double* __restrict__ coef, bool dots,
                              double* __restrict__ dotw, int ldd, int fixed, const double* xfix,
                              double scale, const unsigned char* chosen, double& bv, int& bi,
                              int& cand, double& sq, bool& nonfinite, const EntrySrc& S) {
  constexpr int U = 16 / E;  // panel columns per chunk: 16 loads in flight per thread
  const int64_t ld = L.ld;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const double minPiv = L.minPivot;
  const T* __restrict__ Pr = P;  // columns < k are only read here
  const int kd = dots ? k - 1 : 0;
  bool first = true;
  for (int jb = lo; jb < hi; jb += E * NT, first = false) {
    int jj[E];
    bool ok[E];
    double s[E], vp[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      jj[e] = jb + tid + e * NT;
      ok[e] = jj[e] < hi;
      if (!ok[e]) jj[e] = lo;  // safe address; its products use vp = 0
      s[e] = 0.0;
      vp[e] = (dots && ok[e]) ? (double)Pr[jj[e] + (int64_t)(k - 1) * ld] : 0.0;
    }
    int l = 0;
    for (; l + U <= k; l += U) {
      double v[U][E];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < E; ++e) v[u][e] = (double)Pr[jj[e] + (int64_t)(l + u) * ld];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double c = coef[l + u];
#pragma unroll
        for (int e = 0; e < E; ++e) s[e] = __dadd_rn(s[e], __dmul_rn(c, v[u][e]));
      }
      if (dots) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (l + u >= kd) break;
          double d = 0.0;
#pragma unroll
          for (int e = 0; e < E; ++e) d = fma(v[u][e], vp[e], d);
          d = warp_sum(d);
          if (lane == 0) {
            if (first)
              dotw[w * ldd + l + u] = d;
            else
              dotw[w * ldd + l + u] += d;
          }
        }
      }
    }
    for (; l < k; ++l) {
      const double c = coef[l];
      double d = 0.0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const double v = (double)Pr[jj[e] + (int64_t)l * ld];
        s[e] = __dadd_rn(s[e], __dmul_rn(c, v));
        d = fma(v, vp[e], d);
      }
      if (dots && l < kd) {
        d = warp_sum(d);
        if (lane == 0) {
          if (first)
            dotw[w * ldd + l] = d;
          else
            dotw[w * ldd + l] += d;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (!ok[e]) continue;
      const int j = jj[e];
      double ent = ROW ? src_entry_xi(S, xfix, fixed, B.c0 + j)
                       : src_entry_xj(S, xfix, B.r0 + j, fixed);
      double r = __dsub_rn(ent, s[e]);
      // the panel keeps the value rounded to its type (no rounding for FP64),
      // and the norms of the stopping test use what it keeps
      const T kept = (T)(ROW ? r : __dmul_rn(scale, r));
      const double stored = (double)kept;
      P[j + (int64_t)k * ld] = kept;
      sq = fma(stored, stored, sq);
      double a = fabs(r);
      nonfinite |= !isfinite(r);
      if (a > bv) {  // increasing j per thread: the first maximum
        bv = a;
        bi = j;
      }
      if (cand == INT_MAX && a > minPiv && __ldcg(chosen + j) == 0) cand = j;
    }
  }
}

// Partial dots of step k-1 over this CTA's slices when they could not be
// fused into a residual pass (a zero residual row, or the capacity limit).
template <int NT, typename T>
__device__ void dots_only_pass(const AcaLaunch& L, const T* BW, const T* BV, int k, int i_lo,
                               int i_hi, int j_lo, int j_hi, int kcap, double* bank) {
  const int64_t ld = L.ld;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* wk = BW + (int64_t)(k - 1) * ld;
  const T* vk = BV + (int64_t)(k - 1) * ld;
  for (int l = w; l < k - 1; l += NT / 32) {
    const T* wl = BW + (int64_t)l * ld;
    const T* vl = BV + (int64_t)l * ld;
    double aw = 0.0, av = 0.0;
    for (int i = i_lo + lane; i < i_hi; i += 32) aw = fma((double)wk[i], (double)wl[i], aw);
    for (int j = j_lo + lane; j < j_hi; j += 32) av = fma((double)vl[j], (double)vk[j], av);
    aw = warp_sum(aw);
    av = warp_sum(av);
    if (lane == 0) {
      bank[l] = av;
      bank[kcap + l] = aw;
    }
  }
}

// epsilon of step k-1 from the G partial dots in the bank at offset bk
// (dotV at bk, dotW at bk + kcap):
// frobNormSq += 2 sum_l (w.W_l)(V_l.v) + |w|^2 |v|^2  (src/lowRank.cpp:234-241)
template <int NT>
__device__ double resolve_eps(Shared& sh, const AcaLaunch& L, const AcaBlock& B,
                              const double* part_grp, int G, int bk, int k, double swp,
                              double svp, double& frob2) {
  double sum_local = 0.0;
  for (int l = threadIdx.x; l < k - 1; l += NT) {
    double dv = 0.0, dw = 0.0;
    for (int q = 0; q < G; ++q) {
      dv += __ldcg(part_grp + q * L.part_stride + bk + l);
      dw += __ldcg(part_grp + q * L.part_stride + bk + B.kcap + l);
    }
    sum_local += dw * dv;
  }
  const double sumNorm = block_sum<NT>(sh, sum_local);
  frob2 += 2 * sumNorm + swp * svp;
  return sqrt(swp) * sqrt(svp) / sqrt(frob2);
}

// T: the element type of the W/V panels (double).
template <int NT, int E, typename T>
__global__ void __launch_bounds__(NT, (NT == 256 ? 2 : 4)) aca_kernel(const __grid_constant__ AcaLaunch L) {
  extern __shared__ __align__(128) double dyn[];
  __shared__ Shared sh;
  // dyn: row[kcap], then (unless L.dotg) per-warp dots[NT/32][kcap]
  constexpr int NW = NT / 32;
  const int b = L.cta_block ? (blockIdx.x < (unsigned)L.ncta ? L.cta_block[blockIdx.x] : L.nblocks)
                            : (int)(blockIdx.x / L.G);
  const int tid = threadIdx.x;
  if (b >= L.nblocks) return;
  const AcaBlock B = L.blocks[b];
  T* const BW = panel_of<T>(B.W);
  T* const BV = panel_of<T>(B.V);
  const int G = L.cta_block ? B.G : L.G;
  const int g = L.cta_block ? (int)blockIdx.x - B.g0 : (int)(blockIdx.x % L.G);
  const int64_t grp0 = L.cta_block ? B.g0 : (int64_t)b * G;
  AcaState* st = B.st;
  if (st->status != ACA_RUNNING && st->status != ACA_POST) return;
  const EntrySrc S = src_for(L.src, B.r0);  // the kernel of this block's system

  const int64_t ld = L.ld;
  const int m = B.m, n = B.n, ub = min(m, n);
  const double tol = L.tol, minPiv = L.minPivot;
  double* row = dyn;
  // per-warp dot partials: shared memory, or for large ranks this CTA's
  // slice of global memory (same writers and order: only the footprint moves)
  double* dotw = L.dotg ? L.dotg + (int64_t)blockIdx.x * L.dotg_stride : dyn + L.kcap_max;
  const int ldd = L.kcap_max;
  double* part_me = L.part + (int64_t)blockIdx.x * L.part_stride;
  const double* part_grp = L.part + grp0 * L.part_stride;
  unsigned* bar = L.bar + b;
  unsigned gen = 0;

  const int sm = (m + G - 1) / G, sn = (n + G - 1) / G;
  const int i_lo = min(m, g * sm), i_hi = min(m, i_lo + sm);
  const int j_lo = min(n, g * sn), j_hi = min(n, j_lo + sn);

  int k = st->k, cur = st->cur, iters = st->iters, status = st->status;
  double frob2 = st->frob2, eps = st->eps, margin = st->margin;
  double swp = st->swp, svp = st->svp;
  int near = st->near, pending = st->pending;
  bool nonfinite = false;

  const int minR = B.minRank, maxR = B.maxRank;  // -1: none (src/lowRank.cpp:149,244-247)
  if (status == ACA_RUNNING && k == 0 && maxR == 0) status = ACA_POST;  // zero columns, rank 1
  auto note_margin = [&](int kcount) {
    if (kcount < ub && kcount >= minR) {
      double gap = fabs(eps - tol) / tol;
      margin = fmin(margin, gap);
      if (gap < 1e-10) ++near;
    }
  };

  while (status == ACA_RUNNING) {
    // loop test of the reference, with epsilon_{k-1} possibly still pending
    if (!pending && !(eps > tol) && k >= minR) { status = ACA_POST; break; }
    if (k >= ub) { status = ACA_POST; break; }
    if (k >= B.kcap) {
      if (pending) {
        const int bk0 = 8 + (k & 1) * (2 * B.kcap + 2);
        dots_only_pass<NT>(L, BW, BV, k, i_lo, i_hi, j_lo, j_hi, B.kcap, part_me + bk0);
        if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }
        eps = resolve_eps<NT>(sh, L, B, part_grp, G, bk0, k, swp, svp, frob2);
        pending = 0;
        note_margin(k);
        if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }
        if (!(eps > tol) && k >= minR) { status = ACA_POST; break; }
      }
      status = ACA_NEED_CAP;  // paused: the host grows the capacity and resumes
      break;
    }
    ++iters;
    const bool fuse = pending && k >= 2;
    // Dot and norm partials alternate between two banks by step parity: a
    // slow CTA may still read step k-1's bank in its phase C while a fast one
    // already writes step k's in phase A.
    const int bk = 8 + (k & 1) * (2 * B.kcap + 2);
    // ---------------- phase A: residual row on this CTA's column slice
    if (g == 0 && tid == 0) B.cR[cur] = 1;
    for (int l = tid; l < k; l += NT) row[l] = (double)__ldcg(BW + cur + (int64_t)l * ld);
    if (fuse && j_lo >= j_hi)  // an empty slice contributes zero dots
      for (int e = tid; e < NW * (k - 1); e += NT) dotw[(e / (k - 1)) * ldd + e % (k - 1)] = 0.0;
    __syncthreads();
    const int gi = B.r0 + cur;
    double xi[3] = {0.0, 0.0, 0.0};
    if (!S.dense) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (d < S.kp.dim) xi[d] = __ldg(S.pts + d * S.ld + gi);
    }
    double bv = -1.0, sv = 0.0;
    int bi = INT_MAX, cand = INT_MAX;
    residual_pass<NT, E, true>(L, B, BV, j_lo, j_hi, k, row, fuse, dotw, ldd, gi, xi, 1.0,
                                 B.cC, bv, bi, cand, sv, nonfinite, S);
    __syncthreads();
    if (fuse)  // CTA partial dots of V, warps summed in order
      for (int l = tid; l < k - 1; l += NT) {
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += dotw[q * ldd + l];
        part_me[bk + l] = t;
      }
    block_argmax<NT>(sh, bv, bi);
    cand = block_min_int<NT>(sh, cand);
    sv = block_sum<NT>(sh, sv);
    if (tid == 0) {
      part_me[0] = bv;
      part_me[1] = (double)bi;
      part_me[2] = (bi != INT_MAX) ? (double)__ldcg(B.cC + bi) : 0.0;
      part_me[3] = (double)cand;
      part_me[bk + 2 * B.kcap + 1] = sv;
    }
    if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }

    // ---------------- phase B: pivot column, residual column on the row slice
    double mv;
    int mi, mflag, mcand;
    reduce_partials(sh, part_grp, L.part_stride, G, 0, mv, mi, mflag, mcand);
    if (mv <= minPiv) {
      // zero residual row (src/lowRank.cpp:187-195).  Whether the reference
      // even reached this step depends on epsilon_{k-1}: settle it first.
      if (pending) {
        dots_only_pass<NT>(L, BW, BV, k, i_lo, i_hi, j_lo, j_hi, B.kcap, part_me + bk);
        if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }
        eps = resolve_eps<NT>(sh, L, B, part_grp, G, bk, k, swp, svp, frob2);
        pending = 0;
        note_margin(k);
        if (!(eps > tol) && k >= minR) {
          --iters;
          status = ACA_POST;
          break;
        }
      }
      int f = INT_MAX;
      for (int i = tid; i < m; i += NT)
        if (__ldcg(B.cR + i) == 0) { f = i; break; }
      f = block_min_int<NT>(sh, f);
      if (f == INT_MAX) { status = ACA_POST; break; }
      cur = f;
      if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }
      continue;
    }
    int cc;
    if (!mflag) {
      cc = mi;
    } else {
      // whichever way epsilon_{k-1} goes, the rank is k (src/lowRank.cpp:200-202)
      if (mcand == INT_MAX) { status = ACA_POST; break; }
      cc = mcand;
    }
    if (g == 0 && tid == 0) B.cC[cc] = 1;
    const double piv = __ddiv_rn(1.0, (double)__ldcg(BV + cc + (int64_t)k * ld));
    for (int l = tid; l < k; l += NT) row[l] = (double)__ldcg(BV + cc + (int64_t)l * ld);
    if (fuse && i_lo >= i_hi)
      for (int e = tid; e < NW * (k - 1); e += NT) dotw[(e / (k - 1)) * ldd + e % (k - 1)] = 0.0;
    __syncthreads();
    const int gj = B.c0 + cc;
    double xj[3] = {0.0, 0.0, 0.0};
    if (!S.dense) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (d < S.kp.dim) xj[d] = __ldg(S.pts + d * S.ld + gj);
    }
    bv = -1.0;
    bi = INT_MAX;
    cand = INT_MAX;
    double sw = 0.0;
    residual_pass<NT, E, false>(L, B, BW, i_lo, i_hi, k, row, fuse, dotw, ldd, gj, xj, piv,
                                  B.cR, bv, bi, cand, sw, nonfinite, S);
    __syncthreads();
    if (fuse)
      for (int l = tid; l < k - 1; l += NT) {
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += dotw[q * ldd + l];
        part_me[bk + B.kcap + l] = t;
      }
    block_argmax<NT>(sh, bv, bi);
    cand = block_min_int<NT>(sh, cand);
    sw = block_sum<NT>(sh, sw);
    if (tid == 0) {
      part_me[4] = bv;
      part_me[5] = (double)bi;
      part_me[6] = (bi != INT_MAX) ? (double)__ldcg(B.cR + bi) : 0.0;
      part_me[7] = (double)cand;
      part_me[bk + 2 * B.kcap] = sw;
    }
    if (!group_sync(L, bar, G, gen, L.err)) { status = ACA_ERROR; break; }

    // ---------------- phase C: epsilon of step k-1, then step k's next row
    if (pending) {
      eps = fuse ? resolve_eps<NT>(sh, L, B, part_grp, G, bk, k, swp, svp, frob2)
                 : [&]() {  // k == 1: no earlier columns, the dots are empty
                     frob2 += swp * svp;
                     return sqrt(swp) * sqrt(svp) / sqrt(frob2);
                   }();
      pending = 0;
      note_margin(k);
      if (!(eps > tol) && k >= minR) {  // step k is discarded: the reference stopped before it
        --iters;
        status = ACA_POST;
        break;
      }
    }
    int nflag, ncand, ni;
    double nv;
    reduce_partials(sh, part_grp, L.part_stride, G, 4, nv, ni, nflag, ncand);
    const int nr = nflag ? ncand : ni;
    if (nr == INT_MAX) {  // no admissible next row: stop before storing (src/lowRank.cpp:226-227)
      status = ACA_POST;
      break;
    }
    double swt = 0.0, svt = 0.0;
    for (int q = 0; q < G; ++q) {
      swt += __ldcg(part_grp + q * L.part_stride + bk + 2 * B.kcap);
      svt += __ldcg(part_grp + q * L.part_stride + bk + 2 * B.kcap + 1);
    }
    if (g == 0 && tid == 0) {
      B.prow[k] = cur;
      B.pcol[k] = cc;
    }
    swp = swt;
    svp = svt;
    pending = 1;
    cur = nr;
    ++k;
    if (k == maxR) {  // the rank ceiling: stop without the last epsilon (src/lowRank.cpp:244-247)
      pending = 0;
      status = ACA_POST;
      break;
    }
    // No barrier needed here: the next writes to the partials come after
    // every CTA has passed barrier 2, and W(:,k) / V(:,k) are final.
  }

  int rank = k;
  if (status == ACA_POST)
    status = aca_post_process<T>(B, S, BW, BV, ld, k, i_lo, i_hi, j_lo, j_hi, NT, &rank);
  if (nonfinite) atomicOr(L.err, DEV_ERR_NONFINITE);
  // Every CTA of the group reached the same state; CTA 0 records it after a
  // last barrier, so that no CTA of the group can still be about to read the
  // entry state (a block that starts in post-processing has no barrier before).
  if (status != ACA_ERROR && !group_sync(L, bar, G, gen, L.err)) status = ACA_ERROR;
  if (g == 0 && tid == 0) {
    st->k = k;
    st->cur = cur;
    st->iters = iters;
    st->status = status;
    st->frob2 = frob2;
    st->eps = eps;
    st->margin = margin;
    st->near = near;
    st->rank = rank;
    st->swp = swp;
    st->svp = svp;
    st->pending = pending;
  }
}

}  // namespace

static size_t aca_smem(int nt, int kcap_max, bool global_dots) {
  return sizeof(double) * (size_t)(global_dots ? 1 : 1 + nt / 32) * (size_t)kcap_max;
}

// The per-warp dot partials move to global memory once the CTA's shared
// memory would pass 100 KB (beyond that fewer than two 256-thread CTAs fit on
// an SM).
bool aca_dots_global(int nt, int kcap_max) { return aca_smem(nt, kcap_max, false) > 100 * 1024; }

size_t aca_smem_bytes(int nt, int kcap_max) {
  return aca_smem(nt, kcap_max, aca_dots_global(nt, kcap_max));
}

static const void* aca_fn(int nt, bool narrow) {
  if (nt == 256)
    return narrow ? (const void*)aca_kernel<256, 2, double> : (const void*)aca_kernel<256, 4, double>;
  return (const void*)aca_kernel<128, 2, double>;
}

// Dynamic shared memory above 48 KB; the default shared-memory carveout
// otherwise, for its larger L1 (the panels are loaded per thread).
static int set_smem(const void* fn, size_t smem) {
  cudaError_t e = smem_opt_in(fn, smem);
  if (e != cudaSuccess) cudaGetLastError();  // consume it: later launch checks stay clean
  return (int)e;
}

int aca_launch(const AcaLaunch& L, int nt, int kcap_max, bool cooperative, cudaStream_t s) {
  const size_t smem = aca_smem(nt, kcap_max, L.dotg != nullptr);
  dim3 grid(L.cta_block ? L.ncta : L.nblocks * L.G), block(nt);
  void* args[] = {(void*)&L};
  const void* fn = aca_fn(nt, L.narrow != 0);
  if (int e = set_smem(fn, smem)) return e;
  cudaError_t e = cooperative ? cudaLaunchCooperativeKernel(fn, grid, block, args, smem, s)
                              : cudaLaunchKernel(fn, grid, block, args, smem, s);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

int aca_max_coresident(int nt, int kcap_max, int* per_sm) {
  const size_t smem = aca_smem_bytes(nt, kcap_max);
  const void* fn = aca_fn(nt, false);
  *per_sm = 0;
  if (int e = set_smem(fn, smem)) return e;
  int nb = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, nt, smem);
  if (e != cudaSuccess) cudaGetLastError();
  *per_sm = nb;
  return e == cudaSuccess ? 0 : (int)e;
}
