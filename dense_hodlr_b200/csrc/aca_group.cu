// Partial-pivot ACA of the blocks that a group of CTAs shares (the upper tree
// levels), one group per block.  The same loop, values and pivots as
// aca_kernel (aca.cu): entries and residual sums are formed by the same
// separately rounded operations in the same order.
//
// What bounds it: a step streams the block's W and V panels once (HBM or L2
// bytes) and has two points where every CTA of the group needs what all the
// others found (the row maximum, then the column maximum).  So:
//
// * Panel bytes.  CTA g owns a slice of the block's rows (W) and columns (V).
//   A slice is cut into chunks (GroupCfg::ROWS) and streamed, TC panel columns
//   at a time, through one ring in shared memory that the whole CTA shares: a
//   tile is exactly the slice's rows, whatever their number, so no
//   byte is fetched that is not used.  While a launch runs, slices are kept
//   tile after tile (GroupSlice), not as columns of the level's arenas: a
//   column's piece of a slice is 1 to 2 KB, 8 N bytes from the next one, and
//   148 CTAs streaming such pieces reached 28 GB/s an SM from HBM, against the
//   44 of a plain copy.  The ring's copy warp runs ahead into
//   the next pass: after a row pass the column pass of the same step is
//   certain (unless the residual row is zero), after a column pass the next
//   step's row pass, and both read only columns that are final.  Its tiles
//   cross the exchange between them, so the bytes of the next pass arrive
//   while the CTAs wait for each other.
// * Warp roles.  SW sum warps hold E rows a thread (the sum over the earlier
//   columns is a chain in l order, so rows are the parallelism); the norm
//   update's dots come from two sets of dot warps that take alternate tiles
//   (E = 1), or from the sum warps (E = 4); one warp copies; the exchange warp
//   talks to the other CTAs and, with the other reduce warps, sums dots.
// * Exchanges.  A CTA's result is one slot of three 16-byte words that each
//   carry the exchange's number, read and written whole (128-bit accesses), so
//   an exchange is one store and one load latency, with no fence in between.
//   While the exchange warp waits, the others publish the row of the panel
//   that the next pass needs if this CTA's candidate wins, one tagged word a
//   column: the winner's row is then read in one piece instead of every CTA
//   gathering it with the panel's stride (a 2^21-byte stride at N = 262144: 33
//   us a pass).  What else one CTA writes and another reads (dots) is
//   published half a step later, by a fence of the exchange warp that nobody
//   waits for.
// * The stopping test of a step needs, for every earlier column, the sum of
//   its dot over the group.  CTA g sums the columns of its share while the
//   next step's column pass streams, and the shares' sums travel with that
//   pass's exchange: epsilon of a step is known one step later, and the work
//   begun meanwhile is discarded if the loop had ended (the same ranks,
//   pivots and iteration counts).
// * Pauses.  Blocks of a long launch pause so that the host shares the CTAs anew:
//   once a third of them are out of work, which depends on the clock, or (AcaBlock::
//   kstop) at a column count.  A block goes on in a group of another size, which adds
//   the norms and dots up in another order: with pauses by the clock the last bits of
//   epsilon differ from run to run, and a rank can where epsilon is within rounding
//   of the tolerance (counted: AcaState::near).  W, V and the pivots up to there are
//   the same bits whatever the groups.
//
// Measured on B200, all group levels of one compression, against per-warp
// rings of 128-row tiles (panels loaded per thread for an odd N), a counter
// barrier, a sum of all CTAs' dots in every CTA, and one launch a level:
// N = 20011 2D Matern-3/2 tol 1e-8 15 ms (90), sphere N = 16384 tol 1e-10 113
// ms (796), 3D Gaussian N = 40000 89 ms (288), 1D N = 4096 0.3 ms (1.7),
// 2D N = 262144 111 ms (142).
#include "aca_post.cuh"
#include "common.cuh"
#include "hodlr_internal.h"

enum { ACA_GROUP_NONE = 0, ACA_GROUP_8x1, ACA_GROUP_8x4 };

namespace {

constexpr int GR_SMAX = 16;  // most stages of a ring
constexpr int GR_SMIN = 3;

// SW sum warps of E rows a thread.  E = 1: the dots are formed by warps of
// their own from the same tiles.  E = 4: a sum thread's four rows make the
// reduction over the warp cheap enough to form them in place, and the tile is
// read from shared memory once.
template <int SW_, int E_>
struct GroupCfg {
  static constexpr int SW = SW_, E = E_;
  static constexpr int TC = E == 1 ? 16 : 4;  // panel columns of a tile
  static constexpr int DT = E == 1 ? SW / 2 : 0;  // dot warps that share a tile
  static constexpr int DW = 2 * DT;         // all of them: alternate tiles
  static constexpr int RW = 2;
  static constexpr int COPY = SW + DW;      // the copy warp
  static constexpr int EX = COPY + 1;       // the exchange warp, first of the RW reduce warps
  static constexpr int NT = 32 * (SW + DW + 1 + RW);
  static constexpr int ROWS = 32 * SW * E;  // most rows of a chunk
  static constexpr int DC = E == 1 ? TC / (DT > 0 ? DT : 1) : 4;  // tile columns of a dot warp
};

struct GroupShared {
  double red_v[8], red_s[8];
  int red_i[8], red_c[8];
  double lag[4];         // the reduce warps' shares of the lagging norm update
  // the group's result of an exchange
  double mv;
  int mi, mflag, mcand, fail, imin, stop, yield;
  // the stopping test, kept by thread 0: squared norms of column k-1 (its
  // epsilon pending) and of column k-2 (its epsilon lagging), and of the row
  // residual of this step
  double frob2, eps, margin, swp, svp, swl, svl, svt;
  int near;
};

// What one turn of a CTA's loop does: a row or a column pass; a fence (all that
// the group wrote before is visible after it); the sum of the lagging or the
// pending epsilon's dots; the scan for the first row not chosen yet.  Each
// ends in one exchange.
enum { OP_TOP = 0, OP_ROW, OP_COL, OP_FENCE, OP_LAG, OP_PEND, OP_SCAN };
// Where a fenced sum was asked for, and how the loop goes on after it.
enum { AT_CAP = 0, AT_ROW, AT_END, AT_MAX };

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait on an mbarrier phase; once the error word is set, waits give
// up soon, so that a failed launch ends quickly (its next exchange fails).
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, unsigned* err) {
  if (mbar_try_wait(bar, parity)) return;
  for (uint32_t polls = 0;; ++polls) {
    if (mbar_try_wait(bar, parity)) return;
    if (polls >= (1u << 20) || ((polls & 63) == 63 && *(volatile unsigned*)err)) {
      atomicOr(err, DEV_ERR_TIMEOUT);
      return;
    }
    if (polls >= 64) __nanosleep(64);
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Argmax over a warp (value >= 0, or -1 with index INT_MAX for none; the
// lowest index wins ties), the result in every lane: the order of doubles
// >= 0 is that of their bits.
__device__ __forceinline__ void warp_argmax_all(double& v, int& i) {
  const unsigned m = 0xffffffffu;
  const bool none = i == INT_MAX;
  const unsigned hi = none ? 0u : (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(m, hi);
  const unsigned ml = __reduce_max_sync(m, !none && hi == mh ? lo : 0u);
  const int mi = __reduce_min_sync(m, !none && hi == mh && lo == ml ? i : INT_MAX);
  v = mi == INT_MAX ? -1.0 : __hiloint2double((int)mh, (int)ml);
  i = mi;
}
__device__ __forceinline__ double warp_sum_all(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ void st_b128(void* p, uint64_t lo, uint64_t hi) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(lo), "l"(hi)
      : "memory");
}
__device__ __forceinline__ void ld_b128(const void* p, uint64_t& lo, uint64_t& hi) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
}

// The ring as one warp sees it: tiles consumed (and, in the copy warp,
// issued) so far, as a slot and the parity of its current use.
struct GroupRing {
  double* buf;
  uint64_t* full;
  uint64_t* empty;
  int stages, stage_elems;
  int slot;          // of the next tile to consume
  uint32_t parity;
  int islot;         // copy warp: of the next tile to issue
  uint32_t iparity;
  uint32_t issued;   // copy warp: tiles issued (all of them)
  int ahead;         // tiles of the expected next pass already issued
  int ekind, ek;     // that pass: 0 row / 1 column, and its column count
  __device__ void step() {
    if (++slot == stages) {
      slot = 0;
      parity ^= 1u;
    }
  }
};

// A CTA's slice [lo, hi) of a block's panel (`per` rows a CTA), in the launch's
// working layout: chunks of `cr` rows (a multiple of 16), each chunk's columns
// one after the other, so that a tile is one contiguous piece of memory.
// Column l of row lo + c cr + t is at Q[(c kcap + l) cr + t].
struct GroupSlice {
  double* Q;
  int lo, hi, per, cr, chunks, kcap;
  __device__ double* column(int c, int l) const { return Q + ((int64_t)c * kcap + l) * cr; }
};

__host__ __device__ inline int slice_chunks(int per, int most) { return (per + most - 1) / most; }
__host__ __device__ inline int slice_pitch(int per, int most) {
  const int c = slice_chunks(per, most);
  return ((per + c - 1) / c + 15) & ~15;
}

template <class C>
__device__ GroupSlice make_slice(double* scratch, int64_t stride, int g, int rows, int G, int kcap) {
  const int per = (rows + G - 1) / G, lo = min(rows, g * per), hi = min(rows, lo + per);
  const int cr = slice_pitch(per, C::ROWS);
  return GroupSlice{scratch + g * stride, lo, hi, per, cr, (hi - lo + cr - 1) / cr, kcap};
}

// The columns [0, k) of a slice from or to the level's arena P (row 0 of the
// block, leading dimension ld), by all threads.
__device__ inline void slice_copy(const GroupSlice& s, double* P, int64_t ld, int k, bool in,
                                  int nt) {
  constexpr int U = 16;  // columns in flight
  const int groups = max(1, nt / s.cr), grp = min((int)threadIdx.x / s.cr, groups);
  if (grp >= groups && groups > 1) return;
  for (int c = 0; c < s.chunks; ++c) {
    const int j0 = s.lo + c * s.cr, cnt = min(s.cr, s.hi - j0);
    for (int t = groups > 1 ? (int)threadIdx.x - grp * s.cr : (int)threadIdx.x; t < cnt;
         t += groups > 1 ? s.cr : nt)
      for (int l0 = groups > 1 ? grp * U : 0; l0 < k; l0 += groups * U) {
        double* q = s.column(c, l0) + t;
        double* p = P + j0 + t + (int64_t)l0 * ld;
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (l0 + u < k) v[u] = in ? p[(int64_t)u * ld] : q[u * s.cr];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (l0 + u < k) {
            if (in)
              q[u * s.cr] = v[u];
            else
              p[(int64_t)u * ld] = v[u];
          }
      }
  }
}

// The copy warp: tile `idx` of a pass over the first k columns of a slice
// (chunk idx / tpc, columns TC (idx % tpc) ..) into the ring's next slot, by
// one bulk copy: cr is a multiple of 16, so both ends are 16-byte aligned.
template <class C>
__device__ void ring_issue(GroupRing& R, const GroupSlice& s, int k, int idx, unsigned* err) {
  const int tpc = (k + C::TC - 1) / C::TC;
  const int ch = idx / tpc, l0 = (idx % tpc) * C::TC, nc = min(C::TC, k - l0);
  const uint32_t bytes = (uint32_t)(nc * s.cr) * (uint32_t)sizeof(double);
  if (R.issued >= (uint32_t)R.stages) mbar_wait(R.empty + R.islot, R.iparity ^ 1u, err);
  uint64_t* bar = R.full + R.islot;
  if ((threadIdx.x & 31) == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(saddr(R.buf + (size_t)R.islot * R.stage_elems)),
        "l"(s.column(ch, l0)), "r"(bytes), "r"(saddr(bar))
        : "memory");
  }
  __syncwarp();
  ++R.issued;
  if (++R.islot == R.stages) {
    R.islot = 0;
    R.iparity ^= 1u;
  }
}

// The coefficients of a pass: column l's is element l of a panel row, read
// where the row's owner published it (tagged words), or from the panel.
struct CoefSrc {
  const unsigned char* pub;  // null: from the panel
  uint64_t tag;
  const double* pan;         // the row in its owner's slice
  int stride;
};

__device__ __forceinline__ double coef_load(const CoefSrc& cs, int l, const AcaLaunch& L) {
  if (!cs.pub) return __ldcg(cs.pan + (int64_t)l * cs.stride);
  uint64_t v = 0, t = 0;
  for (unsigned polls = 0;; ++polls) {
    ld_b128(cs.pub + (size_t)l * 16, v, t);
    if (t == cs.tag) break;
    if (polls >= L.spin_limit || ((polls & 63) == 63 && *(volatile unsigned*)L.err)) {
      atomicOr(L.err, DEV_ERR_TIMEOUT);
      break;
    }
    if (polls >= 256) __nanosleep(100);
  }
  return __longlong_as_double((long long)v);
}

__device__ __forceinline__ void bar_all() { asm volatile("bar.sync 0;" ::: "memory"); }

// Four column sums over the warp in one transposed reduction: after the
// exchanges at offsets 16 and 8, lanes 8 u .. 8 u + 7 hold partial sums of
// column u; lane 8 u returns its sum, u = lane / 8.
__device__ __forceinline__ double sum4_over_warp(const double (&d)[4], int lane) {
  const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
  const double s0 = __shfl_xor_sync(0xffffffffu, hi16 ? d[0] : d[2], 16);
  const double s1 = __shfl_xor_sync(0xffffffffu, hi16 ? d[1] : d[3], 16);
  const double p0 = (hi16 ? d[2] : d[0]) + s0;
  const double p1 = (hi16 ? d[3] : d[1]) + s1;
  const double s2 = __shfl_xor_sync(0xffffffffu, hi8 ? p0 : p1, 8);
  double t = (hi8 ? p1 : p0) + s2;
  t += __shfl_xor_sync(0xffffffffu, t, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  return t;
}

// One residual pass over the first k columns of this CTA's slice (see
// residual_pass in aca.cu).
struct Pass {
  bool row;            // row pass (V slice) or column pass (W slice)
  int k, fixed, base;  // columns; the pivot row's or column's point; row 0's point
  bool dots;           // form the dots of column k-1 with the earlier ones
  CoefSrc cs;
  const unsigned char* chosen;
  double* dout;        // E = 1: where the dots go
  double* dotw;        // E = 4: the dots of every chunk and warp, kcap_max apart
};

// Sum warps:  r[j] = entry(j) - sum_{l<k} coef[l] P(j, l),  P(j, k) = r or
// r / coef[k] (a column pass), and in sh the argmax, the first admissible row
// and the sum of squares.  The entries of the first chunk are evaluated while
// the coefficients arrive.
template <class C>
__device__ __forceinline__ void sum_role(const AcaLaunch& L, const EntrySrc& S, const Pass& p,
                                         const GroupSlice& s, const double* coef,
                                         const double* xs, const unsigned char* fl, GroupRing& R,
                                         GroupShared& sh, bool& nonfinite) {
  constexpr int E = C::E, TC = C::TC;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, k = p.k;
  const int tpc = (k + TC - 1) / TC, kd = p.dots ? k - 1 : 0;
  const int t0 = 32 * E * w + lane;  // rows t0 + 32 e of a chunk
  double xf[3] = {0.0, 0.0, 0.0};
  if (!S.dense) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (d < S.kp.dim) xf[d] = __ldg(S.pts + d * S.ld + p.fixed);
  }
  double bv = -1.0, sq = 0.0, scale = 1.0;
  int bi = INT_MAX, cand = INT_MAX;
  if (s.chunks == 0) bar_all();
  for (int c = 0; c < s.chunks; ++c) {
    const int xb = s.lo + c * s.cr;
    double ent[E], acc[E], vp[E];
    int ch[E];
    bool ok[E];
    double xp[E][3];
#pragma unroll
    for (int e = 0; e < E; ++e) {  // all loads first
      const int t = t0 + 32 * e, j = xb + t, gj = p.base + j;
      ok[e] = t < s.cr && j < s.hi;
      acc[e] = 0.0;
      vp[e] = E > 1 && ok[e] && kd > 0 ? s.column(c, k - 1)[t] : 0.0;
      const bool cached = E == 1 && c == 0;
      ch[e] = !ok[e] ? 0 : cached ? (int)fl[t] : (int)__ldcg(p.chosen + j);
      if (S.dense) {
        ent[e] = ok[e] ? __ldg(S.A + (int64_t)(p.row ? gj : p.fixed) * S.ld +
                               (p.row ? p.fixed : gj))
                       : 0.0;
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          xp[e][d] = !ok[e] || d >= S.kp.dim ? 0.0
                     : cached                ? xs[d * C::ROWS + t]
                                             : __ldg(S.pts + d * S.ld + gj);
      }
    }
    if (!S.dense) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        // the squared distance is the same bits either way round
        double r2 = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (d < S.kp.dim) {
            const double q = __dsub_rn(xf[d], xp[e][d]);
            r2 = __dadd_rn(r2, __dmul_rn(q, q));
          }
        ent[e] = hx_kernel_r2(S.kp, r2);
        if (p.base + xb + t0 + 32 * e == p.fixed)
          ent[e] = S.kp.diag_replace ? S.kp.diag_value : __dadd_rn(ent[e], S.kp.shift);
      }
    }
    if (c == 0) {
      bar_all();  // the coefficients are in shared memory
      if (!p.row) scale = __ddiv_rn(1.0, coef[k]);
    }
    const bool live = 32 * E * w < s.cr;  // some lane of this warp has a row
    // lanes without a row read the slice's last one: the padding of a chunk
    // may hold what is not a number, which a product with 0 would keep
    const int thi = min(s.cr, s.hi - xb) - 1;
    for (int q = 0; q < tpc; ++q) {
      mbar_wait(R.full + R.slot, R.parity, L.err);
      const double* tile = R.buf + (size_t)R.slot * R.stage_elems;
      const int l0 = q * TC;
      if (live) {
        if (E == 1) {
          const double* tt = tile + min(t0, thi);
#pragma unroll
          for (int h = 0; h < TC; h += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = tt[(h + u) * s.cr];
            if (l0 + h + 8 <= k) {
#pragma unroll
              for (int u = 0; u < 8; u += 2) {
                const double2 cf = *reinterpret_cast<const double2*>(coef + l0 + h + u);
                acc[0] = __dadd_rn(acc[0], __dmul_rn(cf.x, v[u]));
                acc[0] = __dadd_rn(acc[0], __dmul_rn(cf.y, v[u + 1]));
              }
            } else {  // columns past k: whatever the stage holds, not added
#pragma unroll
              for (int u = 0; u < 8; u += 2) {
                const double2 cf = *reinterpret_cast<const double2*>(coef + l0 + h + u);
                const double a0 = __dadd_rn(acc[0], __dmul_rn(cf.x, v[u]));
                acc[0] = l0 + h + u < k ? a0 : acc[0];
                const double a1 = __dadd_rn(acc[0], __dmul_rn(cf.y, v[u + 1]));
                acc[0] = l0 + h + u + 1 < k ? a1 : acc[0];
              }
            }
          }
        } else {
          double v[TC][E];
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const double* tt = tile + min(t0 + 32 * e, thi);
#pragma unroll
            for (int u = 0; u < TC; ++u) v[u][e] = tt[u * s.cr];
          }
#pragma unroll
          for (int u = 0; u < TC; ++u) {
            const double cf = coef[l0 + u];
            if (l0 + u < k) {
#pragma unroll
              for (int e = 0; e < E; ++e) acc[e] = __dadd_rn(acc[e], __dmul_rn(cf, v[u][e]));
            }
          }
          if (l0 < kd) {
            double d[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              d[u] = 0.0;
#pragma unroll
              for (int e = 0; e < E; ++e) d[u] = fma(v[u][e], vp[e], d[u]);
            }
            const double t = sum4_over_warp(d, lane);
            const int l = l0 + (lane >> 3);
            if ((lane & 7) == 0 && l < kd) p.dotw[(int64_t)(c * C::SW + w) * L.kcap_max + l] = t;
          }
        }
      } else if (E > 1 && lane < 4 && l0 + lane < kd) {
        p.dotw[(int64_t)(c * C::SW + w) * L.kcap_max + l0 + lane] = 0.0;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(R.empty + R.slot);
      R.step();
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (!ok[e]) continue;
      const int j = xb + t0 + 32 * e;
      const double r = __dsub_rn(ent[e], acc[e]);
      const double stored = p.row ? r : __dmul_rn(scale, r);
      s.column(c, k)[t0 + 32 * e] = stored;
      sq = fma(stored, stored, sq);
      const double a = fabs(r);
      nonfinite |= !isfinite(r);
      if (a > bv) {  // increasing j per thread: the first maximum
        bv = a;
        bi = 2 * j + ch[e];  // the row, and whether it was chosen before
      }
      if (cand == INT_MAX && a > L.minPivot && ch[e] == 0) cand = j;
    }
  }
  // this thread's stores before later bulk copies of the same rows
  asm volatile("fence.proxy.async.global;" ::: "memory");
  warp_argmax_all(bv, bi);
  sq = warp_sum_all(sq);
  cand = __reduce_min_sync(0xffffffffu, cand);
  if (lane == 0) {
    sh.red_v[w] = bv;
    sh.red_i[w] = bi;
    sh.red_c[w] = cand;
    sh.red_s[w] = sq;
  }
}

// Dot warps (E = 1): rows over lanes, DC columns of every second tile.
template <class C>
__device__ __forceinline__ void dot_role(const AcaLaunch& L, const Pass& p, const GroupSlice& s,
                                         double* dsm, GroupRing& R) {
  const int lane = threadIdx.x & 31, dw = (int)(threadIdx.x >> 5) - C::SW;
  const int set = dw / C::DT, d0 = (dw % C::DT) * C::DC, k = p.k;
  const int tpc = (k + C::TC - 1) / C::TC, kd = p.dots ? k - 1 : 0;
  double vp[C::SW];
  if (s.chunks == 0 || kd <= 0) bar_all();
  for (int c = 0; c < s.chunks; ++c) {
    const int xb = s.lo + c * s.cr, cnt = min(s.cr, s.hi - xb);
    if (kd > 0) {
#pragma unroll
      for (int i = 0; i < C::SW; ++i) {
        const int t = lane + 32 * i;
        vp[i] = t < cnt ? s.column(c, k - 1)[t] : 0.0;
      }
      if (c == 0) bar_all();
    }
    for (int q = 0; q < tpc; ++q) {
      // every warp waits for and frees every tile, its own or not: one that
      // skipped tiles could run ahead of a copy still in flight, or fall two
      // uses of a stage behind, and mistake the barrier's phase
      mbar_wait(R.full + R.slot, R.parity, L.err);
      if ((q & 1) != set) {
        __syncwarp();
        if (lane == 0) mbar_arrive(R.empty + R.slot);
        R.step();
        continue;
      }
      const int l0 = q * C::TC + d0;
      const double* tile = R.buf + (size_t)R.slot * R.stage_elems + d0 * s.cr;
#pragma unroll
      for (int g4 = 0; g4 < C::DC; g4 += 4) {
        if (l0 + g4 >= kd) break;
        // a column past kd sums what the stage holds and is not stored
        double d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int h = 0; h < C::SW; h += 2) {
          if (32 * h >= cnt) break;
          // lanes without a row: the slice's last one, times 0 (see sum_role)
          const double* t0 = tile + g4 * s.cr + min(lane + 32 * h, cnt - 1);
          const double* t1 = tile + g4 * s.cr + min(lane + 32 * h + 32, cnt - 1);
          double v[2][4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            v[0][u] = t0[u * s.cr];
            v[1][u] = t1[u * s.cr];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) d[u] = fma(v[1][u], vp[h + 1], fma(v[0][u], vp[h], d[u]));
        }
        const double t = sum4_over_warp(d, lane);
        const int l = l0 + g4 + (lane >> 3);
        if ((lane & 7) == 0 && l < kd) {
          if (c == 0)
            dsm[l] = t;
          else
            dsm[l] += t;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(R.empty + R.slot);
      R.step();
    }
  }
  // this CTA's dots, each column by the warp that summed it
  __syncwarp();
  for (int e = lane; e < (tpc + 1) / 2 * C::DC; e += 32) {
    const int l = (2 * (e / C::DC) + set) * C::TC + d0 + e % C::DC;
    if (l < kd) p.dout[l] = s.chunks > 0 ? dsm[l] : 0.0;
  }
}

// The group's norm update sum_l (w . W_l)(V_l . v) of the `nd` dots in the
// bank at `bk` of every CTA's partials: CTA g sums columns [g per, g per + per)
// over the group (the reduce warps, in a fixed order) and leaves the shares
// in sh.lag; the next exchange adds them up.
template <class C>
__device__ __forceinline__ void lag_share(const AcaLaunch& L, int g0, int G, int64_t bk, int nd,
                                          GroupShared& sh) {
  const int r = (int)(threadIdx.x >> 5) - C::EX, lane = threadIdx.x & 31;
  const double* part = L.part + (int64_t)g0 * L.part_stride + bk;
  const int g = (int)blockIdx.x - g0;
  double acc = 0.0;
  if (G == 1) {
    for (int l = 32 * r + lane; l < nd; l += 32 * C::RW)
      acc = fma(__ldcg(part + L.kcap_max + l), __ldcg(part + l), acc);
  } else {
    const int per = (nd + G - 1) / G, lb = g * per, le = min(nd, lb + per);
    constexpr int U = 4;
    for (int l = lb + r * U; l < le; l += C::RW * U) {
      double dv[U], dw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) dv[u] = dw[u] = 0.0;
      for (int q = lane; q < G; q += 32) {
        const double* p = part + q * L.part_stride + l;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (l + u < le) {
            dv[u] += __ldcg(p + u);
            dw[u] += __ldcg(p + L.kcap_max + u);
          }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        dv[u] = warp_sum_all(dv[u]);
        dw[u] = warp_sum_all(dw[u]);
        if (lane == 0) acc = fma(dw[u], dv[u], acc);
      }
    }
  }
  acc = warp_sum_all(acc);
  if (lane == 0) sh.lag[r] = acc;
}

// Dots of column k-1 over this CTA's slices when no pass could form them (a
// zero residual row, the capacity limit), into its bank.
template <class C>
__device__ void group_dots(const AcaLaunch& L, const GroupSlice& sV, const GroupSlice& sW, int k,
                           double* bank) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int l = w; l < k - 1; l += C::NT / 32)
    for (int q = 0; q < 2; ++q) {
      const GroupSlice& s = q ? sW : sV;
      double a = 0.0;
      for (int c = 0; c < s.chunks; ++c) {
        const double *x = s.column(c, l), *y = s.column(c, k - 1);
        const int cnt = min(s.cr, s.hi - s.lo - c * s.cr);
        for (int t = lane; t < cnt; t += 32) a = fma(x[t], y[t], a);
      }
      a = warp_sum(a);
      if (lane == 0) bank[q * L.kcap_max + l] = a;
    }
}

template <int SW, int E>
__global__ void __launch_bounds__(GroupCfg<SW, E>::NT, 1)
    aca_group_kernel(const __grid_constant__ AcaLaunch L) {
  using C = GroupCfg<SW, E>;
  extern __shared__ __align__(128) double dyn[];
  __shared__ GroupShared sh;
  __shared__ AcaBlock B;
  __shared__ EntrySrc S;
  __shared__ GroupSlice sl[2];  // of V (row passes) and of W (column passes)
  __shared__ __align__(8) uint64_t bars[2 * GR_SMAX];
  __shared__ double xs[E == 1 ? 2 * 3 * C::ROWS : 1];       // first chunks' points
  __shared__ unsigned char fl[E == 1 ? 2 * C::ROWS : 1];    // and chosen flags
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  {
    const int b = L.cta_block ? L.cta_block[blockIdx.x] : (int)(blockIdx.x / L.G);
    if (b >= L.nblocks) return;
    if (tid == 0) {
      B = L.blocks[b];
      if (!L.cta_block) {
        B.G = L.G;
        B.g0 = b * L.G;
      }
      S = src_for(L.src, B.r0);
    }
  }
  __syncthreads();
  AcaState* const st = B.st;
  if (st->status != ACA_RUNNING && st->status != ACA_POST) return;
  const int G = B.G, g = (int)blockIdx.x - B.g0;
  double* coef = dyn + (size_t)L.ring_stages * L.stage_elems;
  double* dsm = coef + ((L.kcap_max + 16) & ~15);
  const int ub = min(B.m, B.n);

  GroupRing R{dyn, bars, bars + GR_SMAX, L.ring_stages, L.stage_elems, 0, 0, 0, 0, 0, 0, 0, -1};
  if (tid == 0) {
    sl[1] = make_slice<C>(B.sW, B.strW, g, B.m, G, B.kcap);
    sl[0] = make_slice<C>(B.sV, B.strV, g, B.n, G, B.kcap);
    for (int q = 0; q < L.ring_stages; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(R.full + q)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(R.empty + q)),
                   "r"(C::COPY));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int r = 0; r < 4; ++r) sh.lag[r] = 0.0;
    sh.frob2 = st->frob2;
    sh.eps = st->eps;
    sh.margin = st->margin;
    sh.swp = st->swp;
    sh.svp = st->svp;
    sh.swl = sh.svl = sh.svt = 0.0;
    sh.near = st->near;
    sh.stop = !(st->eps > L.tol) && st->k >= B.minRank;
    sh.fail = sh.yield = 0;
  }
  __syncthreads();
  if (E == 1)
    for (int q = 0; q < 2; ++q)
      for (int t = tid; t < C::ROWS; t += C::NT) {
        const int j = sl[q].lo + t;
        const bool in = j < sl[q].hi;
        fl[q * C::ROWS + t] = in ? (q ? B.cR : B.cC)[j] : 0;
        if (!S.dense)
          for (int d = 0; d < S.kp.dim; ++d)
            xs[(q * 3 + d) * C::ROWS + t] = in ? S.pts[d * S.ld + (q ? B.r0 : B.c0) + j] : 0.0;
      }
  if (st->k > 0) {  // resumed: the columns so far
    slice_copy(sl[0], B.V, L.ld, st->k, true, C::NT);
    slice_copy(sl[1], B.W, L.ld, st->k, true, C::NT);
    asm volatile("fence.proxy.async.global;" ::: "memory");
  }
  __syncthreads();

  int k = st->k, cur = st->cur, iters = st->iters, status = st->status;
  // pending: the dots of column k-1 are not formed yet; lag: those of column
  // k-2 are, in every CTA's bank, but not summed over the group
  int pending = st->pending, cc = 0, next = OP_TOP, from = AT_CAP;
  // resumed: the first row is read from its owner's slice, once that is there
  int op = k > 0 && G > 1 ? OP_FENCE : OP_TOP;
  unsigned gen = 0;
  bool lag = false, fuse = false, nonfinite = false, zero = false;
  // the row the next pass needs: published by its owner at the last exchange,
  // or (direct) in the panel, every column of it visible
  bool direct = true;
  // E = 4: per-warp dots of the last pass that are not added up yet
  int add_n = 0;
  bool add_row = false;
  // the exchange warp's first thread: the columns of an epsilon whose distance
  // to the tolerance is not noted yet; the product of the lagging norms
  int settled = 0;
  double rl = 0.0;
  bool idle = false;
  const int iters0 = st->iters;
  const int maxR = B.maxRank;  // -1: none (src/lowRank.cpp:149,244-247)
  if (status == ACA_RUNNING && k == 0 && maxR == 0) status = ACA_POST;
  auto bank = [&](int kc) { return (int64_t)(kc & 1) * 2 * L.kcap_max; };
  // the dots of epsilon_k formed without a pass, then settled (op, next, from)
  auto settle_pending = [&](int at) {
    group_dots<C>(L, sl[0], sl[1], k, L.part + (int64_t)blockIdx.x * L.part_stride + bank(k));
    add_n = 0;
    op = OP_FENCE;
    next = OP_PEND;
    from = at;
  };

  while (status == ACA_RUNNING) {
    if (op == OP_TOP) {  // a new step
      if (k == 1) pending = 0;  // settled with the column itself: no earlier columns
      if (!pending && !lag && sh.stop) { status = ACA_POST; break; }
      if (k >= ub || k >= min(B.kcap, B.kstop) || sh.yield) {
        if (lag) {
          op = OP_FENCE;
          next = OP_LAG;
          from = AT_CAP;
        } else if (k >= ub) {
          status = ACA_POST;
          break;
        } else if (pending) {
          settle_pending(AT_CAP);
        } else {
          // paused: the host grows the capacity, or shares the CTAs anew, and resumes
          status = k >= B.kcap ? ACA_NEED_CAP : ACA_PAUSED;
          break;
        }
      } else {
        ++iters;
        fuse = pending != 0;
        op = OP_ROW;
      }
    }
    const bool pass = op == OP_ROW || op == OP_COL, row = op == OP_ROW;
    const int kc = op == OP_LAG || (op == OP_COL && lag) ? k - 1 : op == OP_PEND ? k : 0;
    int nd = 0;
    Pass p;
    if (pass) {
      // a row pass (the residual row on this CTA's columns), or a column pass
      // (the residual column on its rows); the chosen flags are their owner's
      const int at = row ? cur : cc;
      const GroupSlice& own = sl[row];
      if (tid == 0 && at >= own.lo && at < own.hi) {
        (row ? B.cR : B.cC)[at] = 1;
        if (E == 1 && at - own.lo < C::ROWS) fl[(int)row * C::ROWS + at - own.lo] = 1;
      }
      const int og = at / own.per, oj = at - og * own.per, oc = oj / own.cr;  // its owner
      p.row = row;
      p.k = k;
      p.fixed = (row ? B.r0 : B.c0) + at;
      p.base = row ? B.c0 : B.r0;
      p.dots = fuse;
      p.cs = CoefSrc{direct || G == 1 ? nullptr
                                      : L.pub + ((size_t)(B.g0 + og) * 2 + (gen & 1)) * L.pub_stride,
                     ((uint64_t)L.launch_tag << 32) | gen,
                     (row ? B.sW + og * B.strW : B.sV + og * B.strV) +
                         (int64_t)oc * own.kcap * own.cr + (oj - oc * own.cr),
                     own.cr};
      p.chosen = row ? B.cC : B.cR;
      p.dout = L.part + (int64_t)blockIdx.x * L.part_stride + bank(k) + (row ? 0 : L.kcap_max);
      p.dotw = E > 1 ? L.dotg + (int64_t)blockIdx.x * L.dotg_stride +
                           (row ? 0 : L.dotg_stride / 2)
                     : nullptr;
      const GroupSlice s = sl[!row];
      const int T = s.chunks * ((k + C::TC - 1) / C::TC);
      // tiles issued for another pass than this one: let them land, unread
      if (R.ekind != (row ? 0 : 1) || R.ek != k) {
        for (int a = 0; a < R.ahead; ++a) {
          if (w < C::COPY) {
            mbar_wait(R.full + R.slot, R.parity, L.err);
            __syncwarp();
            if (lane == 0) mbar_arrive(R.empty + R.slot);
          }
          R.step();
        }
        R.ahead = 0;
      }
      const int have = R.ahead, nk = row ? k : k + 1;
      const int Tn = sl[row].chunks * ((nk + C::TC - 1) / C::TC);
      R.ahead = min(R.stages, Tn);
      R.ekind = row ? 1 : 0;
      R.ek = nk;
      // the coefficients (and the pivot, element k of a column pass's row),
      // read by the warps with no entries to evaluate
      const int nco = row ? k : k + 1;
      if (E > 1)
        for (int l = tid; l < nco; l += C::NT) coef[l] = coef_load(p.cs, l, L);
      else if (w >= C::SW)
        for (int l = tid - 32 * C::SW; l < nco; l += C::NT - 32 * C::SW)
          coef[l] = coef_load(p.cs, l, L);
      if (w < C::SW) {
        sum_role<C>(L, S, p, s, coef, xs + (row ? 0 : 3 * C::ROWS), fl + (row ? 0 : C::ROWS), R, sh,
                    nonfinite);
      } else if (E == 1 && w < C::COPY) {
        dot_role<C>(L, p, s, dsm, R);
      } else {
        bar_all();
        if (w == C::COPY)
          for (int idx = have; idx < T + R.ahead; ++idx) {
            const bool mine = idx < T;
            ring_issue<C>(R, mine ? s : sl[row], mine ? k : nk, mine ? idx : idx - T, L.err);
          }
        for (int q = 0; q < T; ++q) R.step();
      }
      if (op == OP_COL && lag) nd = k - 2;
    } else if (op == OP_LAG || op == OP_PEND) {
      nd = kc - 1;
    } else if (op == OP_SCAN) {
      // the first row not chosen yet (src/lowRank.cpp:189-194)
      if (tid == 0) sh.imin = INT_MAX;
      __syncthreads();
      int f = INT_MAX;
      for (int i = tid; i < B.m; i += C::NT)
        if (__ldcg(B.cR + i) == 0) { f = i; break; }
      if (f != INT_MAX) atomicMin(&sh.imin, f);
    }
    if (w >= C::EX) {
      if (tid == 32 * C::EX) {  // what an exchange need not wait for
        if (settled > 0 && settled < ub && settled >= B.minRank) {
          const double gap = fabs(sh.eps - L.tol) / L.tol;
          sh.margin = fmin(sh.margin, gap);
          if (gap < 1e-10) ++sh.near;
        }
        settled = 0;
        if (op == OP_ROW) {
          rl = sqrt(sh.swl) * sqrt(sh.svl);
          // enough of the launch's CTAs have run out of work: let the host
          // share them among the blocks that still run
          idle = g == 0 && L.yield_at > 0 && iters - iters0 >= 24 &&
                 *(volatile unsigned*)L.idle >= (unsigned)L.yield_at;
        }
      }
      if (E > 1 && add_n > 0) {  // the last pass's dots, chunks and warps in order
        const double* dw = L.dotg + (int64_t)blockIdx.x * L.dotg_stride +
                           (add_row ? 0 : L.dotg_stride / 2);
        const int parts = sl[!add_row].chunks * C::SW;
        double* to = L.part + (int64_t)blockIdx.x * L.part_stride + bank(add_n + 1) +
                     (add_row ? 0 : L.kcap_max);
        for (int l = tid - 32 * C::EX; l < add_n; l += 32 * C::RW) {
          double t = 0.0;
#pragma unroll 8
          for (int q = 0; q < parts; ++q) t += dw[(int64_t)q * L.kcap_max + l];
          to[l] = t;
        }
        if (C::RW > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * C::RW) : "memory");
      }
      // publish what the CTA wrote before this turn (the exchange warp's next
      // post follows), and see what the others had published at the last one
      if (pass && G > 1 && w == C::EX) fence_gpu();
      if (nd > 0) {
        if (pass && C::RW > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * C::RW) : "memory");
        lag_share<C>(L, B.g0, G, bank(kc), nd, sh);
      }
    }
    add_n = pass && fuse ? k - 1 : 0;
    add_row = row;

    // ---------------- the exchange, number gen: the sum warps' results and
    // the lag shares of every CTA, combined into sh (the same in all of
    // them).  Slots and published rows alternate by the exchange's parity: a
    // CTA writes exchange gen + 2 only after all have posted gen + 1, when
    // nobody reads gen any more.
    __syncthreads();
    ++gen;
    {
      double bv = -1.0, sq = 0.0, dot = 0.0;
      int bi = INT_MAX, cand = INT_MAX;
      unsigned yield = 0;
      if (pass && lane < C::SW) {
        bv = sh.red_v[lane];
        bi = sh.red_i[lane];
        cand = sh.red_c[lane];
        sq = sh.red_s[lane];
      }
      if (w == C::EX) {
        bool fail = false;
        warp_argmax_all(bv, bi);
        cand = __reduce_min_sync(0xffffffffu, cand);
        sq = warp_sum_all(sq);
        for (int r = 0; r < C::RW; ++r) dot += sh.lag[r];
        yield = __shfl_sync(0xffffffffu, (unsigned)idle, 0);
        if (G > 1) {
          if (!pass) fence_gpu();
          unsigned char* slots = L.slots + (size_t)B.g0 * 128 + (gen & 1) * 64;
          if (lane < 3) {
            const double v = lane == 0 ? bv : lane == 1 ? sq : dot;
            const uint32_t x = lane == 0 ? (uint32_t)bi : lane == 1 ? (uint32_t)cand : yield;
            st_b128(slots + (size_t)g * 128 + 16 * lane, (uint64_t)__double_as_longlong(v),
                    (uint64_t)x | ((uint64_t)gen << 32));
          }
          bv = -1.0;
          sq = dot = 0.0;
          bi = cand = INT_MAX;
          const unsigned want = gen + L.bar_extra;
          for (int q = lane; q < G; q += 32) {
            const unsigned char* sp = slots + (size_t)q * 128;
            uint64_t a0, a1, b0, b1, e0, e1;
            for (unsigned polls = 0;; ++polls) {
              ld_b128(sp, a0, a1);
              ld_b128(sp + 16, b0, b1);
              ld_b128(sp + 32, e0, e1);
              if ((unsigned)(a1 >> 32) == want && (unsigned)(b1 >> 32) == want &&
                  (unsigned)(e1 >> 32) == want)
                break;
              if (polls >= L.spin_limit || ((polls & 63) == 63 && *(volatile unsigned*)L.err)) {
                fail = true;
                break;
              }
              if (polls >= 256) __nanosleep(100);
            }
            argmax_merge(bv, bi, __longlong_as_double((long long)a0), (int)(uint32_t)a1);
            cand = min(cand, (int)(uint32_t)b1);
            sq += __longlong_as_double((long long)b0);
            dot += __longlong_as_double((long long)e0);
            yield |= (unsigned)e1;
          }
          if (!pass) fence_gpu();
          warp_argmax_all(bv, bi);
          cand = __reduce_min_sync(0xffffffffu, cand);
          sq = warp_sum_all(sq);
          dot = warp_sum_all(dot);
          fail = __any_sync(0xffffffffu, fail);
          yield = __reduce_or_sync(0xffffffffu, yield);
        } else if (L.bar_extra) {  // a group of one waits for nobody, unless it is told to
          fail = true;
        }
        if (lane == 0) {
          if (fail) atomicOr(L.err, DEV_ERR_TIMEOUT);
          sh.fail = fail;
          if (pass) {
            sh.mv = bv;
            sh.mi = bi == INT_MAX ? INT_MAX : bi >> 1;
            sh.mflag = bi == INT_MAX ? 0 : bi & 1;
            sh.mcand = cand;
          }
          if (row) {
            sh.svt = sq;
            sh.yield = (int)yield;
          }
          // epsilon after kce columns (src/lowRank.cpp:234-241), from the norms
          // of the lagging or the pending column and the dots just summed
          int kce = kc;
          double sw = sh.swp, sv = sh.svp, root = rl;
          if (op == OP_LAG || op == OP_COL) {
            sw = sh.swl;
            sv = sh.svl;
          }
          if (op != OP_COL) root = sqrt(sw) * sqrt(sv);
          if (op == OP_COL && (sh.mflag ? sh.mcand : sh.mi) != INT_MAX) {  // the column is stored
            sh.swl = sh.swp;
            sh.svl = sh.svp;
            sh.swp = sq;
            sh.svp = sh.svt;
            if (k == 0 && maxR != 1) {  // after the first column: no dots
              kce = 1;
              sw = sq;
              sv = sh.svt;
              dot = 0.0;
              root = sqrt(sw) * sqrt(sv);
            }
          }
          if (kce > 0) {
            sh.frob2 += 2 * dot + sw * sv;
            const double eps = root / sqrt(sh.frob2);
            sh.eps = eps;
            sh.stop = !(eps > L.tol) && kce >= B.minRank;
            settled = kce;
          }
        }
      } else if (pass && G > 1 && w < C::COPY) {
        // publish this CTA's candidate row of the panel just extended
        warp_argmax_all(bv, bi);
        if (bi != INT_MAX) {
          const GroupSlice s = sl[!row];
          const int oj = (bi >> 1) - s.lo, oc = oj / s.cr;
          const double* from_row = s.column(oc, 0) + (oj - oc * s.cr);
          const uint64_t tag = ((uint64_t)L.launch_tag << 32) | gen;
          unsigned char* to = L.pub + ((size_t)blockIdx.x * 2 + (gen & 1)) * L.pub_stride;
          for (int l = tid; l <= k; l += 32 * C::COPY)
            st_b128(to + (size_t)l * 16,
                    (uint64_t)__double_as_longlong(__ldcg(from_row + (int64_t)l * s.cr)), tag);
        }
      }
    }
    __syncthreads();
    if (sh.fail) { status = ACA_ERROR; break; }

    // ---------------- what follows
    if (op == OP_FENCE) {
      direct = true;
      op = next;
    } else if (op == OP_ROW) {
      direct = false;
      zero = sh.mv <= L.minPivot;
      if (zero || (sh.mflag && sh.mcand == INT_MAX)) {
        // a zero residual row (src/lowRank.cpp:187-195), or no column left to
        // choose (:200-202).  Whether the reference even reached this step
        // depends on the lagging epsilon, then (a zero row) on the pending one.
        if (lag) {
          op = OP_FENCE;
          next = OP_LAG;
          from = AT_ROW;
        } else if (!zero) {
          status = ACA_POST;  // the rank is k whichever way the pending one goes
        } else if (pending) {
          settle_pending(AT_ROW);
        } else {
          op = OP_FENCE;  // every chosen flag
          next = OP_SCAN;
        }
      } else {
        cc = sh.mflag ? sh.mcand : sh.mi;
        op = OP_COL;
        if (sh.mflag) {  // not the row that its owner published: read it from the panel
          op = OP_FENCE;
          next = OP_COL;
        }
      }
    } else if (op == OP_COL) {
      direct = false;
      if (lag && sh.stop) {  // the last column and this step are discarded
        --k;
        iters -= 2;
        status = ACA_POST;
        break;
      }
      lag = false;
      const int nr = sh.mflag ? sh.mcand : sh.mi;
      if (nr == INT_MAX) {  // no admissible next row: stop before storing (src/lowRank.cpp:226-227)
        if (!fuse) { status = ACA_POST; break; }
        op = OP_FENCE;
        next = OP_PEND;
        from = AT_END;
      } else {
        if (g == 0 && tid == 0) {
          B.prow[k] = cur;
          B.pcol[k] = cc;
        }
        lag = fuse;
        pending = 1;
        cur = nr;
        ++k;
        op = OP_TOP;
        if (sh.mflag) {
          op = OP_FENCE;
          next = OP_TOP;
        }
        if (k == maxR) {  // the rank ceiling: stop without the last epsilon (src/lowRank.cpp:244-247)
          if (!lag) { status = ACA_POST; break; }
          op = OP_FENCE;
          next = OP_LAG;
          from = AT_MAX;
        }
      }
    } else if (op == OP_LAG) {
      lag = false;
      op = OP_TOP;
      if (sh.stop) {  // the column after it (and the step begun) are discarded
        --k;
        iters -= from == AT_ROW ? 2 : 1;
        status = ACA_POST;
      } else if (from == AT_MAX || (from == AT_ROW && !zero)) {
        status = ACA_POST;
      } else if (from == AT_ROW) {
        if (pending) {
          settle_pending(AT_ROW);
        } else {
          op = OP_FENCE;
          next = OP_SCAN;
        }
      }
    } else if (op == OP_PEND) {
      pending = 0;
      op = OP_TOP;  // AT_CAP: the top of the loop stops, or pauses
      if (from == AT_END || (from == AT_ROW && sh.stop)) {
        if (sh.stop) --iters;
        status = ACA_POST;
      } else if (from == AT_ROW) {
        op = OP_FENCE;
        next = OP_SCAN;
      }
    } else {  // OP_SCAN
      cur = sh.imin;
      direct = true;
      op = OP_TOP;
      if (cur == INT_MAX) status = ACA_POST;
    }
  }
  if (status == ACA_POST) pending = 0;
  if (tid == 32 * C::EX && settled > 0 && settled < ub && settled >= B.minRank) {
    const double gap = fabs(sh.eps - L.tol) / L.tol;
    sh.margin = fmin(sh.margin, gap);
    if (gap < 1e-10) ++sh.near;
  }

  // the columns into the level's arenas (a block stored in full replaces them)
  if (status != ACA_ERROR && k > 0) {
    slice_copy(sl[0], B.V, L.ld, k, false, C::NT);
    slice_copy(sl[1], B.W, L.ld, k, false, C::NT);
    __syncthreads();
  }
  int rank = k;
  if (status == ACA_POST)
    status = aca_post_process<double>(B, S, B.W, B.V, L.ld, k, sl[1].lo, sl[1].hi, sl[0].lo,
                                      sl[0].hi, C::NT, &rank);
  if (nonfinite) atomicOr(L.err, DEV_ERR_NONFINITE);
  // Every CTA of the group reached the same state, and each has read the
  // entry state before its first exchange or, with none made, waits for the
  // others here: CTA 0 records the state when nobody will read it any more.
  if (G > 1 && status != ACA_ERROR) {
    __syncthreads();
    ++gen;
    if (w == C::EX) {
      unsigned char* slots = L.slots + (size_t)B.g0 * 128 + (gen & 1) * 64;
      bool fail = false;
      if (lane == 0) st_b128(slots + (size_t)g * 128, 0, (uint64_t)gen << 32);
      for (int q = lane; g == 0 && q < G; q += 32)
        for (unsigned polls = 0;; ++polls) {
          uint64_t a0, a1;
          ld_b128(slots + (size_t)q * 128, a0, a1);
          if ((unsigned)(a1 >> 32) == gen + L.bar_extra) break;
          if (polls >= L.spin_limit || ((polls & 63) == 63 && *(volatile unsigned*)L.err)) {
            fail = true;
            break;
          }
          if (polls >= 256) __nanosleep(100);
        }
      if (__any_sync(0xffffffffu, fail) && lane == 0) {
        atomicOr(L.err, DEV_ERR_TIMEOUT);
        sh.fail = 1;
      }
    }
    __syncthreads();
    if (sh.fail) status = ACA_ERROR;
  }
  __syncthreads();
  if (tid == 0 && L.yield_at > 0) atomicAdd(L.idle, 1u);
  if (g == 0 && tid == 0) {
    st->k = k;
    st->cur = cur;
    st->iters = iters;
    st->status = status;
    st->frob2 = sh.frob2;
    st->eps = sh.eps;
    st->margin = sh.margin;
    st->near = sh.near;
    st->rank = rank;
    st->swp = sh.swp;
    st->svp = sh.svp;
    st->pending = pending;
  }
  // No CTA releases its shared memory under a copy: wait (bounded) for the
  // last tile issued into each slot.
  if (w == C::COPY) {
    const uint32_t last = min(R.issued, (uint32_t)R.stages);
    for (uint32_t t = 0; t < last; ++t) {
      if (R.islot == 0) {
        R.islot = R.stages;
        R.iparity ^= 1u;
      }
      --R.islot;
      for (uint32_t polls = 0; polls < (1u << 20) && !mbar_try_wait(R.full + R.islot, R.iparity);
           ++polls)
        __nanosleep(64);
    }
  }
}

struct GroupVariant {
  const void* fn;
  int threads, rows, tc, sw;
  bool dots;  // dots by chunk and warp in global memory (E = 4)
};

template <int SW, int E>
GroupVariant variant_of() {
  using C = GroupCfg<SW, E>;
  return {(const void*)aca_group_kernel<SW, E>, C::NT, C::ROWS, C::TC, C::SW, E > 1};
}

GroupVariant group_variant(int v) {
  return v == ACA_GROUP_8x1 ? variant_of<8, 1>() : variant_of<8, 4>();
}

}  // namespace

// Dots by chunk and warp of a CTA whose slices have at most `rows` rows, in
// units of kcap_max doubles (row and column passes apart).
int64_t aca_group_dots(int v, int rows) {
  const GroupVariant g = group_variant(v);
  return g.dots ? 2 * (int64_t)g.sw * slice_chunks(rows, g.rows) : 0;
}

// Doubles of a CTA's slice of `per` rows in the working layout, kcap columns.
int64_t aca_group_slice(int v, int per, int kcap) {
  const int most = group_variant(v).rows;
  return (int64_t)slice_chunks(per, most) * slice_pitch(per, most) * kcap;
}

// The ring of a launch whose slices have at most `rows` rows and whose blocks
// at most `kcap` columns, in `budget` bytes of dynamic shared memory: its
// stages (0: fewer than GR_SMIN fit), the doubles of a stage, the bytes in all.
// A slice of `rows` or fewer has a pitch of at most that of one chunk.
int aca_group_ring(int v, int rows, int kcap, size_t budget, int* stage_elems, size_t* bytes) {
  const GroupVariant g = group_variant(v);
  *stage_elems = g.tc * std::min(g.rows, (rows + 15) & ~15);
  const size_t fixed = sizeof(double) * ((size_t)((kcap + 16) & ~15) + (g.dots ? 0 : (size_t)kcap));
  const size_t stage = sizeof(double) * (size_t)*stage_elems;
  const int st = fixed >= budget ? 0 : (int)std::min<size_t>(GR_SMAX, (budget - fixed) / stage);
  *bytes = stage * st + fixed;
  return st >= GR_SMIN ? st : 0;
}

int aca_group_max_coresident(int v, size_t smem, int* per_sm) {
  const GroupVariant g = group_variant(v);
  *per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(g.fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) e = smem_opt_in(g.fn, smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, g.fn, g.threads, smem);
  if (e != cudaSuccess) cudaGetLastError();
  return (int)e;
}

int aca_group_launch(const AcaLaunch& L, int v, size_t smem, bool cooperative, cudaStream_t s) {
  if (L.ring_stages < GR_SMIN || L.ring_stages > GR_SMAX)
    return (int)cudaErrorInvalidValue;
  const GroupVariant g = group_variant(v);
  int per_sm = 0;
  if (int e = aca_group_max_coresident(v, smem, &per_sm)) return e;
  dim3 grid(L.ncta), block(g.threads);
  void* args[] = {(void*)&L};
  cudaError_t e = cooperative ? cudaLaunchCooperativeKernel(g.fn, grid, block, args, smem, s)
                              : cudaLaunchKernel(g.fn, grid, block, args, smem, s);
  if (e != cudaSuccess) cudaGetLastError();
  return (int)e;
}
