// storeLRinTree (src/HODLR_Matrix.cpp:257-272,274-430): partial-pivot ACA of
// every off-diagonal block, level by level (aca.cu kernels).
#include "handle.h"

namespace hodlr_impl {

// Grow level L to `cap` columns, keeping the first kcap ones.
int grow_level(hodlr_t h, Level& L, int cap) {
  const int64_t N = h->ldp();
  double *W2 = nullptr, *V2 = nullptr;
  CK(dalloc(h, &W2, (size_t)(N * cap)));
  cudaError_t e = dalloc(h, &V2, (size_t)(N * cap));
  if (e != cudaSuccess) {
    dfree(h, W2);
    return cuda_fail(h, e, "grow_level");
  }
  if (L.W && L.kcap > 0) {
    CK(cudaMemcpyAsync(W2, L.W, sizeof(double) * N * L.kcap, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(V2, L.V, sizeof(double) * N * L.kcap, cudaMemcpyDeviceToDevice, h->stream));
  }
  CK(cudaStreamSynchronize(h->stream));
  dfree(h, L.W);
  dfree(h, L.V);
  L.W = W2;
  L.V = V2;
  L.kcap = cap;
  return HODLR_OK;
}

void fill_block(hodlr_t h, Level& L, int q, AcaBlock& B) {
  int r0, c0, m, n;
  block_geom(L, q, r0, c0, m, n);
  (void)h;
  B.st = L.d_st + q;
  B.W = L.W + r0;
  B.V = L.V + c0;
  B.cR = L.cR + r0;
  B.cC = L.cC + c0;
  B.prow = L.prow + r0;
  B.pcol = L.pcol + c0;
  B.r0 = r0;
  B.c0 = c0;
  B.m = m;
  B.n = n;
  B.kcap = L.kcap;
  B.level = 0;
  B.g0 = 0;
  B.G = 1;
  const int p = q >> 1;
  B.kstop = INT_MAX;
  B.sW = B.sV = nullptr;
  B.strW = B.strV = 0;
  B.minRank = (q & 1) ? L.bmin[p] : L.tmin[p];
  B.maxRank = (q & 1) ? L.bmax[p] : L.tmax[p];
}

bool level_done(const Level& L) {
  for (auto& s : L.st)
    if (s.status != ACA_DONE) return false;
  return true;
}

// Dynamic shared memory of a group launch (one CTA an SM), beside its static
// arrays.
size_t group_smem_budget(int v) { return v == ACA_GROUP_8x1 ? 212 * 1024 : 224 * 1024; }

// One ACA launch over `blocks`: groups of G CTAs each, or, with `groups`,
// groups[i] CTAs for block i (a CTA table maps CTAs to blocks).  variant:
// ACA_GROUP_NONE for aca_kernel with nt threads, else of aca_group_kernel.
// yield_at: with so many CTAs out of work the others' blocks pause (0: never).
int run_aca(hodlr_t h, std::vector<AcaBlock>& blocks, int G, int nt, int kcap_max, int variant,
            const std::vector<int>* groups, int yield_at) {
  const int nb = (int)blocks.size();
  if (nb == 0) return HODLR_OK;
  int ncta = nb * G;
  if (groups) {
    ncta = 0;
    for (int i = 0; i < nb; ++i) {
      blocks[i].g0 = ncta;
      blocks[i].G = (*groups)[i];
      ncta += (*groups)[i];
    }
    std::vector<int> table((size_t)ncta);
    for (int i = 0; i < nb; ++i)
      for (int c = 0; c < blocks[i].G; ++c) table[(size_t)(blocks[i].g0 + c)] = i;
    CK(dgrow(h, h->d_cta, h->cta_cap, ncta));
    CK(cudaMemcpyAsync(h->d_cta, table.data(), sizeof(int) * ncta, cudaMemcpyHostToDevice,
                       h->stream));
  }
  CK(dgrow(h, h->d_blocks, h->blocks_cap, nb));
  CK(cudaMemcpyAsync(h->d_blocks, blocks.data(), sizeof(AcaBlock) * nb, cudaMemcpyHostToDevice,
                     h->stream));
  int64_t stride = 12 + 4 * (int64_t)kcap_max;  // args + two banks of dots and norms
  CK(dgrow(h, h->part, h->part_cap, stride * ncta));
  CK(dgrow(h, h->bar, h->bar_cap, nb));
  CK(cudaMemsetAsync(h->bar, 0, sizeof(unsigned) * nb, h->stream));
  AcaLaunch L;
  L.blocks = h->d_blocks;
  L.nblocks = nb;
  L.G = G;
  L.ld = h->ldp();
  L.tol = h->tol;
  L.minPivot = (double)h->minPivot;
  L.kcap_max = kcap_max;
  L.part = h->part;
  L.part_stride = stride;
  L.bar = h->bar;
  L.err = h->d_err;
  L.src = make_src(h);
  L.cta_block = groups ? h->d_cta : nullptr;
  L.ncta = ncta;
  L.dotg = nullptr;
  L.dotg_stride = 0;
  L.spin_limit = h->spin_limit ? h->spin_limit : variant ? HODLR_SPIN_LIMIT >> 4 : HODLR_SPIN_LIMIT;
  L.bar_extra = h->bar_unreachable ? 1u : 0u;
  L.narrow = 0;
  L.ring_stages = L.stage_elems = 0;
  L.slots = nullptr;
  size_t smem = 0;
  if (variant) {
    int rows = 1;
    for (int i = 0; i < nb; ++i) {
      const int g = groups ? (*groups)[i] : G;
      rows = std::max(rows, (std::max(blocks[i].m, blocks[i].n) + g - 1) / g);
    }
    L.ring_stages = aca_group_ring(variant, rows, kcap_max, group_smem_budget(variant), &L.stage_elems,
                                   &smem);
    if (!L.ring_stages) return fail(h, HODLR_ERR_STATE, "ACA ring does not fit");
    CK(dgrow(h, h->slots, h->slots_cap, (int64_t)ncta * 128 + 128));
    L.slots = h->slots;
    CK(cudaMemsetAsync(h->slots, 0, (size_t)ncta * 128 + 128, h->stream));
    L.idle = reinterpret_cast<unsigned*>(h->slots + (size_t)ncta * 128);
    L.yield_at = yield_at;
    L.pub_stride = 16 * ((int64_t)kcap_max + 1);
    const int64_t pneed = 2 * L.pub_stride * ncta;
    if (pneed > h->pub_cap) {
      CK(dgrow(h, h->pub, h->pub_cap, pneed));
      CK(cudaMemsetAsync(h->pub, 0, (size_t)pneed, h->stream));
    }
    L.pub = h->pub;
    L.launch_tag = ++h->aca_tag;
    L.dotg_stride = aca_group_dots(variant, rows) * kcap_max;
  } else {
    // slices of a group shorter than 768 rows: the 2-element instance (512-row
    // chunks) leaves fewer lanes idle than the 4-element one (1024-row chunks)
    if (nt == 256) {
      int longest = 0;
      for (int i = 0; i < nb; ++i) {
        const int g = groups ? (*groups)[i] : G;
        longest = std::max(longest, (std::max(blocks[i].m, blocks[i].n) + g - 1) / g);
      }
      L.narrow = longest < 768 ? 1 : 0;
    }
    if (aca_smem_bytes(nt, kcap_max) > 227 * 1024)
      return fail(h, HODLR_ERR_UNSUPPORTED, "block rank above the shared-memory limit of ACA");
    if (aca_dots_global(nt, kcap_max)) L.dotg_stride = (int64_t)(nt / 32) * kcap_max;
  }
  if (L.dotg_stride > 0) {
    CK(dgrow(h, h->dotg, h->dotg_cap, L.dotg_stride * ncta));
    L.dotg = h->dotg;
  }
  bool coop = G > 1;
  if (groups)
    for (int g : *groups) coop |= g > 1;
  CK(cudaEventRecord(h->ev0, h->stream));
  int rc = variant ? aca_group_launch(L, variant, smem, coop, h->stream)
                   : aca_launch(L, nt, kcap_max, coop, h->stream);
  if (rc == (int)cudaErrorCooperativeLaunchTooLarge) return HODLR_ERR_RETRY_SMALLER;
  if (rc) return cuda_fail(h, (cudaError_t)rc, "aca_launch");
  h->nlaunch += 1;
  CK(cudaEventRecord(h->ev1, h->stream));
  CK(cudaEventSynchronize(h->ev1));
  float ms = 0;
  CK(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  h->aca_seconds += ms * 1e-3;
  h->aca_launches += 1;
  return check_dev_err(h, "ACA");
}

// Allocate the per-level arrays of level L with `cap` low-rank columns.
int init_level(hodlr_t h, Level& L, int cap) {
  const int64_t N = h->n;
  int rc = grow_level(h, L, std::max(1, std::min(L.ub_max, cap)));
  if (rc) return rc;
  CK(dalloc(h, &L.cR, (size_t)N));
  CK(dalloc(h, &L.cC, (size_t)N));
  CK(dalloc(h, &L.prow, (size_t)N));
  CK(dalloc(h, &L.pcol, (size_t)N));
  CK(cudaMemsetAsync(L.cR, 0, N, h->stream));
  CK(cudaMemsetAsync(L.cC, 0, N, h->stream));
  const int nb = L.nblocks();
  CK(dalloc(h, &L.d_st, (size_t)nb));
  L.st.assign(nb, AcaState());
  for (auto& s : L.st) {
    s.frob2 = 0;
    s.eps = 1;
    s.margin = HUGE_VAL;
    s.swp = s.svp = 0;
    s.k = 0;
    s.cur = 0;
    s.status = ACA_RUNNING;
    s.iters = 0;
    s.rank = 0;
    s.near = 0;
    s.pending = 0;
    s.pad = 0;
  }
  CK(cudaMemcpyAsync(L.d_st, L.st.data(), sizeof(AcaState) * nb, cudaMemcpyHostToDevice,
                     h->stream));
  return HODLR_OK;
}

// Read the level's block states back; grow the level where blocks paused for
// capacity and re-arm them.  *done = every block of the level finished.
int sync_level(hodlr_t h, Level& L, bool* done) {
  const int nb = L.nblocks();
  CK(cudaMemcpyAsync(L.st.data(), L.d_st, sizeof(AcaState) * nb, cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  int need = 0;
  bool resume = false;
  *done = true;
  for (auto& s : L.st) {
    if (s.status == ACA_ERROR) return fail(h, HODLR_ERR_TIMEOUT, "ACA group failed");
    if (s.status == ACA_NEED_CAP) need = std::max(need, L.kcap + std::max(32, L.kcap / 2));
    if (s.status == ACA_NEED_CAP_POST) need = std::max(need, s.rank);
    resume |= s.status == ACA_PAUSED;
    if (s.status != ACA_DONE) *done = false;
  }
  if (need > 0 || resume) {
    int cap = std::min(std::max(need, L.kcap + 1), std::max(L.ub_max, L.kcap + 1));
    int rc = need > 0 ? grow_level(h, L, cap) : HODLR_OK;
    if (rc) return rc;
    for (auto& s : L.st) {
      if (s.status == ACA_NEED_CAP || s.status == ACA_PAUSED) s.status = ACA_RUNNING;
      if (s.status == ACA_NEED_CAP_POST) s.status = ACA_POST;
    }
    CK(cudaMemcpyAsync(L.d_st, L.st.data(), sizeof(AcaState) * nb, cudaMemcpyHostToDevice,
                       h->stream));
  }
  return HODLR_OK;
}

int level_kmax(const Level& L) {
  int k = 0;
  for (auto& s : L.st) k = std::max(k, s.rank);
  return k;
}

// storeLRinTree (src/HODLR_Matrix.cpp:257-272,274-430) for every block.
// Levels with many blocks run together in one launch, one CTA per block
// (G = 1); the top levels, with few large blocks, run one cooperative launch
// each with a group of CTAs per block.  They go bottom-up so that each
// level's W/V capacity can be sized from the ranks of the level below it
// (ranks shrink down the tree); a level that needs more grows and resumes.
std::vector<int4> block_geoms(hodlr_t h) {
  std::vector<int4> geom;
  for (auto& L : h->lv)
    for (int q = 0; q < L.nblocks(); ++q) {
      int r0, c0, m, n;
      block_geom(L, q, r0, c0, m, n);
      geom.push_back(make_int4(r0, c0, m, n));
    }
  return geom;
}

// Features of every block (nb x HODLR_MLP_INPUTS, device) for length scale l.
int block_features_dev(hodlr_t h, const std::vector<int4>& geom, double l, float* d_F) {
  const int nb = (int)geom.size();
  int4* d_geom = nullptr;
  CK(dalloc(h, &d_geom, (size_t)nb));
  CK(cudaMemcpyAsync(d_geom, geom.data(), sizeof(int4) * nb, cudaMemcpyHostToDevice, h->stream));
  int e = block_features_launch(h->d_pts, h->n, h->dim, d_geom, nb, (float)std::log(l),
                                (float)std::log(h->tol), d_F, h->stream);
  if (e) return cuda_fail(h, (cudaError_t)e, "block features");
  h->nlaunch += 1;
  dfree(h, d_geom);
  return HODLR_OK;
}

// Predicted ACA rank of every block (level-major order, as
// hodlr_get_block_info numbers them) from the rank model: block features on
// the device, the MLP forward, rank = exp(y) - 1 rounded and clamped.
int predict_ranks(hodlr_t h) {
  const std::vector<int4> geom = block_geoms(h);
  const int nb = (int)geom.size();
  h->pred.assign(nb, 0);
  if (nb == 0) return HODLR_OK;
  float *d_F = nullptr, *d_y = nullptr;
  CK(dalloc(h, &d_F, (size_t)nb * HODLR_MLP_INPUTS));
  CK(dalloc(h, &d_y, (size_t)nb));
  int rc = block_features_dev(h, geom, h->model_l, d_F);
  if (rc) return rc;
  int e = mlp_forward_launch(h->d_model, d_F, nb, d_y, h->stream);
  if (e) return cuda_fail(h, (cudaError_t)e, "rank prediction");
  h->nlaunch += 1;
  std::vector<float> y((size_t)nb);
  CK(d2h(h, y.data(), d_y, sizeof(float) * nb));
  dfree(h, d_F);
  dfree(h, d_y);
  for (int i = 0; i < nb; ++i) {
    const double r = std::expm1((double)std::min(y[i], 20.0f));
    const int ub = std::min(geom[i].z, geom[i].w);
    h->pred[i] = std::max(0, std::min(ub, (int)std::lround(r)));
  }
  return HODLR_OK;
}

// ---- launches of the few-block levels
//
// Time of a block's ACA from k0 to k columns, in us: steps of two passes.  A pass is a fixed part
// (5 alone, 8 with an exchange over a group), the start of every further chunk
// of the slice (its entries), and its tiles: GR 8x1 takes 16 columns of up to
// 256 rows in 0.3 us or more and streams at 44 KB/us, 8x4 takes 4 columns of
// up to 1024 rows in 0.3 us or more at 48 KB/us (measured on B200, one CTA an
// SM: the rates are the SM's share of the memory rate).
double group_time(int variant, double rows, double k0, double k, int G) {
  const double r = std::ceil(rows / G), kh = 0.5 * (k0 + k), fixed = G > 1 ? 8.0 : 5.0;
  double pass;
  if (variant == ACA_GROUP_8x1) {
    const double c = std::ceil(r / 256.0);
    pass = fixed + 0.9 * (c - 1.0) + std::ceil(kh / 16.0) * c * std::max(0.3, r / c * 128.0 / 44e3);
  } else {
    const double c = std::ceil(r / 1024.0);
    pass = fixed + 1.0 + 2.5 * (c - 1.0) +
           std::ceil(kh / 4.0) * c * std::max(0.3, r / c * 32.0 / 48e3);
  }
  return 2.0 * (k - k0) * pass;
}

struct GroupJob {
  int level, q, rows, G;
  double k0, k, t;
  int64_t work = 0, strW = 0, strV = 0;  // the block's slices in the working memory
};

// Share `ctas` CTAs among the jobs: always to the slowest one, as many more as
// make it faster.  Returns the slowest job's time; < 0: more jobs than CTAs.
double share_ctas(std::vector<GroupJob>& jobs, int ctas, int variant) {
  if ((int)jobs.size() > ctas) return -1.0;
  int left = ctas - (int)jobs.size();
  auto slower = [&](int a, int b) { return jobs[a].t < jobs[b].t; };
  std::vector<int> heap;
  for (size_t i = 0; i < jobs.size(); ++i) {
    jobs[i].G = 1;
    jobs[i].t = group_time(variant, jobs[i].rows, jobs[i].k0, jobs[i].k, 1);
    heap.push_back((int)i);
  }
  std::make_heap(heap.begin(), heap.end(), slower);
  while (!heap.empty()) {
    GroupJob& j = jobs[heap.front()];
    int more = 0;
    const int most = std::min(left, j.rows / 16);  // at least 16 rows a CTA
    for (int d = 1; d <= most && !more; ++d)
      if (group_time(variant, j.rows, j.k0, j.k, j.G + d) < j.t) more = d;
    if (!more) break;
    j.G += more;
    left -= more;
    j.t = group_time(variant, j.rows, j.k0, j.k, j.G);
    std::pop_heap(heap.begin(), heap.end(), slower);
    std::push_heap(heap.begin(), heap.end(), slower);
  }
  return heap.empty() ? 0.0 : jobs[heap.front()].t;
}

std::vector<GroupJob> group_jobs(hodlr_t h, const std::vector<int>& levels,
                                 const std::vector<double>& rank_est) {
  std::vector<GroupJob> jobs;
  for (int l : levels) {
    const Level& L = h->lv[l];
    for (int q = 0; q < L.nblocks(); ++q) {
      if (!L.st.empty() && L.st[q].status == ACA_DONE) continue;
      int r0, c0, m, n;
      block_geom(L, q, r0, c0, m, n);
      const double k0 = L.st.empty() ? 0.0 : L.st[q].k, most = std::min(m, n);
      const double k = std::min(most, std::max(rank_est[l], 1.25 * k0 + 4.0));
      GroupJob j{l, q, std::max(m, n), 1, k0, std::max(k0 + 1.0, k), 0.0};
      jobs.push_back(j);
    }
  }
  return jobs;
}

// The levels still to do (uppermost first) are cut into sets of neighbours
// whose blocks run in one launch: few-step and many-step blocks side by side
// keep the SMs busy where one level alone waits on its exchanges or on its
// slowest block, but a block in a crowd has fewer CTAs.  The cut minimises the
// sum of the sets' times as group_time has them.  Returns the index of the
// uppermost level of the deepest set, which runs first.
int group_set_top(hodlr_t h, const std::vector<int>& levels, const std::vector<double>& rank_est) {
  const int n = (int)levels.size();
  std::vector<double> best((size_t)n + 1, HUGE_VAL);  // of levels [0, i)
  std::vector<int> cut((size_t)n + 1, 0);
  best[0] = 0.0;
  for (int i = 1; i <= n; ++i)
    for (int j = i - 1; j >= 0; --j) {
      std::vector<int> set(levels.begin() + j, levels.begin() + i);
      std::vector<GroupJob> jobs = group_jobs(h, set, rank_est);
      const double t1 = share_ctas(jobs, h->num_sms, ACA_GROUP_8x1);
      if (t1 < 0 && j < i - 1) break;  // more levels only add blocks
      double t = t1 < 0 ? 0.0 : std::min(t1, share_ctas(jobs, h->num_sms, ACA_GROUP_8x4));
      t += 60.0;  // a launch and its read-back
      if (best[j] + t < best[i]) {
        best[i] = best[j] + t;
        cut[i] = j;
      }
    }
  return cut[n];
}

// One launch over every unfinished block of the set's levels.
int run_group_set(hodlr_t h, const std::vector<int>& set, const std::vector<double>& rank_est) {
  std::vector<GroupJob> jobs = group_jobs(h, set, rank_est);
  int ctas = h->num_sms, kcap_max = 1;
  for (int l : set) kcap_max = std::max(kcap_max, h->lv[l].kcap);
  for (;;) {  // a cooperative launch the driver refuses is retried with half the CTAs
    int variant = ACA_GROUP_NONE;
    const double t1 = share_ctas(jobs, ctas, ACA_GROUP_8x1);
    if (h->aca_ring && h->aca_ring_fits && t1 >= 0) {
      // the faster form, or the other one where only that has room for a ring
      // beside the coefficients of so many columns; neither: per thread
      const double t4 = share_ctas(jobs, ctas, ACA_GROUP_8x4);
      const int first = t1 <= t4 ? ACA_GROUP_8x1 : ACA_GROUP_8x4;
      for (int v : {first, ACA_GROUP_8x1 + ACA_GROUP_8x4 - first}) {
        int rows = 1, elems = 0, ps = 0;
        size_t bytes = 0;
        share_ctas(jobs, ctas, v);
        for (auto& j : jobs) rows = std::max(rows, (j.rows + j.G - 1) / j.G);
        if (!aca_group_ring(v, rows, kcap_max, group_smem_budget(v), &elems, &bytes)) continue;
        if (aca_group_max_coresident(v, bytes, &ps) || ps < 1)
          return fail(h, HODLR_ERR_CUDA, "occupancy query failed");
        variant = v;
        break;
      }
      // the slices' working layout, in the pool's scratch; without memory for it
      // the panels are loaded from the arenas per thread
      int64_t work = 0;
      for (auto& j : jobs) {
        if (!variant) break;
        int r0, c0, m, n;
        block_geom(h->lv[j.level], j.q, r0, c0, m, n);
        const int kcap = h->lv[j.level].kcap;
        j.work = work;
        j.strW = aca_group_slice(variant, (m + j.G - 1) / j.G, kcap);
        j.strV = aca_group_slice(variant, (n + j.G - 1) / j.G, kcap);
        work += (j.strW + j.strV) * j.G;
      }
      if (variant && h->pool.grow_scratch(sizeof(double) * (size_t)work, h->stream)) {
        cudaGetLastError();
        variant = ACA_GROUP_NONE;
      }
    }
    if (!variant) {
      // panels loaded per thread, several CTAs an SM: the same shares of what fits
      int ps = 0;
      if (aca_max_coresident(256, kcap_max, &ps))
        return fail(h, HODLR_ERR_CUDA, "occupancy query failed");
      const int most = std::max(1, ps) * ctas;
      if (share_ctas(jobs, most, ACA_GROUP_8x4) < 0)
        for (auto& j : jobs) j.G = 1;
    }
    std::vector<AcaBlock> bl(jobs.size());
    std::vector<int> groups(jobs.size());
    bool any = false;
    for (size_t i = 0; i < jobs.size(); ++i) {
      Level& L = h->lv[jobs[i].level];
      fill_block(h, L, jobs[i].q, bl[i]);
      if (variant) {
        bl[i].sW = (double*)h->pool.scratch + jobs[i].work;
        bl[i].sV = bl[i].sW + jobs[i].strW * jobs[i].G;
        bl[i].strW = jobs[i].strW;
        bl[i].strV = jobs[i].strV;
      }
      groups[i] = jobs[i].G;
      L.G = jobs[i].G;
      any |= jobs[i].G > 1;
    }
    int most = 0;
    double slowest = 0.0;
    for (auto& j : jobs) {
      most += j.G;
      slowest = std::max(slowest, j.t);
    }
    // ranks differ from block to block: share the CTAs anew when a third of them are
    // out of work, where a launch takes far longer than its overhead, or
    // (hodlr_set_aca_streaming(1), the same bits of epsilon every time) when a block
    // has the rank that was expected of it; in a forest first at a fifth of that,
    // which is the largest system's.  ACA in ms, fixed shares | by the clock | at column
    // counts: 2D N = 262144 131 | 111 | 117, sphere 16384 107.8 | 107.3 | 109.6, sphere
    // 65536 - | 373 | 400 (with a rank model 427), cube 40000 92.7 | 87.8 | 88.9, forest
    // of 40 - | 54.1 | 53.8.
    const bool share = variant && jobs.size() > 1 && slowest > 2000.0;
    const int yield_at = share && !h->aca_by_count ? std::max(1, most / 3) : 0;
    if (share && h->aca_by_count)
      for (size_t i = 0; i < jobs.size(); ++i)
        bl[i].kstop = (int)std::max(jobs[i].k0 + 24.0,
                                    h->nsys && jobs[i].k0 == 0.0 ? 0.2 * jobs[i].k : jobs[i].k);
    h->pool.scratch_busy = variant != ACA_GROUP_NONE;
    const int rc = run_aca(h, bl, 1, any ? 256 : 128, kcap_max, variant, &groups, yield_at);
    h->pool.scratch_busy = false;
    if (rc != HODLR_ERR_RETRY_SMALLER) return rc;
    if (ctas == 1) return fail(h, HODLR_ERR_CUDA, "aca_launch: cooperative launch refused");
    ctas = std::max(1, ctas / 2);
  }
}

static int compress_levels(hodlr_t h) {
  free_compress(h);
  h->aca_launches = 0;
  h->aca_seconds = 0;
  h->aca_bytes = 0;
  const int nlev = (int)h->lv.size();
  // predicted ranks, when a rank model is set: level capacities and the
  // order of the pooled blocks (largest predicted work first) follow them;
  // ACA's stopping test still decides every rank (a block that needs more
  // columns pauses and resumes after its level grows)
  std::vector<int> lbase(nlev + 1, 0);
  for (int l = 0; l < nlev; ++l) lbase[l + 1] = lbase[l] + h->lv[l].nblocks();
  const bool have_pred = h->d_model != nullptr;
  if (have_pred) {
    int rc = predict_ranks(h);
    if (rc) return rc;
  }
  auto pred = [&](int l, int q) { return h->pred[(size_t)(lbase[l] + q)]; };
  auto pred_cap = [&](int l) {
    int mx = 0;
    for (int q = 0; q < h->lv[l].nblocks(); ++q) mx = std::max(mx, pred(l, q));
    return std::max(16, ((mx + mx / 4 + 8) + 7) / 8 * 8);
  };
  auto hint = [&](int l) {
    if (l < (int)h->cap_hint.size() && h->cap_hint[l] > 0) return h->cap_hint[l];
    return have_pred ? pred_cap(l) : 0;
  };
  auto pred_or = [&](int l, int q) -> int64_t { return have_pred ? pred(l, q) + 1 : 1; };
  int per_sm = 0;
  if (aca_max_coresident(256, 256, &per_sm))
    return fail(h, HODLR_ERR_CUDA, "occupancy query failed");
  const int P0 = std::max(1, per_sm) * h->num_sms;
  std::vector<int> pooled_levels, group_levels;
  for (int l = 0; l < nlev; ++l)
    (h->lv[l].nblocks() * 2 > P0 ? pooled_levels : group_levels).push_back(l);
  // 1. the many-block levels, together
  for (int l : pooled_levels) {
    int rc = init_level(h, h->lv[l], hint(l) ? hint(l) : 64);
    if (rc) return rc;
  }
  for (int round = 0; round < 64 && !pooled_levels.empty(); ++round) {
    int kcap_max = 1;
    std::vector<std::pair<int64_t, AcaBlock>> sorted;
    for (int l : pooled_levels) {
      Level& L = h->lv[l];
      kcap_max = std::max(kcap_max, L.kcap);
      L.G = 1;
      for (int q = 0; q < L.nblocks(); ++q) {
        if (L.st[q].status == ACA_DONE) continue;
        AcaBlock B;
        fill_block(h, L, q, B);
        const int64_t k1 = pred_or(l, q);
        sorted.push_back({have_pred ? (int64_t)(B.m + B.n) * k1 * k1 : (int64_t)B.m * B.n, B});
      }
    }
    if (sorted.empty()) break;
    std::stable_sort(sorted.begin(), sorted.end(),
                     [](const std::pair<int64_t, AcaBlock>& a,
                        const std::pair<int64_t, AcaBlock>& b) { return a.first > b.first; });
    std::vector<AcaBlock> blocks;
    for (auto& pb : sorted) blocks.push_back(pb.second);
    int rc = run_aca(h, blocks, 1, 128, kcap_max);
    if (rc) return rc;
    bool all = true;
    for (int l : pooled_levels) {
      bool done;
      rc = sync_level(h, h->lv[l], &done);
      if (rc) return rc;
      all &= done;
    }
    if (all) break;
  }
  // 2. the few-block levels, in sets of neighbouring levels, deepest first:
  // the blocks of a set run in one launch (group_set_top)
  std::vector<double> rank_est((size_t)nlev, 0.0);
  double growth = 1.0;  // of the rank from one level to the next above it
  int known = -1;       // the uppermost level compressed so far
  auto note_rank = [&](int l) {
    rank_est[l] = std::max(1, level_kmax(h->lv[l]));
    if (known == l + 1 && rank_est[known] > 0)
      growth = std::min(1.5, std::max(1.0, rank_est[l] / rank_est[known]));
    known = l;
  };
  for (auto it = pooled_levels.rbegin(); it != pooled_levels.rend(); ++it) note_rank(*it);
  while (!group_levels.empty()) {
    for (auto it = group_levels.rbegin(); it != group_levels.rend(); ++it) {
      const int l = *it;
      const double below = l + 1 < nlev ? rank_est[l + 1] : 0.0;
      rank_est[l] = std::min((double)h->lv[l].ub_max, below > 0 ? below * growth : 32.0);
    }
    const int top = group_set_top(h, group_levels, rank_est);
    std::vector<int> set(group_levels.begin() + top, group_levels.end());
    group_levels.resize(top);
    for (int l : set) {
      const double below = l + 1 < nlev ? rank_est[l + 1] : 0.0;
      int rc = init_level(h, h->lv[l],
                          hint(l) ? hint(l) : std::max(64, ((int)below * 3 + 1) / 2 + 16));
      if (rc) return rc;
    }
    for (int round = 0; round < 256; ++round) {
      bool all = true;
      for (int l : set) all &= level_done(h->lv[l]);
      if (all) break;
      int rc = run_group_set(h, set, rank_est);
      if (rc) return rc;
      for (int l : set) {
        bool done;
        rc = sync_level(h, h->lv[l], &done);
        if (rc) return rc;
      }
    }
    for (auto it = set.rbegin(); it != set.rend(); ++it) note_rank(*it);
  }
  for (auto& L : h->lv)
    if (!level_done(L)) return fail(h, HODLR_ERR_STATE, "ACA did not converge in its launches");
  // ranks, level widths, column offsets, algorithmic bytes
  int64_t coff = 0;
  double bytes = 0;
  const double es = 8.0;  // bytes of a panel element
  for (auto& L : h->lv) {
    L.kmax = 0;
    for (int q = 0; q < L.nblocks(); ++q) {
      L.kmax = std::max(L.kmax, L.st[q].rank);
      int r0, c0, m, n;
      block_geom(L, q, r0, c0, m, n);
      // one read of the W and V panels per step (the norm dots ride along),
      // the two new columns and the coordinates of the entries evaluated
      double K = L.st[q].iters;
      bytes += (double)(m + n) * (es / 2.0 * K * (K - 1) + es * K + 8.0 * K * h->dim);
    }
    L.coff = (int)coff;
    coff += L.kmax;
  }
  h->C = coff;
  h->aca_bytes = bytes;
  h->compressed = true;
  return HODLR_OK;
}

int do_compress(hodlr_t h) {
  if (h->compressed) return HODLR_OK;
  h->aca_ring_fits = true;
  int rc = compress_levels(h);
  if (rc == HODLR_ERR_ALLOC && h->aca_ring) {
    // not with the group form's working layout, slots, published rows and dots:
    // once more with the panels loaded per thread, which needs none of them
    h->pool.free_scratch(h->stream);
    dfree(h, h->slots);
    dfree(h, h->pub);
    dfree(h, h->dotg);
    dfree(h, h->part);
    h->slots_cap = 0;
    h->pub_cap = h->dotg_cap = h->part_cap = 0;
    h->aca_ring_fits = false;
    rc = compress_levels(h);
  }
  return rc;
}

}  // namespace hodlr_impl
