// Device memory, host<->device copies, error words and handle set-up shared
// by the host orchestration units (handle.h).
#include "handle.h"

#include "common.cuh"

cudaError_t smem_opt_in(const void* fn, size_t dyn_bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> granted;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  size_t& have = granted[{dev, fn}];
  if (dyn_bytes <= have) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_bytes);
  if (e == cudaSuccess) have = dyn_bytes;
  return e;
}

namespace hodlr_impl {

// Device memory of every handle on a device comes from one stream-ordered
// pool owned by the library (cudaMallocFromPoolAsync / cudaFreeAsync) whose
// release threshold keeps freed memory reserved, so a new handle for the next
// system reuses the previous one's arenas instead of paying cudaMalloc /
// cudaFree for gigabytes.  hodlr_trim_device_memory hands it back.
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;

cudaMemPool_t device_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pools.find(dev);
  if (it != g_pools.end()) return it->second;
  cudaMemPoolProps props;
  memset(&props, 0, sizeof(props));
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
  uint64_t keep = UINT64_MAX;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  g_pools[dev] = pool;
  return pool;
}

int fail(hodlr_t h, int code, const std::string& msg) {
  if (h) h->err = msg;
  return code;
}

int cuda_fail(hodlr_t h, cudaError_t e, const char* where) {
  return fail(h, e == cudaErrorMemoryAllocation ? HODLR_ERR_ALLOC : HODLR_ERR_CUDA,
              std::string(where) + ": " + cudaGetErrorString(e));
}

void free_plan(hodlr_t h, DevPlan& p) {
  dfree(h, p.probs);
  dfree(h, p.tiles);
  p = DevPlan();
}

void drop_solve_graph(hodlr_t h) {
  if (h->sg_exec) cudaGraphExecDestroy(h->sg_exec);
  h->sg_exec = nullptr;
  h->sg_nrhs = -1;
}

void free_factor(hodlr_t h) {
  drop_solve_graph(h);
  ++h->factor_gen;
  for (auto& L : h->lv) {
    dfree(h, L.S);
    dfree(h, L.piv);
    dfree(h, L.d_nodes);
    dfree(h, L.perm);
    dfree(h, L.d_caps);
    dfree(h, L.d_stn);
    dfree(h, L.d_snn);
    free_plan(h, L.tn);
    free_plan(h, L.nn);
    free_plan(h, L.stn);
    free_plan(h, L.snn);
    L.solve_nrhs = -1;
    L.nodes.clear();
  }
  dfree(h, h->d_lu);
  dfree(h, h->d_lu_off);
  dfree(h, h->d_perm);
  for (auto& L : h->lv) {
    if (!L.y_alias) dfree(h, L.Yl);
    L.Yl = nullptr;
    L.y_alias = false;
  }
  if (h->w_consumed) h->compressed = false;  // the U panels are gone: compress again
  h->w_consumed = false;
  h->factored = false;
}

void free_compress(hodlr_t h) {
  free_factor(h);
  for (auto& L : h->lv) {
    dfree(h, L.W);
    dfree(h, L.V);
    dfree(h, L.cR);
    dfree(h, L.cC);
    dfree(h, L.prow);
    dfree(h, L.pcol);
    dfree(h, L.d_st);
    L.st.clear();
    L.kcap = 0;
  }
  h->compressed = false;
}

int ensure_ws(hodlr_t h, int64_t elems) {
  CK(dgrow(h, h->ws, h->ws_cap, elems));
  return HODLR_OK;
}

// Host copies on the handle's stream.  The handle's own stream is a
// non-blocking stream, so a synchronous cudaMemcpy (legacy default stream) is
// not ordered with its kernels; every copy goes through these instead and
// returns after the stream has drained.
// Each of them drains the stream, after which the pinned staging memory of
// h2d_async is free again.
static cudaError_t drained(hodlr_t h, cudaError_t e) {
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) h->pin_cur = h->pin_used = 0;
  return e;
}
cudaError_t h2d(hodlr_t h, void* dst, const void* src, size_t bytes) {
  return drained(h, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, h->stream));
}
cudaError_t d2h(hodlr_t h, void* dst, const void* src, size_t bytes) {
  return drained(h, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, h->stream));
}

// Pinned staging blocks, shared by all handles of the process.  Pinning and
// unpinning memory costs milliseconds (8 MB: 5 to 8 ms, now and then 100), more
// than a 4096-point system takes to solve, so a destroyed handle's blocks wait
// here, at most PIN_KEEP bytes, for the next handle; hodlr_trim_device_memory
// frees them.  A block belongs to one handle at a time and changes hands only
// after its stream has drained.  Measured on B200, a new system built, factored
// and solved once, blocks pinned per handle -> kept: N = 1024 13.4 -> 2.0 ms,
// N = 4096 13.2 -> 2.9 ms.
static std::mutex g_pin_mu;
static std::vector<PinBlock> g_pins;
static size_t g_pin_bytes = 0;
constexpr size_t PIN_BLOCK = (size_t)1 << 20;
constexpr size_t PIN_HANDLE = (size_t)8 << 20;  // a handle waits instead of going on
constexpr size_t PIN_KEEP = (size_t)64 << 20;

static cudaError_t take_pin(size_t need, PinBlock* out) {
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    size_t best = g_pins.size();  // the smallest that fits
    for (size_t i = 0; i < g_pins.size(); ++i)
      if (g_pins[i].bytes >= need && (best == g_pins.size() || g_pins[i].bytes < g_pins[best].bytes))
        best = i;
    if (best < g_pins.size()) {
      *out = g_pins[best];
      g_pins[best] = g_pins.back();
      g_pins.pop_back();
      g_pin_bytes -= out->bytes;
      return cudaSuccess;
    }
  }
  PinBlock b;
  b.bytes = (need + PIN_BLOCK - 1) / PIN_BLOCK * PIN_BLOCK;
  // any thread's next device may use it; and a failure is not left behind
  const cudaError_t e = cudaHostAlloc((void**)&b.p, b.bytes, cudaHostAllocPortable);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  *out = b;
  return cudaSuccess;
}

static void give_pin(const PinBlock& b) {
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    if (g_pin_bytes + b.bytes <= PIN_KEEP) {
      g_pins.push_back(b);
      g_pin_bytes += b.bytes;
      return;
    }
  }
  cudaFreeHost(b.p);
}

void release_pins(hodlr_t h) {
  for (auto& b : h->pins) give_pin(b);
  h->pins.clear();
  h->pin_cur = h->pin_used = 0;
}

void trim_pins() {
  std::vector<PinBlock> all;
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    all.swap(g_pins);
    g_pin_bytes = 0;
  }
  for (auto& b : all) cudaFreeHost(b.p);
}

// A pageable cudaMemcpyAsync to the device synchronises the stream before it
// starts, so the host would wait for every queued kernel before planning the
// next launches.  These uploads go through pinned staging memory instead:
// the host copies the bytes there and queues the copy.  The blocks are filled
// one after the other and reused once the stream has drained (any of the calls
// above), or here when a handle has filled PIN_HANDLE bytes.
cudaError_t h2d_async(hodlr_t h, void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return cudaSuccess;
  const size_t need = (bytes + 255) & ~(size_t)255;
  while (h->pin_cur < h->pins.size() && h->pin_used + need > h->pins[h->pin_cur].bytes) {
    ++h->pin_cur;
    h->pin_used = 0;
  }
  if (h->pin_cur == h->pins.size()) {
    size_t have = 0;
    for (auto& b : h->pins) have += b.bytes;
    if (have && have + need > PIN_HANDLE) {
      const cudaError_t e = cudaStreamSynchronize(h->stream);
      if (e != cudaSuccess) return e;
      h->pin_cur = h->pin_used = 0;
      while (h->pin_cur < h->pins.size() && need > h->pins[h->pin_cur].bytes) ++h->pin_cur;
      if (h->pin_cur == h->pins.size()) release_pins(h);  // one too small: take a larger one
    }
    if (h->pin_cur == h->pins.size()) {
      PinBlock b;
      const cudaError_t e = take_pin(need, &b);
      if (e != cudaSuccess) return e;
      h->pins.push_back(b);
    }
  }
  char* p = h->pins[h->pin_cur].p + h->pin_used;
  memcpy(p, src, bytes);
  h->pin_used += need;
  return cudaMemcpyAsync(dst, p, bytes, cudaMemcpyHostToDevice, h->stream);
}

// A[i][j] <-> A[j][i], 32 x 32 tiles swapped in pairs: one read and one write of
// the matrix at device bandwidth, where the host's strided pass over a row-major
// matrix took 17 ms at n = 2001.
__global__ void __launch_bounds__(256) transpose_square_kernel(double* A, int n) {
  __shared__ double up[32][33], lo[32][33];
  const int r = blockIdx.y * 32, c = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
  if (c < r) return;
  for (int k = ty; k < 32; k += 8) {
    if (r + k < n && c + tx < n) up[k][tx] = A[(int64_t)(r + k) * n + c + tx];
    if (c + k < n && r + tx < n) lo[k][tx] = A[(int64_t)(c + k) * n + r + tx];
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    if (r + k < n && c + tx < n) A[(int64_t)(r + k) * n + c + tx] = lo[tx][k];
    if (c != r && c + k < n && r + tx < n) A[(int64_t)(c + k) * n + r + tx] = up[tx][k];
  }
}

cudaError_t transpose_square(double* A, int n, cudaStream_t s) {
  const int t = (n + 31) / 32;
  if (t > 65535) return cudaErrorInvalidValue;
  transpose_square_kernel<<<dim3(t, t), dim3(32, 8), 0, s>>>(A, n);
  return cudaGetLastError();
}
cudaError_t copy2d(hodlr_t h, void* dst, size_t dpitch, const void* src, size_t spitch,
                   size_t width, size_t rows, cudaMemcpyKind kind) {
  return drained(h, cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, kind, h->stream));
}

int check_dev_err(hodlr_t h, const char* where) {
  unsigned e = 0;
  CK(d2h(h, &e, h->d_err, sizeof(unsigned)));
  if (e == 0) return HODLR_OK;
  CK(cudaMemsetAsync(h->d_err, 0, sizeof(unsigned), h->stream));
  if (e & DEV_ERR_TIMEOUT) return fail(h, HODLR_ERR_TIMEOUT, std::string(where) + ": device wait timed out");
  if (e & DEV_ERR_NONFINITE) return fail(h, HODLR_ERR_NONFINITE, std::string(where) + ": non-finite value");
  if (e & DEV_ERR_SINGULAR) return fail(h, HODLR_ERR_SINGULAR, std::string(where) + ": exact-zero pivot");
  if (e & DEV_ERR_INDEX) {
    std::string at;
    if (e & DEV_ERR_AT_LEAF_PERM) at += " [leaf permutation]";
    if (e & DEV_ERR_AT_SOLVE_PIV) at += " [capacitance solve pivots]";
    if (e & DEV_ERR_AT_BLOCKED_PIV) at += " [blocked solve pivots]";
    if (e & DEV_ERR_AT_LU_SWAP) at += " [multi-CTA LU interchanges]";
    return fail(h, HODLR_ERR_CHECK, std::string(where) + ": pivot or permutation index out of range" + at);
  }
  return fail(h, HODLR_ERR_CUDA, where);
}

int check_phase(hodlr_t h, const char* where) {
  if (!h->checked) return HODLR_OK;
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, where);
  return check_dev_err(h, where);
}

int check_extent(hodlr_t h, const void* p, size_t bytes, const char* what, const char* where) {
  if (!h->checked || bytes == 0 || h->pool.holds(p, bytes)) return HODLR_OK;
  char msg[256];
  snprintf(msg, sizeof msg, "%s: %s [%p, +%zu bytes) is outside the handle's allocations", where,
           what, p, bytes);
  return fail(h, HODLR_ERR_CHECK, msg);
}

int check_gemm(hodlr_t h, const std::vector<GemmProblem>& probs, bool tn, const char* where) {
  if (!h->checked) return HODLR_OK;
  const size_t e = sizeof(double);
  for (const auto& p : probs) {
    if (p.M <= 0 || p.N <= 0 || p.K <= 0) continue;
    // A: K x M (tn) or M x K, B: K x N, C: M x N, all column-major
    const size_t a = tn ? (size_t)(p.M - 1) * p.lda + p.K : (size_t)(p.K - 1) * p.lda + p.M;
    int rc = check_extent(h, p.A, a * e, "GEMM operand A", where);
    if (!rc) rc = check_extent(h, p.B, ((size_t)(p.N - 1) * p.ldb + p.K) * e, "GEMM operand B", where);
    if (!rc) rc = check_extent(h, p.C, ((size_t)(p.N - 1) * p.ldc + p.M) * e, "GEMM result C", where);
    if (!rc && p.splits > 1)
      rc = check_extent(h, h->ws + p.ws_off, (size_t)p.splits * p.M * p.N * e, "split-K slice",
                        where);
    if (rc) return rc;
  }
  return HODLR_OK;
}

EntrySrc make_src(hodlr_t h) {
  EntrySrc s;
  s.pts = h->d_pts;
  s.A = h->d_A;
  s.ld = h->n;
  s.kp = h->kp;
  s.dense = h->dense ? 1 : 0;
  s.kps = h->nsys ? h->d_kps : nullptr;
  s.psys = h->nsys ? h->d_psys : nullptr;
  return s;
}

int init_common(hodlr_t h) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, dev));
  int coop = 0;
  CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) return fail(h, HODLR_ERR_UNSUPPORTED, "device lacks cooperative launch");
  const char* chk = getenv("HODLR_CHECKED");
  h->checked = chk && *chk && strcmp(chk, "0") != 0;
  // HODLR_ACA_STREAMING=0|1|2: the ACA panel streaming mode of new handles
  // (hodlr_set_aca_streaming); unset or anything else keeps the default
  const char* acs = getenv("HODLR_ACA_STREAMING");
  if (acs && acs[0] >= '0' && acs[0] <= '2' && acs[1] == 0) {
    h->aca_ring = acs[0] != '0';
    h->aca_by_count = acs[0] == '1';
  }
  // HODLR_CAPACITANCE_SMEM=bytes: shared memory a CTA of a capacitance solve may
  // use in new handles; systems beyond it run from device memory
  const char* cap = getenv("HODLR_CAPACITANCE_SMEM");
  if (cap && atoll(cap) > 0) h->cap_smem = (size_t)std::min<long long>(atoll(cap), CAP_SMEM);
  CK(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking));
  h->stream = h->own_stream;
  CK(cudaEventCreate(&h->ev0));
  CK(cudaEventCreate(&h->ev1));
  CK(dalloc(h, &h->d_err, 1));
  CK(cudaMemsetAsync(h->d_err, 0, sizeof(unsigned), h->stream));
  build_tree(h);
  const int nl = (int)h->leaf_min.size();
  if (h->smax > 160) return fail(h, HODLR_ERR_UNSUPPORTED, "leaf size above 160");
  CK(dalloc(h, &h->d_leaf_min, (size_t)nl));
  CK(dalloc(h, &h->d_leaf_size, (size_t)nl));
  CK(h2d(h, h->d_leaf_min, h->leaf_min.data(), 4 * nl));
  CK(h2d(h, h->d_leaf_size, h->leaf_size.data(), 4 * nl));
  return HODLR_OK;
}

}  // namespace hodlr_impl
