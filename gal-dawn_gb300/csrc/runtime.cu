// Host runtime of libdawn_gb300.so: error state, device buffers, the driver
// that runs a single-source traversal as one conditional CUDA graph per
// source, CSR validation, in-edge (transpose) construction and the exact
// closeness reductions.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "dawn_device.cuh"

namespace dawn {

namespace {
thread_local char g_err[1024] = "";
}

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
void clear_error() { g_err[0] = 0; }
const char* last_error() { return g_err; }

namespace {
std::once_flag g_pool_once[64];
}

dawn_status pool_alloc(void** p, size_t bytes, cudaStream_t s) {
  int dev = 0;
  DAWN_CUDA(cudaGetDevice(&dev));
  std::call_once(g_pool_once[dev & 63], [dev]() {
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
  });
  DAWN_CUDA(cudaMallocAsync(p, bytes ? bytes : 16, s));
  return DAWN_OK;
}

void pool_free(void* p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

namespace {
std::mutex g_pin_mu;
std::vector<void*> g_pin_free;
constexpr int kPinnedChunkSlots = 64;
}  // namespace

dawn_status pinned_slot(void** p) {
  std::lock_guard<std::mutex> lock(g_pin_mu);
  if (g_pin_free.empty()) {
    char* chunk = nullptr;
    DAWN_CUDA(cudaMallocHost((void**)&chunk, kPinnedSlot * kPinnedChunkSlots));
    for (int i = kPinnedChunkSlots - 1; i >= 0; i--) g_pin_free.push_back(chunk + (size_t)i * kPinnedSlot);
  }
  *p = g_pin_free.back();
  g_pin_free.pop_back();
  return DAWN_OK;
}

void pinned_slot_release(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lock(g_pin_mu);
  g_pin_free.push_back(p);
}

dawn_status ensure(DevBuf& b, size_t bytes, cudaStream_t s) {
  if (bytes == 0) bytes = 16;
  if (b.bytes >= bytes) return DAWN_OK;
  if (b.p) pool_free(b.p, b.stream);
  b.p = nullptr;
  b.bytes = 0;
  DAWN_CHECK(pool_alloc(&b.p, bytes, s));
  b.bytes = bytes;
  b.stream = s;
  return DAWN_OK;
}

void release(DevBuf& b) {
  if (b.p) pool_free(b.p, b.stream);
  b.p = nullptr;
  b.bytes = 0;
}

bool cluster_fits(const void* fn, int ctas, int threads) {
  static std::mutex mu;
  static std::vector<std::pair<const void*, bool>> known;
  std::lock_guard<std::mutex> lock(mu);
  for (const auto& k : known)
    if (k.first == fn) return k.second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  int clusters = 0;
  const bool fits = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0;
  cudaGetLastError();
  known.emplace_back(fn, fits);
  return fits;
}

int persistent_blocks(const void* fn, int block, size_t smem, int cap) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  if (cap > 0 && cap < per_sm) per_sm = cap;
  return sms * per_sm;
}

dawn_status upload_ctl(dawn_graph* g, const SsCtl& c) {
  // Pageable source: the runtime stages it before returning, so the stack
  // copy may go out of scope while the transfer is still queued.
  g->ss_call = g->ss_ctl.as<SsCtl>();
  DAWN_CUDA(cudaMemcpyAsync(g->ss_ctl.p, &c, sizeof(SsCtl), cudaMemcpyHostToDevice, g->stream));
  return DAWN_OK;
}

dawn_status download_ctl(dawn_graph* g, SsCtl* out) {
  DAWN_CUDA(cudaMemcpyAsync(&g->h_ctl[1], g->ss_call, sizeof(SsCtl), cudaMemcpyDeviceToHost, g->stream));
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  *out = g->h_ctl[1];
  return DAWN_OK;
}

namespace {

// The persisting-L2 carve-out of each device, set once to the device's
// maximum (a limit of this process's context; it ends with the process).
struct L2Persist {
  std::once_flag once;
  size_t carve = 0, max_window = 0;
};
L2Persist g_l2[64];

// Access-policy window of a family's body kernels: its hot arrays (the
// frontier words every level gathers from) marked persisting, so the edge
// arrays that stream through L2 at every level do not evict them.
bool family_window(const SsFamily& fam, cudaAccessPolicyWindow* w) {
  if (!fam.l2_base || fam.l2_bytes == 0) return false;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  L2Persist& p = g_l2[dev];
  std::call_once(p.once, [&p, dev] {
    int carve = 0, win = 0;
    if (cudaDeviceGetAttribute(&carve, cudaDevAttrMaxPersistingL2CacheSize, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&win, cudaDevAttrMaxAccessPolicyWindowSize, dev) != cudaSuccess || carve <= 0 ||
        win <= 0 || cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, (size_t)carve) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    p.carve = (size_t)carve;
    p.max_window = (size_t)win;
  });
  if (p.carve == 0) return false;
  w->base_ptr = const_cast<void*>(fam.l2_base);
  w->num_bytes = fam.l2_bytes < p.max_window ? fam.l2_bytes : p.max_window;
  w->hitRatio = (float)((double)p.carve / (double)w->num_bytes);
  if (w->hitRatio > 1.0f) w->hitRatio = 1.0f;
  w->hitProp = cudaAccessPropertyPersisting;
  w->missProp = cudaAccessPropertyStreaming;
  return true;
}

dawn_status add_kernel(cudaGraph_t graph, cudaGraphNode_t* node, const cudaGraphNode_t* dep, const Launch& l,
                       const cudaAccessPolicyWindow* w = nullptr) {
  cudaKernelNodeParams p = {};
  p.func = const_cast<void*>(l.fn);
  p.gridDim = l.grid;
  p.blockDim = l.block;
  p.sharedMemBytes = (unsigned)l.smem;
  p.kernelParams = l.args;
  p.extra = nullptr;
  DAWN_CUDA(cudaGraphAddKernelNode(node, graph, dep, dep ? 1 : 0, &p));
  if (w) {
    cudaKernelNodeAttrValue v = {};
    v.accessPolicyWindow = *w;
    DAWN_CUDA(cudaGraphKernelNodeSetAttribute(*node, cudaKernelNodeAttributeAccessPolicyWindow, &v));
  }
  return DAWN_OK;
}

dawn_status build_graph(SsFamily& fam, cudaGraphExec_t* exec) {
  cudaGraph_t graph = nullptr;
  DAWN_CUDA(cudaGraphCreate(&graph, 0));
  dawn_status st = DAWN_OK;
  do {
    cudaGraphNode_t prev = nullptr, node = nullptr, loop = nullptr;
    for (int i = 0; i < fam.npre && st == DAWN_OK; i++) {
      st = add_kernel(graph, &node, prev ? &prev : nullptr, fam.pre[i]);
      prev = node;
    }
    if (st != DAWN_OK) break;
    cudaGraphConditionalHandle h = 0;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) {
      set_error("cudaGraphConditionalHandleCreate: %s", cudaGetErrorString(e));
      st = DAWN_ERR_CUDA;
      break;
    }
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    e = cudaGraphAddNode(&loop, graph, prev ? &prev : nullptr, nullptr, prev ? 1 : 0, &cp);
    if (e != cudaSuccess) {
      set_error("cudaGraphAddNode(while): %s", cudaGetErrorString(e));
      st = DAWN_ERR_CUDA;
      break;
    }
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    *fam.handle = h;
    *fam.in_graph = 1;
    cudaAccessPolicyWindow win;
    const bool has_win = family_window(fam, &win);
    cudaGraphNode_t bprev = nullptr;
    for (int i = 0; i < fam.nbody && st == DAWN_OK; i++) {
      st = add_kernel(body, &node, bprev ? &bprev : nullptr, fam.body[i], has_win ? &win : nullptr);
      bprev = node;
    }
    if (st != DAWN_OK) break;
    cudaGraphNode_t pprev = loop;
    for (int i = 0; i < fam.npost && st == DAWN_OK; i++) {
      st = add_kernel(graph, &node, &pprev, fam.post[i]);
      pprev = node;
    }
    if (st != DAWN_OK) break;
    e = cudaGraphInstantiate(exec, graph, 0);
    if (e != cudaSuccess) {
      set_error("cudaGraphInstantiate: %s", cudaGetErrorString(e));
      *exec = nullptr;
      st = DAWN_ERR_CUDA;
      break;
    }
  } while (0);
  cudaGraphDestroy(graph);
  *fam.in_graph = 0;
  *fam.handle = 0;
  return st;
}

dawn_status launch(const Launch& l, cudaStream_t s, const cudaAccessPolicyWindow* w = nullptr) {
  if (!w) {
    DAWN_CUDA(cudaLaunchKernel(l.fn, l.grid, l.block, l.args, l.smem, s));
    return DAWN_OK;
  }
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeAccessPolicyWindow;
  attr.val.accessPolicyWindow = *w;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = l.grid;
  cfg.blockDim = l.block;
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  DAWN_CUDA(cudaLaunchKernelExC(&cfg, l.fn, l.args));
  return DAWN_OK;
}

constexpr int kPollLevels = 4;  // host-loop form: levels launched between polls

}  // namespace

// Traced form: level by level from the host, CUDA events around each kernel
// that does work at that level, one trace record per kernel.
dawn_status ss_run_traced(dawn_graph* g, SsFamily& fam, int32_t nruns) {
  if (fam.in_graph) *fam.in_graph = 0;
  cudaAccessPolicyWindow win;
  const bool has_win = family_window(fam, &win);
  for (int i = 0; i < 10; i++)
    if (!g->trace_ev[i]) DAWN_CUDA(cudaEventCreate(&g->trace_ev[i]));
  std::vector<unsigned char> host(fam.ctl_bytes);
  struct Pending {
    int body;
    LevelProbe p;
  };
  // Times the launches of one stage (pre or post kernels) as level 0 / -1 records.
  auto timed_stage = [&](const Launch* ls, int cnt, int run, int level) -> dawn_status {
    for (int j = 0; j < cnt; j++) {
      DAWN_CUDA(cudaEventRecord(g->trace_ev[0], g->stream));
      DAWN_CHECK(launch(ls[j], g->stream));
      DAWN_CUDA(cudaEventRecord(g->trace_ev[1], g->stream));
      DAWN_CUDA(cudaEventSynchronize(g->trace_ev[1]));
      dawn_trace_rec r = {};
      std::snprintf(r.kernel, sizeof(r.kernel), "%s", ls[j].name);
      r.run = run;
      r.level = level;
      r.mode = -1;
      DAWN_CUDA(cudaEventElapsedTime(&r.ms, g->trace_ev[0], g->trace_ev[1]));
      g->trace_log.push_back(r);
    }
    return DAWN_OK;
  };
  for (int32_t run = 0; run < nruns; run++) {
    DAWN_CHECK(timed_stage(fam.pre, fam.npre, run, 0));
    for (;;) {
      DAWN_CUDA(cudaMemcpyAsync(host.data(), fam.ctl, fam.ctl_bytes, cudaMemcpyDeviceToHost, g->stream));
      DAWN_CUDA(cudaStreamSynchronize(g->stream));
      LevelProbe p;
      fam.probe(host.data(), &p);
      if (p.done) break;
      Pending pend[5];
      int np = 0;
      const int nwork = fam.decide_in_body ? fam.nbody : fam.nbody - 1;
      for (int b = 0; b < nwork; b++) {
        const int bm = fam.body[b].mode;
        const bool match = bm < 0 || bm == p.mode || (bm == kModeStep && (p.mode == kModePush || p.mode == kModePull));
        if (!match) continue;
        DAWN_CUDA(cudaEventRecord(g->trace_ev[2 * np], g->stream));
        DAWN_CHECK(launch(fam.body[b], g->stream, has_win ? &win : nullptr));
        DAWN_CUDA(cudaEventRecord(g->trace_ev[2 * np + 1], g->stream));
        pend[np++] = {b, p};
        if (fam.decide_in_body) break;  // the kernel ran the level and its bookkeeping
      }
      if (!fam.decide_in_body) DAWN_CHECK(launch(fam.body[fam.nbody - 1], g->stream, has_win ? &win : nullptr));
      DAWN_CUDA(cudaStreamSynchronize(g->stream));
      for (int i = 0; i < np; i++) {
        dawn_trace_rec r = {};
        std::snprintf(r.kernel, sizeof(r.kernel), "%s", fam.body[pend[i].body].name);
        r.run = run;
        r.level = pend[i].p.level;
        r.mode = pend[i].p.mode;
        r.frontier = pend[i].p.frontier;
        r.frontier_edges = pend[i].p.frontier_edges;
        r.unvisited_edges = pend[i].p.unvisited_edges;
        DAWN_CUDA(cudaEventElapsedTime(&r.ms, g->trace_ev[2 * i], g->trace_ev[2 * i + 1]));
        g->trace_log.push_back(r);
      }
    }
    DAWN_CHECK(timed_stage(fam.post, fam.npost, run, -1));
  }
  return DAWN_OK;
}

dawn_status launch_cooperative(const SsFamily& fam, const void* fn, int ctas, int threads, void** args,
                               cudaStream_t s) {
  cudaAccessPolicyWindow win;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (family_window(fam, &win)) {
    attr[1].id = cudaLaunchAttributeAccessPolicyWindow;
    attr[1].val.accessPolicyWindow = win;
    cfg.numAttrs = 2;
  }
  DAWN_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  return DAWN_OK;
}

dawn_status device_status(dawn_graph* g) {
  const int32_t e = *static_cast<volatile int32_t*>(g->h_err);
  if (!e) return DAWN_OK;
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  *static_cast<volatile int32_t*>(g->h_err) = 0;
  // what the launches expect as the last one should have left it: the arrivals of
  // bfs_traverse, the touched bitmap, the accumulators of heavy rows, the counts
  // of betweenness
  release(g->bfs_sync);
  release(g->bs_queues);
  if (g->hv_acc.p) DAWN_CUDA(cudaMemsetAsync(g->hv_acc.p, 0, g->hv_acc.bytes, g->stream));
  g->bc_blocks = 0;
  set_error("a device wait ran out: the results of this call, or of an earlier one on this handle, are unfinished");
  return e;
}

dawn_status ss_run(dawn_graph* g, SsFamily& fam, int32_t nruns, cudaGraphExec_t* exec) {
  if (g->trace && fam.probe) return ss_run_traced(g, fam, nruns);
  if (g->graphs_ok && !*exec) {
    if (build_graph(fam, exec) != DAWN_OK) {
      g->graphs_ok = false;  // report once, then run the host level loop
      std::fprintf(stderr, "dawn: conditional graphs unavailable (%s); using the host level loop\n",
                   last_error());
      cudaGetLastError();
      clear_error();
    }
  }
  if (g->graphs_ok && *exec) {
    for (int32_t i = 0; i < nruns; i++) DAWN_CUDA(cudaGraphLaunch(*exec, g->stream));
    return DAWN_OK;
  }
  *fam.in_graph = 0;
  cudaAccessPolicyWindow win;
  const bool has_win = family_window(fam, &win);
  int32_t* h_done = &g->h_ctl[1].done;
  for (int32_t i = 0; i < nruns; i++) {
    for (int j = 0; j < fam.npre; j++) DAWN_CHECK(launch(fam.pre[j], g->stream));
    for (;;) {
      for (int j = 0; j < kPollLevels; j++)
        for (int b = 0; b < fam.nbody; b++) DAWN_CHECK(launch(fam.body[b], g->stream, has_win ? &win : nullptr));
      DAWN_CUDA(cudaMemcpyAsync(h_done, fam.done_flag, sizeof(int32_t), cudaMemcpyDeviceToHost, g->stream));
      DAWN_CUDA(cudaStreamSynchronize(g->stream));
      if (*h_done) break;
    }
    for (int j = 0; j < fam.npost; j++) DAWN_CHECK(launch(fam.post[j], g->stream));
  }
  return DAWN_OK;
}

// --- CSR validation -----------------------------------------------------------

namespace {

// Weight k of the handle's own copy, as a word; a float -0.0 (what -log(1.0f)
// gives) becomes 0.0 there first.  The traversals compare distances as words, and
// its word, 0x80000000, sorts above every distance as unsigned and below them as
// signed.
__device__ __forceinline__ int32_t weight_word(int32_t* val, int wtype, size_t k) {
  const int32_t w = val[k];
  if (wtype != DAWN_W_F32 || w != INT_MIN) return w;
  val[k] = 0;
  return 0;
}

__device__ __forceinline__ int check_entry(int32_t c, int32_t n, int32_t* val, int wtype, size_t k) {
  int f = (c < 0 || c >= n) ? 8 : 0;
  if (wtype == DAWN_W_NONE) return f;
  const int32_t w = weight_word(val, wtype, k);
  if (w < 0 || (wtype == DAWN_W_F32 && !isfinite(__int_as_float(w)))) f |= 16;
  return f;
}

// One pass over row_ptr and col (128-bit loads) checking the CSR invariants
// the kernels rely on: monotone row_ptr from 0 to m, columns in [0, n),
// weights finite and non-negative.
__global__ void validate_csr_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                    int32_t* __restrict__ val, int wtype, int32_t n, long long m,
                                    int* __restrict__ flags) {
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  int f = 0;
  if (tid == 0) {
    if (rp[0] != 0) f |= 1;
    if ((long long)rp[n] != m) f |= 2;
  }
  for (size_t i = tid; i < (size_t)n; i += stride)
    if (rp[i] > rp[i + 1]) f |= 4;
  const size_t m4 = (size_t)m / 4;
  const int4* c4 = reinterpret_cast<const int4*>(col);
  for (size_t q = tid; q < m4; q += stride) {
    const int4 c = c4[q];
    const int32_t cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; j++) f |= check_entry(cc[j], n, val, wtype, 4 * q + j);
  }
  for (size_t k = 4 * m4 + tid; k < (size_t)m; k += stride) f |= check_entry(col[k], n, val, wtype, k);
  if (f) atomicOr(flags, f);
}

// Whether any weight has its sign bit set (-0.0 aside).
__global__ void weight_signs(int32_t* __restrict__ val, int wtype, long long m, int* __restrict__ flag) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  bool neg = false;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < (size_t)m; k += stride)
    neg |= weight_word(val, wtype, k) < 0;
  if (neg) atomicOr(flag, 1);
}

}  // namespace

dawn_status read_weight_signs(dawn_graph* g) {
  if (g->wtype == DAWN_W_NONE) return DAWN_OK;
  int *d_flag = nullptr, flag = 0;
  DAWN_CHECK(pool_alloc((void**)&d_flag, sizeof(int), g->stream));
  DAWN_CUDA(cudaMemsetAsync(d_flag, 0, sizeof(int), g->stream));
  weight_signs<<<g->geo.sms * 8, kBlock, 0, g->stream>>>(static_cast<int32_t*>(g->val), g->wtype, g->m, d_flag);
  DAWN_CUDA(cudaGetLastError());
  DAWN_CUDA(cudaMemcpyAsync(&flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
  pool_free(d_flag, g->stream);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  g->negative_weights = flag != 0;
  return DAWN_OK;
}

dawn_status validate_csr(dawn_graph* g) {
  int* d_flags = nullptr;
  DAWN_CUDA(cudaMallocAsync(&d_flags, sizeof(int), g->stream));
  DAWN_CUDA(cudaMemsetAsync(d_flags, 0, sizeof(int), g->stream));
  validate_csr_kernel<<<g->geo.sms * 8, kBlock, 0, g->stream>>>(g->row_ptr, g->col, static_cast<int32_t*>(g->val),
                                                                 g->wtype, g->n, g->m, d_flags);
  DAWN_CUDA(cudaGetLastError());
  int flags = 0;
  DAWN_CUDA(cudaMemcpyAsync(&flags, d_flags, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
  DAWN_CUDA(cudaFreeAsync(d_flags, g->stream));
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  if (flags) {
    set_error("invalid CSR:%s%s%s%s%s", (flags & 1) ? " row_ptr[0] != 0;" : "",
              (flags & 2) ? " row_ptr[n] != m;" : "", (flags & 4) ? " row_ptr decreases;" : "",
              (flags & 8) ? " col index outside [0, n);" : "",
              (flags & 16) ? " negative or non-finite weight;" : "");
    return DAWN_ERR_INVALID_ARG;
  }
  return DAWN_OK;
}

// --- longest row --------------------------------------------------------------

namespace {

__global__ void __launch_bounds__(kBlock) max_degree(const int32_t* __restrict__ row_ptr, int32_t n,
                                                     int32_t* __restrict__ out) {
  int deg = 0;
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    deg = max(deg, row_ptr[v + 1] - row_ptr[v]);
  deg = __reduce_max_sync(kFull, deg);
  if (lane_id() == 0 && deg) atomicMax(out, deg);
}

}  // namespace

dawn_status longest_row(dawn_graph* g) {
  if (g->max_row >= 0) return DAWN_OK;
  int32_t* d = nullptr;
  int32_t deg = 0;
  DAWN_CHECK(pool_alloc((void**)&d, sizeof(int32_t), g->stream));
  DAWN_CUDA(cudaMemsetAsync(d, 0, sizeof(int32_t), g->stream));
  max_degree<<<g->geo.sms * 4, kBlock, 0, g->stream>>>(g->row_ptr, g->n, d);
  DAWN_CUDA(cudaGetLastError());
  DAWN_CUDA(cudaMemcpyAsync(&deg, d, sizeof(int32_t), cudaMemcpyDeviceToHost, g->stream));
  pool_free(d, g->stream);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  g->max_row = deg;
  return DAWN_OK;
}

// --- growth ---------------------------------------------------------------------

namespace {

constexpr int kGrowthSamples = 4, kGrowthReach = 8192, kGrowthLevels = 16;

// How fast the neighbourhoods of a few vertices grow: one CTA per sample walks
// levels until it has seen `reach` vertices, for kGrowthLevels at most.
// out: levels, vertices seen.
__global__ void __launch_bounds__(1024) grow(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                                             int32_t n, int reach, uint32_t* bitmaps, size_t nwords, int32_t* queues,
                                             int2* __restrict__ out) {
  __shared__ int s_count, s_start;
  uint32_t* const seen = bitmaps + blockIdx.x * nwords;
  int32_t* const q = queues + (size_t)blockIdx.x * reach;
  const int lane = lane_id();
  if (threadIdx.x == 0) s_start = n;
  __syncthreads();
  // the first vertex with a row, of 1,024 from the sample's place on
  const int32_t v0 = (int32_t)((long long)n * (2 * blockIdx.x + 1) / (2 * kGrowthSamples));
  if (threadIdx.x < n - v0 && row_ptr[v0 + threadIdx.x] < row_ptr[v0 + threadIdx.x + 1])
    atomicMin(&s_start, v0 + (int)threadIdx.x);
  __syncthreads();
  if (s_start == n) {
    if (threadIdx.x == 0) out[blockIdx.x] = make_int2(0, 0);
    return;
  }
  if (threadIdx.x == 0) {
    q[0] = s_start;
    seen[s_start >> 5] |= 1u << (s_start & 31);
    s_count = 1;
  }
  int lo = 0, L = 0;
  for (;; L++) {
    __syncthreads();
    const int hi = s_count;
    __syncthreads();
    if (hi >= reach || hi == lo || L == kGrowthLevels) break;
    for (int i = lo + (int)(threadIdx.x >> 5); i < hi; i += 32) {
      const int32_t v = q[i];
      const int e = row_ptr[v + 1];
      for (int k = row_ptr[v] + lane; k < e; k += 32) {
        const int32_t u = col[k];
        const uint32_t bit = 1u << (u & 31);
        if (atomicOr(seen + (u >> 5), bit) & bit) continue;
        const int at = atomicAdd(&s_count, 1);
        if (at < reach) q[at] = u;
      }
    }
    lo = hi;
  }
  if (threadIdx.x == 0) out[blockIdx.x] = make_int2(L, s_count);
}

}  // namespace

dawn_status read_growth(dawn_graph* g) {
  if (g->growth >= 0.0) return DAWN_OK;
  const int reach = std::max(64, std::min(kGrowthReach, g->n / 2));
  const size_t nwords = ((size_t)g->n + 31) / 32;
  const size_t words = 2 * kGrowthSamples + kGrowthSamples * (nwords + (size_t)reach);
  int32_t* d = nullptr;
  int2 h[kGrowthSamples];
  const dawn_status s = pool_alloc((void**)&d, sizeof(int32_t) * words, g->stream);
  if (s == DAWN_ERR_OOM) {  // not read: taken as a mesh by this call
    cudaGetLastError();
    clear_error();
    return DAWN_OK;
  }
  DAWN_CHECK(s);
  uint32_t* const bitmaps = reinterpret_cast<uint32_t*>(d + 2 * kGrowthSamples);
  cudaError_t e = cudaMemsetAsync(bitmaps, 0, sizeof(uint32_t) * kGrowthSamples * nwords, g->stream);
  grow<<<kGrowthSamples, 1024, 0, g->stream>>>(g->row_ptr, g->col, g->n, reach, bitmaps, nwords,
                                                d + 2 * kGrowthSamples + kGrowthSamples * nwords,
                                                reinterpret_cast<int2*>(d));
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
  pool_free(d, g->stream);
  DAWN_CUDA(e);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  // per level, of the samples that reached far enough; 1 for those that did not
  // within the levels or at all
  double most = 1.0;
  for (const int2& x : h)
    if (x.x > 0 && x.y >= reach) most = std::max(most, std::pow((double)x.y, 1.0 / x.x));
  g->growth = most;
  return DAWN_OK;
}

// --- exclusive scan (int64), used for the in-edge CSR ---------------------------

namespace {

constexpr int kScanBlock = 1024;

__global__ void __launch_bounds__(kScanBlock) scan_block(const int64_t* __restrict__ in, int64_t* __restrict__ out,
                                                         long long n, int64_t* __restrict__ sums) {
  __shared__ long long warp_tot[kScanBlock / 32];
  const long long i = blockIdx.x * (long long)kScanBlock + threadIdx.x;
  const long long x = i < n ? in[i] : 0;
  long long v = x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    long long y = __shfl_up_sync(kFull, v, d);
    if (lane >= d) v += y;
  }
  if (lane == 31) warp_tot[w] = v;
  __syncthreads();
  if (w == 0) {
    long long t = warp_tot[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      long long y = __shfl_up_sync(kFull, t, d);
      if (lane >= d) t += y;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  const long long incl = v + (w ? warp_tot[w - 1] : 0);
  if (i < n) out[i] = incl - x;
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = incl;
}

__global__ void add_block_offsets(int64_t* __restrict__ out, long long n, const int64_t* __restrict__ offs) {
  const long long i = blockIdx.x * (long long)kScanBlock + threadIdx.x;
  if (i < n) out[i] += offs[blockIdx.x];
}

}  // namespace

dawn_status exclusive_scan_i64(const int64_t* d_in, int64_t* d_out, int64_t n, cudaStream_t s) {
  if (n <= 0) return DAWN_OK;
  const long long nb = (n + kScanBlock - 1) / kScanBlock;
  int64_t* sums = nullptr;
  DAWN_CUDA(cudaMallocAsync(&sums, sizeof(int64_t) * 2 * nb, s));
  scan_block<<<(unsigned)nb, kScanBlock, 0, s>>>(d_in, d_out, n, sums);
  DAWN_CUDA(cudaGetLastError());
  if (nb > 1) {
    DAWN_CHECK(exclusive_scan_i64(sums, sums + nb, nb, s));
    add_block_offsets<<<(unsigned)nb, kScanBlock, 0, s>>>(d_out, n, sums + nb);
    DAWN_CUDA(cudaGetLastError());
  }
  DAWN_CUDA(cudaFreeAsync(sums, s));
  return DAWN_OK;
}

// --- in-edge CSR -------------------------------------------------------------------

namespace {

__global__ void count_in_degree(const int32_t* __restrict__ col, long long m,
                                unsigned long long* __restrict__ deg) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < (size_t)m; k += stride)
    atomicAdd(deg + col[k], 1ull);
}

__global__ void offsets_to_rowptr(const int64_t* __restrict__ off, int32_t* __restrict__ rp,
                                  unsigned long long* __restrict__ cursor, int32_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i <= (size_t)n; i += stride) {
    rp[i] = (int32_t)off[i];
    cursor[i] = (unsigned long long)off[i];
  }
}

__global__ void scatter_in_edges(const int32_t* __restrict__ rp, const int32_t* __restrict__ col, int32_t n,
                                 unsigned long long* __restrict__ cursor, int32_t* __restrict__ t_col) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    const int e = rp[u + 1];
    for (int k = rp[u] + lane; k < e; k += 32) {
      const int32_t v = col[k];
      t_col[atomicAdd(cursor + v, 1ull)] = u;
    }
  }
}

// Where a row's light entries go (from its start up) and its others (from its
// end down).
__global__ void init_cursors(const int32_t* __restrict__ t_row_ptr, int2* __restrict__ cursor, int32_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += stride)
    cursor[i] = make_int2(t_row_ptr[i], t_row_ptr[i + 1]);
}

// The light entries' end of every row, and the vertex of most in-edges.
__global__ void finish_weighted_in_edges(const int32_t* __restrict__ t_row_ptr, const int2* __restrict__ cursor,
                                         int32_t n, int32_t* __restrict__ light, unsigned long long* __restrict__ hub) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  unsigned long long best = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += stride) {
    light[i] = cursor[i].x;
    const unsigned long long x = (unsigned long long)(t_row_ptr[i + 1] - t_row_ptr[i]) << 32 | (unsigned)i;
    best = x > best ? x : best;
  }
#pragma unroll
  for (int d = 16; d; d >>= 1) {
    const unsigned long long x = __shfl_xor_sync(kFull, best, d);
    best = x > best ? x : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(hub, best);
}

__global__ void scatter_weighted_in_edges(const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                          const int32_t* __restrict__ val, int32_t n, uint32_t most,
                                          int2* __restrict__ cursor, int32_t* __restrict__ t_col,
                                          int32_t* __restrict__ t_val) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    const int e = rp[u + 1];
    for (int k = rp[u] + lane; k < e; k += 32) {
      const int32_t w = val[k];
      int2* const c = cursor + col[k];
      const int slot = (uint32_t)w <= most ? atomicAdd(&c->x, 1) : atomicSub(&c->y, 1) - 1;
      t_col[slot] = u;
      t_val[slot] = w;
    }
  }
}

__global__ void sample_weights(const int32_t* __restrict__ val, long long m, int samples, int32_t* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < samples; i += gridDim.x * blockDim.x)
    out[i] = val[(long long)i * m / samples];
}

}  // namespace

// The light weights, from a sample of 4,096: about three entries a vertex (an eighth
// to a half of them).  A stage of their own pays where two of them in a row are
// shorter than most other edges.  64 sources on RMAT-18, ms with the stage / without
// / whole pulls alone: lengths 1-63 1.25 / 1.9 / 2.5, 1-4 1.49 / 1.66 / 1.88, 1-3
// 1.56 / 1.60 / 1.83, 1-2 1.93 / 1.50 / 1.54, 61-123 1.95 / 1.51 / 1.55, equal
// 2.1 / 1.48 / 1.50; on RMAT-20 with four entries a vertex 1-63 2.4 / 3.5 / 3.4.
dawn_status light_weights(dawn_graph* g) {
  if (g->light_read) return DAWN_OK;
  constexpr int kSamples = 4096;
  constexpr double kHeavier = 2.6;  // mean of the others, in means of the light ones
  const int samples = (int)std::min<int64_t>(g->m, kSamples);
  g->light_most = 0;
  g->light_pays = false;
  if (samples > 0) {
    std::vector<uint32_t> w((size_t)samples);
    int32_t* d = nullptr;
    DAWN_CHECK(pool_alloc((void**)&d, sizeof(int32_t) * w.size(), g->stream));
    sample_weights<<<16, kBlock, 0, g->stream>>>(static_cast<const int32_t*>(g->val), g->m, samples, d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(w.data(), d, sizeof(uint32_t) * w.size(), cudaMemcpyDeviceToHost, g->stream);
    pool_free(d, g->stream);
    DAWN_CUDA(e);
    DAWN_CUDA(cudaStreamSynchronize(g->stream));
    const double share = std::min(0.5, std::max(0.125, 3.0 * g->n / (double)g->m));
    std::sort(w.begin(), w.end());
    g->light_most = w[(size_t)(share * (double)(w.size() - 1))];
    double sum[2] = {0.0, 0.0};
    size_t cnt[2] = {0, 0};
    for (uint32_t x : w) {
      float f;
      std::memcpy(&f, &x, sizeof(f));
      const int heavy = x > g->light_most;
      sum[heavy] += g->wtype == DAWN_W_F32 ? (double)f : (double)x;
      cnt[heavy]++;
    }
    g->light_pays = (double)cnt[0] <= 0.6 * samples && kHeavier * sum[0] / cnt[0] < sum[1] / cnt[1];
  }
  g->light_read = true;
  return DAWN_OK;
}

// In-edges with their weights, a row's light entries first, for the batched
// traversal, which reaches most of its distances through these alone.
dawn_status build_weighted_in_edges(dawn_graph* g) {
  if (g->wt_col.p) return DAWN_OK;
  const int32_t n = g->n;
  const cudaStream_t s = g->stream;
  const int grid = g->geo.sms * 8;
  DAWN_CHECK(light_weights(g));
  int2* cursor = nullptr;
  DAWN_CHECK(pool_alloc((void**)&cursor, sizeof(int2) * (size_t)n + sizeof(unsigned long long), s));
  unsigned long long* const hub = reinterpret_cast<unsigned long long*>(cursor + n);
  DAWN_CUDA(cudaMemsetAsync(hub, 0, sizeof(*hub), s));
  DAWN_CHECK(ensure(g->wt_light, sizeof(int32_t) * (size_t)n, s));
  DAWN_CHECK(ensure(g->wt_val, sizeof(int32_t) * (size_t)(g->m > 0 ? g->m : 1) + 16, s));
  DAWN_CHECK(ensure(g->wt_col, sizeof(int32_t) * (size_t)(g->m > 0 ? g->m : 1) + 16, s));
  init_cursors<<<grid, kBlock, 0, s>>>(g->t_row_ptr, cursor, n);
  DAWN_CUDA(cudaGetLastError());
  // 32-bit weights (int32 or float32 bit patterns, not negative) move as words
  scatter_weighted_in_edges<<<grid, kBlock, 0, s>>>(g->row_ptr, g->col, static_cast<const int32_t*>(g->val), n,
                                                    g->light_most, cursor, g->wt_col.as<int32_t>(),
                                                    g->wt_val.as<int32_t>());
  DAWN_CUDA(cudaGetLastError());
  finish_weighted_in_edges<<<g->geo.sms * 4, kBlock, 0, s>>>(g->t_row_ptr, cursor, n, g->wt_light.as<int32_t>(), hub);
  DAWN_CUDA(cudaGetLastError());
  unsigned long long h = 0;
  DAWN_CUDA(cudaMemcpyAsync(&h, hub, sizeof(h), cudaMemcpyDeviceToHost, s));
  pool_free(cursor, s);
  DAWN_CUDA(cudaStreamSynchronize(s));
  g->wt_hub = (int32_t)(uint32_t)h;
  // Without a hub the bounds leave too much for a light stage to pay, and without a
  // light stage they leave too much of a hub's rows: both or neither.
  g->wt_has_light = g->light_pays && (double)(h >> 32) * n >= kHubDegree * (double)g->m;
  return DAWN_OK;
}

dawn_status build_transpose(dawn_graph* g) {
  const int32_t n = g->n;
  const cudaStream_t s = g->stream;
  unsigned long long* deg = nullptr;
  int64_t* off = nullptr;
  DAWN_CUDA(cudaMallocAsync(&deg, sizeof(unsigned long long) * ((size_t)n + 1), s));
  DAWN_CUDA(cudaMallocAsync(&off, sizeof(int64_t) * ((size_t)n + 1), s));
  DAWN_CUDA(cudaMemsetAsync(deg, 0, sizeof(unsigned long long) * ((size_t)n + 1), s));
  const int grid = g->geo.sms * 8;
  count_in_degree<<<grid, kBlock, 0, s>>>(g->col, g->m, deg);
  DAWN_CUDA(cudaGetLastError());
  DAWN_CHECK(exclusive_scan_i64(reinterpret_cast<const int64_t*>(deg), off, (int64_t)n + 1, s));
  DAWN_CHECK(pool_alloc((void**)&g->t_row_ptr, sizeof(int32_t) * ((size_t)n + 1), s));
  DAWN_CHECK(pool_alloc((void**)&g->t_col, sizeof(int32_t) * (size_t)(g->m > 0 ? g->m : 1) + 32, s));
  offsets_to_rowptr<<<grid, kBlock, 0, s>>>(off, g->t_row_ptr, deg, n);
  DAWN_CUDA(cudaGetLastError());
  scatter_in_edges<<<grid, kBlock, 0, s>>>(g->row_ptr, g->col, n, deg, g->t_col);
  DAWN_CUDA(cudaGetLastError());
  DAWN_CUDA(cudaFreeAsync(deg, s));
  DAWN_CUDA(cudaFreeAsync(off, s));
  return DAWN_OK;
}

// --- closeness: exact per-row reductions ----------------------------------------------

namespace {

// kind 0: hop rows (-1 unreachable); 1: int32 weights (INT32_MAX); 2: float (FLT_MAX).
template <bool kDegree>
__global__ void __launch_bounds__(kBlock) row_sums(const void* __restrict__ dist, int32_t n,
                                                   const int32_t* __restrict__ row_ptr,
                                                   const int32_t* __restrict__ sources, int kind, int row0,
                                                   long long* __restrict__ isum, double* __restrict__ fsum,
                                                   unsigned long long* __restrict__ cnt) {
  const int row = row0 + blockIdx.y;
  const int32_t s = sources[row];
  long long is = 0;
  double fs = 0.0;
  unsigned long long c = 0;
  const size_t base = (size_t)row * n;
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    bool reached;
    double fd = 0.0;
    long long id = 0;
    if (kind == 2) {
      const float d = static_cast<const float*>(dist)[base + v];
      reached = d != 3.402823466e+38f;
      fd = (double)d;
    } else {
      const int32_t d = static_cast<const int32_t*>(dist)[base + v];
      reached = kind == 0 ? d >= 0 : d != 0x7fffffff;
      id = d;
    }
    if (kDegree) {
      if (reached) is += row_ptr[v + 1] - row_ptr[v];
    } else if (reached && v != s) {
      if (kind == 2) fs += fd; else is += id;
      c++;
    }
  }
  __shared__ long long s_i[kBlock / 32];
  __shared__ double s_f[kBlock / 32];
  __shared__ unsigned long long s_c[kBlock / 32];
  for (int d = 16; d; d >>= 1) {
    is += __shfl_xor_sync(kFull, is, d);
    fs += __shfl_xor_sync(kFull, fs, d);
    c += __shfl_xor_sync(kFull, c, d);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    s_i[w] = is;
    s_f[w] = fs;
    s_c[w] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long ti = 0;
    double tf = 0;
    unsigned long long tc = 0;
    for (int i = 0; i < kBlock / 32; i++) {
      ti += s_i[i];
      tf += s_f[i];
      tc += s_c[i];
    }
    if (ti) atomicAdd(reinterpret_cast<unsigned long long*>(isum + row), (unsigned long long)ti);
    if (tf != 0.0) atomicAdd(fsum + row, tf);
    if (tc) atomicAdd(cnt + row, tc);
  }
}

}  // namespace

dawn_status row_reduce(dawn_graph* g, const void* d_dist, int32_t nsrc, const int32_t* d_sources, int kind,
                       int degree, double* d_sum, long long* d_cnt) {
  // Integer sums are exact; a float64 sum is exact while the distances are
  // integer-valued (the benchmark weights), otherwise order-dependent in the
  // last bits.  d_sum holds int64 bits for kinds 0/1 and for degree sums.
  DAWN_CUDA(cudaMemsetAsync(d_sum, 0, sizeof(double) * nsrc, g->stream));
  DAWN_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(long long) * nsrc, g->stream));
  int bx = (g->n + kBlock * 8 - 1) / (kBlock * 8);
  if (bx > 4 * g->geo.sms) bx = 4 * g->geo.sms;
  if (bx < 1) bx = 1;
  for (int32_t r0 = 0; r0 < nsrc; r0 += 65535) {
    const int rows = nsrc - r0 < 65535 ? nsrc - r0 : 65535;
    dim3 grid(bx, rows);
    if (degree)
      row_sums<true><<<grid, kBlock, 0, g->stream>>>(d_dist, g->n, g->row_ptr, d_sources, kind, r0,
                                                     reinterpret_cast<long long*>(d_sum), d_sum,
                                                     reinterpret_cast<unsigned long long*>(d_cnt));
    else
      row_sums<false><<<grid, kBlock, 0, g->stream>>>(d_dist, g->n, g->row_ptr, d_sources, kind, r0,
                                                      reinterpret_cast<long long*>(d_sum), d_sum,
                                                      reinterpret_cast<unsigned long long*>(d_cnt));
    DAWN_CUDA(cudaGetLastError());
  }
  return DAWN_OK;
}

}  // namespace dawn
