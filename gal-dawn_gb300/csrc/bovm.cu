// Single-source boolean expand (BOVM) on sm_103a.
//
// Replaces the reference's SOVM kernel and its host level loop
// (src/algorithm/gpu/bfs.cu:9-105).  The reference launches one thread per
// vertex over all n rows every level, walks each row serially and polls a
// racy flag from the host every third level.  Here a level is one of
//   push: the compacted frontier queue is expanded warp-cooperatively; rows
//         of >= 32 entries are swept by the whole warp with coalesced col
//         loads, shorter rows are packed across lanes through a warp scan;
//         a visited bitmap (L2-resident, n/8 bytes) is claimed with atomicOr;
//   pull: every still-unvisited vertex scans its in-edges and stops at the
//         first neighbour in the frontier bitmap (one warp owns 32 vertices,
//         so bitmap words are written without atomics);
// and the device picks the next level's direction (Beamer's alpha/beta rule).
// Either direction can follow the other: both emit the next frontier as a queue,
// and its bitmap is written by a level or set from the queue.  Distances are
// written once, when a vertex is claimed.
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <mutex>

#include "cluster_levels.cuh"
#include "dawn_device.cuh"
#include "selector.cuh"

namespace dawn {
namespace {

constexpr long long kAlpha = 14, kBeta = 24;


__device__ __forceinline__ uint32_t* rot(uint32_t* fbm, int i, int nwords) {
  return fbm + (size_t)(i % 3) * nwords;
}

// Fill the current source's distance row with -1 and clear the bitmaps.
__global__ void __launch_bounds__(kBlock) bfs_clear(SsCtl* __restrict__ ctl, uint32_t* __restrict__ bitmaps,
                                                    int32_t n, int32_t nwords) {
  int32_t* dist = ctl->dist_base + (size_t)ctl->src_idx * n;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += stride) dist[i] = -1;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)4 * nwords; i += stride)
    bitmaps[i] = 0;
}

// The first level of the current source (one thread): distance 0, the
// source in the visited bitmap and the level-0 frontier, its row as the
// level-1 work, the level counters.
// lq: the list of long rows in place of the segments (the persistent launch).
__device__ __forceinline__ void seed(SsCtl* ctl, int32_t s, int32_t* dist, const int32_t* __restrict__ row_ptr,
                                     int32_t* q, Seg* segs, int32_t* lq, uint32_t* vbm, int32_t n, long long m) {
  const int32_t deg = row_ptr[s + 1] - row_ptr[s];
  ctl->source = s;
  dist[s] = 0;
  vbm[s >> 5] |= 1u << (s & 31);
  // level-0 frontier bitmap (the first of the three rotating ones, right
  // after the visited words): read when the first level is a pull
  vbm[(n + 31) / 32 + (s >> 5)] |= 1u << (s & 31);
  if (deg >= kLongRow && lq) {
    lq[0] = s;
    ctl->qsize[0] = 0;
    ctl->lpack[0] = 1ull << 32;
  } else if (deg >= kLongRow) {
    const int nseg = (deg + kSeg - 1) / kSeg;
    for (int j = 0; j < nseg; j++) segs[j] = Seg{s, row_ptr[s] + j * kSeg};
    ctl->qsize[0] = 0;
    ctl->lpack[0] = (1ull << 32) | (unsigned)nseg;
  } else {
    q[0] = s;
    ctl->qsize[0] = 1;
    ctl->lpack[0] = 0;
  }
  ctl->qsize[1] = 0;
  ctl->lpack[1] = 0;
  ctl->mf[0] = (unsigned long long)deg;
  ctl->mf[1] = 0;
  ctl->mu = m - deg;
  ctl->reached = (unsigned long long)deg;
  ctl->level = 1;
  ctl->mode = ctl->force - 1 == kVarPull ? kModePull : kModePush;
  ctl->done = deg == 0;
  ctl->prev_nf = 1;
  ctl->n_push = 0;
  ctl->n_pull = 0;
}
__device__ __forceinline__ void init_source(SsCtl* __restrict__ ctl, const int32_t* __restrict__ row_ptr,
                                            int32_t* __restrict__ q, Seg* __restrict__ segs,
                                            uint32_t* __restrict__ vbm, int32_t n, long long m) {
  seed(ctl, ctl->sources[ctl->src_idx], ctl->dist_base + (size_t)ctl->src_idx * n, row_ptr, q, segs, nullptr, vbm, n, m);
}

// A distance row filled with -1 (16-byte stores over its aligned middle) and
// the bitmaps cleared.
__device__ __forceinline__ void fill_row(const Team& tm, int32_t* dist, uint32_t* bitmaps, int32_t n, size_t words) {
  const size_t tid = tm.thread(), stride = tm.threads();
  const size_t head = ((16 - (reinterpret_cast<uintptr_t>(dist) & 15)) & 15) / 4;
  const size_t h = head < (size_t)n ? head : (size_t)n;
  const size_t nvec = ((size_t)n - h) / 4;
  if (tid < h) dist[tid] = -1;
  int4* d4 = reinterpret_cast<int4*>(dist + h);
  for (size_t i = tid; i < nvec; i += stride) d4[i] = make_int4(-1, -1, -1, -1);
  for (size_t i = h + 4 * nvec + tid; i < (size_t)n; i += stride) dist[i] = -1;
  for (size_t i = tid; i < words; i += stride) bitmaps[i] = 0;
}

__global__ void bfs_init(SsCtl* __restrict__ ctl, const int32_t* __restrict__ row_ptr,
                         int32_t* __restrict__ q, Seg* __restrict__ segs, uint32_t* __restrict__ vbm, int32_t n,
                         long long m) {
  if (threadIdx.x != 0) return;
  init_source(ctl, row_ptr, q, segs, vbm, n, m);
}

// bfs_clear and bfs_init in one launch: fill_row, then the last CTA to finish (arrival count in the control block, which it
// resets) seeds the source.
__global__ void __launch_bounds__(kBlock) bfs_start(SsCtl* __restrict__ ctl, const int32_t* __restrict__ row_ptr,
                                                    int32_t* __restrict__ q, Seg* __restrict__ segs,
                                                    uint32_t* __restrict__ bitmaps, int32_t n, int32_t nwords,
                                                    long long m) {
  __shared__ int s_last;
  fill_row(Team{(int)blockIdx.x, (int)gridDim.x}, ctl->dist_base + (size_t)ctl->src_idx * n, bitmaps, n,
           4 * (size_t)nwords);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&ctl->arrive, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    ctl->arrive = 0;
    init_source(ctl, row_ptr, q, segs, bitmaps, n, m);
  }
}

// Shared memory of one level kernel: the push's row dealing, the queue
// staging both directions use, and the sums of the level's end.
template <int kWarps>
struct LevelSmem {
  int excl[kWarps][32];
  int rs[kWarps][32];
  int v[kWarps][32];
  int32_t q[kWarps][kWarpQueueBig];
  int32_t lq[kWarps][kWarpQueue];
  uint32_t n[2][kWarps];
  unsigned long long mf;
};

// Where a level's vertices go: short rows to the queue; long rows as segments,
// reserved per warp step (segs), or by their ids to a list of their own, staged
// like the queue, for the launch that cuts them only if a push follows (a pull
// of RMAT-22 finds long rows in most warp steps: 100,000 atomics on one word).
struct LongQueue {
  int32_t *buf, *out;
  unsigned long long* lpack;  // vertices << 32
  int n = 0;
  __device__ __forceinline__ void push(bool pred, int32_t v) {
    const uint32_t m = __ballot_sync(kFull, pred);
    if (m == 0) return;
    const int c = __popc(m);
    if (n + c > kWarpQueue) {
      uint32_t base = 0;
      if (lane_id() == 0) base = (uint32_t)(atomicAdd(lpack, (unsigned long long)n << 32) >> 32);
      base = __shfl_sync(kFull, base, 0);
      __syncwarp();
      for (int i = lane_id(); i < n; i += 32) out[base + i] = buf[i];
      __syncwarp();
      n = 0;
    }
    if (pred) buf[n + __popc(m & lanemask_lt())] = v;
    n += c;
  }
};
constexpr int kStepWarps = kBlock / 32;

// The end of a CTA's share of a level: what its warps still stage goes out
// with one reservation per list, and the out-edges with one atomic.
template <int kWarps>
__device__ __forceinline__ void end_level(LevelSmem<kWarps>& sm, WarpQueueBig& wq, LongQueue* lq,
                                          unsigned long long my_mf, unsigned long long* mf) {
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  if (threadIdx.x == 0) sm.mf = 0;
  if (lane == 0) {
    sm.n[0][wib] = (uint32_t)wq.n;
    sm.n[1][wib] = lq ? (uint32_t)lq->n : 0u;
  }
  __syncthreads();
  my_mf = warp_sum(my_mf);
  if (lane == 0 && my_mf) atomicAdd(&sm.mf, my_mf);
  if (wib == 0) {
#pragma unroll
    for (int l = 0; l < 2; l++) {
      const int x = lane < kWarps ? (int)sm.n[l][lane] : 0;
      const int incl = warp_incl_scan(x);
      const int tot = __shfl_sync(kFull, incl, 31);
      int base = 0;
      if (tot && lane == 0)
        base = l ? (int)(atomicAdd(lq->lpack, (unsigned long long)tot << 32) >> 32) : atomicAdd(wq.count, tot);
      base = __shfl_sync(kFull, base, 0);
      if (lane < kWarps) sm.n[l][lane] = (uint32_t)(base + incl - x);
    }
  }
  __syncthreads();
  for (int i = lane; i < wq.n; i += 32) wq.out[sm.n[0][wib] + i] = wq.buf[i];
  if (lq)
    for (int i = lane; i < lq->n; i += 32) lq->out[sm.n[1][wib] + i] = lq->buf[i];
  if (threadIdx.x == 0 && sm.mf) atomicAdd(mf, sm.mf);
}

// Top-down level: the frontier's rows are dealt to warps; unvisited
// targets are claimed in the visited bitmap and queued for the next level.
// kBits: the next level's frontier goes into its bitmap too (a pull may
// follow), the bitmap after that is cleared, and long rows go out as segments,
// not to lq.
template <bool kBits, int kWarps>
__device__ __forceinline__ void push_level(const Team& tm, const int32_t* __restrict__ row_ptr,
                                           const int32_t* __restrict__ col, SsCtl* ctl, int32_t* dist, int L, int qn,
                                           int ln, int32_t* q, Seg* segs, size_t segcap, int32_t* lq, size_t lcap,
                                           uint32_t* vbm, uint32_t* fbm, int32_t n, int32_t nwords,
                                           LevelSmem<kWarps>& sm) {
  const int pin = (L - 1) & 1, pout = L & 1;
  const int32_t* qin = q + (size_t)pin * n;
  const Seg* sin = segs + (size_t)pin * segcap;
  Seg* sout = segs + (size_t)pout * segcap;
  uint32_t* fout = rot(fbm, L, nwords);
  unsigned long long* lpack = &ctl->lpack[pout];
  const int wib = threadIdx.x >> 5;
  if (kBits) {
    uint32_t* fclr = rot(fbm, L + 1, nwords);
    for (size_t i = tm.thread(); i < (size_t)nwords; i += tm.threads()) fclr[i] = 0;
  }
  unsigned long long my_mf = 0;
  WarpQueueBig wq(sm.q[wib], q + (size_t)pout * n, &ctl->qsize[pout]);
  LongQueue wl{sm.lq[wib], kBits ? nullptr : lq + (size_t)pout * lcap, lpack};
  auto op = [&](int32_t, int k, bool valid) {
    const int32_t u = valid ? __ldg(col + k) : -1;
    const bool found = valid && claim_bit(vbm, u);
    int deg = 0, rs = 0;
    if (found) {
      rs = __ldg(row_ptr + u);
      deg = __ldg(row_ptr + u + 1) - rs;
      dist[u] = L;
      if (kBits) atomicOr(fout + (u >> 5), 1u << (u & 31));
      my_mf += (unsigned long long)deg;
    }
    if (kBits) {
      emit_routed(found, u, deg, rs, wq, sout, lpack);
    } else {
      wq.push(found && deg < kLongRow, u);
      wl.push(found && deg >= kLongRow, u);
    }
  };
  if (ln * (kSeg / 32) <= tm.warps()) {
    // few segments: 32 entries a warp, one chain of claims each instead of four
    for (int i = tm.warp(); i < ln * (kSeg / 32); i += tm.warps()) {
      const int32_t v = __ldcg(&sin[i / (kSeg / 32)].v);
      const int k0 = __ldcg(&sin[i / (kSeg / 32)].k0);
      const int k = k0 + (i % (kSeg / 32)) * 32 + lane_id();
      op(v, k, k < min(k0 + kSeg, __ldg(row_ptr + v + 1)));
    }
  } else {
    seg_expand<true>(tm.warp(), tm.warps(), row_ptr, sin, ln, op);
  }
  warp_expand<true>(tm.warp(), tm.warps(), row_ptr, qin, qn, sm.excl[wib], sm.rs[wib], sm.v[wib], op);
  end_level(sm, wq, kBits ? nullptr : &wl, my_mf, &ctl->mf[pout]);
}

__global__ void __launch_bounds__(kBlock) bfs_push(const int32_t* __restrict__ row_ptr,
                                                   const int32_t* __restrict__ col, SsCtl* __restrict__ ctl,
                                                   int32_t* __restrict__ q, Seg* __restrict__ segs, size_t segcap,
                                                   uint32_t* __restrict__ vbm, uint32_t* __restrict__ fbm,
                                                   int32_t n, int32_t nwords) {
  __shared__ LevelSmem<kStepWarps> sm;
  if (ctl->done || ctl->mode != kModePush) return;
  const int L = ctl->level, pin = (L - 1) & 1;
  push_level<true>(Team{(int)blockIdx.x, (int)gridDim.x}, row_ptr, col, ctl, ctl->dist_base + (size_t)ctl->src_idx * n,
                   L, ctl->qsize[pin], seg_count(ctl->lpack[pin]), q, segs, segcap, nullptr, 0, vbm, fbm, n, nwords, sm);
}

// Small frontiers: a single cluster of kSmallCtas CTAs runs push levels one
// after another in one launch.
//   * Each CTA appends the vertices its warps discover to its own shared-
//     memory slice (by level parity); the next level deals the rows of all
//     the cluster's slices to the cluster's warps, reading them through
//     distributed shared memory, so the frontier never goes through HBM.
//   * One cluster barrier per level (release/acquire at cluster scope)
//     orders the slices and the visited-bitmap claims; a kept vertex's
//     distance is written when the next level reads it from its slice;
//     after it every warp reads the eight slices' counters and takes the same
//     continue/stop decision.  A CTA resets its slice of the other parity
//     after the barrier: every reader of that slice (the level before) has
//     arrived at it.
//   * The loop stops after a level whose frontier is empty, holds a row of
//     >= kLongRow entries, outgrows kSmallFrontier vertices, kSmallEdges
//     out-edges or one slice (the entries past it went to the global queue
//     at once), at level n - 1, or after kSmallMaxLevels levels.  That last
//     level is handed to the per-level kernels in their format: slices ->
//     global queue and segment lists, a fresh frontier bitmap of the level
//     (the three rotating bitmaps are cleared first, since these levels did
//     not maintain them), and the counters the decide kernel reads, which
//     then does that level's bookkeeping as after a push.
// The first level reads the global queue and segments the kernels before
// wrote; its input counters are zeroed (behind one extra barrier) before a
// later level of that parity can spill into them.
struct Decision {
  int done, mode, level;  // of the next level
  int nf, qn;             // its frontier: vertices, of them with short rows
};
template <bool kStaySmall = false>
__device__ __forceinline__ Decision decide_level(SsCtl* __restrict__ ctl, int32_t n, const float* __restrict__ sel_w,
                                                 cudaGraphConditionalHandle loop, int in_graph);

__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallBlock)
    bfs_small(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col, SsCtl* ctl, int32_t* q,
              Seg* segs, size_t segcap, uint32_t* __restrict__ vbm, uint32_t* __restrict__ fbm, int32_t n,
              int32_t nwords, const float* __restrict__ sel_w, cudaGraphConditionalHandle loop, int in_graph) {
  __shared__ SmallSlice s_sl[2];
  // per parity: vertices appended (past kSmallCap they spilled), whether
  // one has a row of >= kLongRow entries, and their out-degree sum (the
  // degrees of distinct vertices sum to at most m < 2^31)
  __shared__ int32_t s_cnt[2], s_nlong[2];
  __shared__ uint32_t s_mf[2];
  if (ctl->done || ctl->mode != kModeSmall) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  constexpr int kWarps = kSmallBlock / 32;
  const int cwarp = rank * kWarps + wib;  // warp index within the cluster
  int32_t* dist = ctl->dist_base + (size_t)ctl->src_idx * n;
  if (threadIdx.x < 2) {
    s_cnt[threadIdx.x] = 0;
    s_nlong[threadIdx.x] = 0;
    s_mf[threadIdx.x] = 0;
  }
  __syncthreads();

  int L = ctl->level;
  int pre = INT_MAX, tot = 0;       // dealing of the previous level's slices (lane r < kSmallCtas: slice r)
  unsigned long long sum_mf = 0;    // out-edges of the levels finished here
  int nlev = 0, last_nf = 0, nf = 0;
  unsigned long long mf = 0;
  for (int iter = 0;; iter++) {
    const int p = L & 1;
    uint32_t my_mf = 0;
    bool my_long = false;
    auto op = [&](int k, bool valid) {
      const int32_t u = valid ? __ldg(col + k) : -1;
      bool found = false;
      int rs = 0, deg = 0;
      if (valid) {
        // the row bounds are loaded alongside the claim (most claims
        // succeed on small frontiers), so they add no round trip
        const uint32_t bit = 1u << (u & 31);
        rs = __ldg(row_ptr + u);
        const int re = __ldg(row_ptr + u + 1);
        found = !(atomicOr(vbm + (u >> 5), bit) & bit);
        deg = re - rs;
      }
      if (found) {
        my_mf += (uint32_t)deg;
        my_long |= deg >= kLongRow;
      }
      const uint32_t m = __ballot_sync(kFull, found);
      if (m == 0) return;
      const int leader = __ffs(m) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&s_cnt[p], __popc(m));
      const int slot = __shfl_sync(kFull, base, leader) + __popc(m & lanemask_lt());
      if (found && slot < kSmallCap) {
        s_sl[p].u[slot] = u;
        s_sl[p].rs[slot] = rs;
        s_sl[p].deg[slot] = deg;
      }
      const bool spill = found && slot >= kSmallCap;
      if (spill) dist[u] = L;  // kept vertices get theirs when the next level reads them
      if (__any_sync(kFull, spill))
        emit_routed(spill, u, deg, rs, q + (size_t)p * n, &ctl->qsize[p], segs + (size_t)p * segcap, &ctl->lpack[p]);
    };
    if (iter == 0) {
      // the previous level in the global format
      const int pin = p ^ 1;
      const int32_t* qin = q + (size_t)pin * n;
      const int qn = ctl->qsize[pin], ln = seg_count(ctl->lpack[pin]);
      seg_expand(row_ptr, segs + (size_t)pin * segcap, ln, [&](int32_t, int k, bool valid) { op(k, valid); });
      const int bs = batch_rows(qn);
      for (int b = cwarp * bs; b < qn; b += kSmallCtas * kWarps * bs) {
        const int i = b + lane;
        const bool ok = lane < bs && i < qn;
        int rs = 0, deg = 0;
        if (ok) {
          const int32_t v = qin[i];
          rs = row_ptr[v];
          deg = row_ptr[v + 1] - rs;
        }
        expand_rows(ok, rs, deg, op);
      }
    } else {
      // the previous level's slices, across the cluster
      const int bs = batch_rows(tot);
      for (int b = cwarp * bs; b < tot; b += kSmallCtas * kWarps * bs) {
        const int e = lane < bs ? b + lane : INT_MAX;
        int r = 0;  // last slice whose first index is <= e
#pragma unroll
        for (int step = kSmallCtas / 2; step; step >>= 1) {
          const int ex = __shfl_sync(kFull, pre, r + step);
          if (ex <= e) r += step;
        }
        const int off = e - __shfl_sync(kFull, pre, r);
        int rs = 0, deg = 0;
        if (e < tot) {
          const SmallSlice* src = cluster.map_shared_rank(&s_sl[p ^ 1], r);
          rs = src->rs[off];
          deg = src->deg[off];
          dist[src->u[off]] = L - 1;
        }
        expand_rows(e < tot, rs, deg, op);
      }
    }
    my_mf = __reduce_add_sync(kFull, my_mf);
    my_long = __any_sync(kFull, my_long);
    if (lane == 0) {
      if (my_mf) atomicAdd(&s_mf[p], my_mf);
      if (my_long) s_nlong[p] = 1;
    }
    cluster.sync();
    // this level's counters, slice by slice (lane r reads slice r)
    int cnt = 0, nl = 0;
    uint32_t mr = 0;
    if (lane < kSmallCtas) {
      cnt = *cluster.map_shared_rank(&s_cnt[p], lane);
      nl = *cluster.map_shared_rank(&s_nlong[p], lane);
      mr = *cluster.map_shared_rank(&s_mf[p], lane);
    }
    const int kept = cnt < kSmallCap ? cnt : kSmallCap;
    int incl = kept;  // inclusive scan over the kSmallCtas slice lanes
#pragma unroll
    for (int d = 1; d < kSmallCtas; d <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += t;
    }
    nf = (int)__reduce_add_sync(kFull, (uint32_t)cnt);
    mf = __reduce_add_sync(kFull, mr);
    const bool longs = __any_sync(kFull, nl != 0);
    const bool over = __any_sync(kFull, cnt > kSmallCap);
    const bool stop = nf == 0 || longs || over || nf > kSmallFrontier || (long long)mf > kSmallEdges ||
                      L + 1 >= n || iter + 1 == kSmallMaxLevels;
    if (stop) break;
    pre = lane < kSmallCtas ? incl - kept : INT_MAX;
    tot = __shfl_sync(kFull, incl, kSmallCtas - 1);
    sum_mf += mf;
    nlev++;
    last_nf = nf;
    if (threadIdx.x == 0) {
      s_cnt[p ^ 1] = 0;
      s_nlong[p ^ 1] = 0;
      s_mf[p ^ 1] = 0;
      if (iter == 0 && rank == 0) {
        ctl->qsize[p ^ 1] = 0;
        ctl->lpack[p ^ 1] = 0;
        ctl->mf[p ^ 1] = 0;
      }
    }
    if (iter == 0) cluster.sync(); else __syncthreads();
    L++;
  }

  // hand-off of level L (slice parity p) to the per-level kernels
  const int p = L & 1;
  const int mine = s_cnt[p] < kSmallCap ? s_cnt[p] : kSmallCap;
  for (int b = wib * 32; b < mine; b += kWarps * 32) {
    const int i = b + lane;
    const bool ok = i < mine;
    const int32_t u = ok ? s_sl[p].u[i] : 0;
    if (ok) dist[u] = L;
    emit_routed(ok, u, ok ? s_sl[p].deg[i] : 0, ok ? s_sl[p].rs[i] : 0, q + (size_t)p * n, &ctl->qsize[p],
                segs + (size_t)p * segcap, &ctl->lpack[p]);
  }
  const size_t tid = (size_t)rank * kSmallBlock + threadIdx.x;
  const size_t stride = (size_t)kSmallCtas * kSmallBlock;
  for (size_t i = tid; i < (size_t)3 * nwords; i += stride) fbm[i] = 0;
  if (rank == 0 && threadIdx.x == 0) {
    ctl->mf[p] = mf;
    ctl->reached += sum_mf;
    ctl->mu -= (long long)sum_mf;
    ctl->n_push += nlev;
    if (nlev) ctl->prev_nf = last_nf;
    ctl->level = L;
  }
  cluster.sync();  // also keeps every CTA resident until no one reads its shared memory
  uint32_t* fcur = rot(fbm, L, nwords);
  const int qn = __ldcg(&ctl->qsize[p]), ln = seg_count(__ldcg(&ctl->lpack[p]));
  for (size_t i = tid; i < (size_t)qn; i += stride) {
    const int32_t v = __ldcg(q + (size_t)p * n + i);
    atomicOr(fcur + (v >> 5), 1u << (v & 31));
  }
  // a long row's segments are contiguous: its first one sets the bit
  const Seg* sl = segs + (size_t)p * segcap;
  for (size_t i = tid; i < (size_t)ln; i += stride) {
    const int32_t v = __ldcg(&sl[i].v);
    if (i == 0 || __ldcg(&sl[i - 1].v) != v) atomicOr(fcur + (v >> 5), 1u << (v & 31));
  }
  // The handed-off level's bookkeeping, as after a push level.  Every
  // counter it reads was written before the cluster barrier above; it
  // writes the other parity's counters and the level fields, which no CTA
  // reads after that barrier.
  if (rank == 0 && threadIdx.x < 32) {
    __threadfence();
    decide_level(ctl, n, sel_w, loop, in_graph);
  }
}

// A frontier word written earlier in the same launch: not through the
// read-only path.
__device__ __forceinline__ bool frontier_bit(const uint32_t* bm, int32_t u) {
  uint32_t w;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(w) : "l"(bm + (u >> 5)));
  return (w >> (u & 31)) & 1u;
}

// Bottom-up level: a warp owns 32 vertices (one bitmap word); each
// unvisited one scans its in-edges until a frontier bit.
// While 32 rows are scanned, the first columns of the next 32 load and the bounds
// of the 32 after (from DRAM on RMAT-22: the pull is a chain of such loads, 21
// times per warp at its widest level).  A lane tests
// its row's first two columns, where most rows end once the frontier is large,
// then reads eight (one sector) at a time.  The last few lanes' rows are swept
// by the whole warp, so that one long row without a hit does not hold it.
constexpr int kSweepLanes = 4;
template <bool kSegs, int kWarps>
__device__ __forceinline__ void pull_level(const Team& tm, const int32_t* __restrict__ row_ptr,
                                           const int32_t* __restrict__ t_row_ptr, const int32_t* __restrict__ t_col,
                                           SsCtl* ctl, int32_t* dist, int L, int32_t* q, Seg* segs, size_t segcap,
                                           int32_t* lq, size_t lcap, uint32_t* vbm, uint32_t* fbm, int32_t n, int32_t nwords,
                                           LevelSmem<kWarps>& sm) {
  const int pout = L & 1;
  Seg* sout = segs + (size_t)pout * segcap;
  unsigned long long* lpack = &ctl->lpack[pout];
  const uint32_t* fin = rot(fbm, L - 1, nwords);
  uint32_t* fout = rot(fbm, L, nwords);
  uint32_t* fclr = rot(fbm, L + 1, nwords);
  const int lane = lane_id();
  const bool wide = (reinterpret_cast<uintptr_t>(t_col) & 31) == 0;

  for (size_t i = tm.thread(); i < (size_t)nwords; i += tm.threads()) fclr[i] = 0;

  unsigned long long my_mf = 0;
  WarpQueueBig wq(sm.q[threadIdx.x >> 5], q + (size_t)pout * n, &ctl->qsize[pout]);
  LongQueue wl{sm.lq[threadIdx.x >> 5], kSegs ? nullptr : lq + (size_t)pout * lcap, lpack};
  const int stride = tm.warps();
  uint32_t vis_a = ~0u, vis_b = ~0u;
  int k_a = 0, e_a = 0, k_b = 0, e_b = 0;  // rows to scan: empty where the vertex is visited
  int32_t c0_b = -1, c1_b = -1;
  auto load_bounds = [&](int w) {
    vis_a = ~0u;
    k_a = e_a = 0;
    if (w < nwords) {
      vis_a = __ldcg(vbm + w);
      const int32_t u = w * 32 + lane;
      if (u < n) {
        k_a = __ldg(t_row_ptr + u);
        e_a = __ldg(t_row_ptr + u + 1);
      }
    }
  };
  auto load_columns = [&]() {
    vis_b = vis_a;
    k_b = k_a;
    e_b = (vis_a >> lane) & 1u ? k_a : e_a;
    c0_b = k_b < e_b ? __ldg(t_col + k_b) : -1;
    c1_b = k_b + 1 < e_b ? __ldg(t_col + k_b + 1) : -1;
  };
  load_bounds(tm.warp());
  load_columns();
  load_bounds(tm.warp() + stride);
  for (int w = tm.warp(); w < nwords; w += stride) {
    const uint32_t vis = vis_b;
    const int k0 = k_b, e = e_b;
    const int32_t c0 = c0_b, c1 = c1_b;
    load_columns();
    load_bounds(w + 2 * stride);
    if (__all_sync(kFull, k0 == e)) continue;
    const int32_t u = w * 32 + lane;
    int k = k0;
    bool found = false;
    {
      const bool h0 = c0 >= 0 && frontier_bit(fin, c0), h1 = c1 >= 0 && frontier_bit(fin, c1);
      found = h0 || h1;
      k = found ? e : k + 2;
    }
    uint32_t left = __ballot_sync(kFull, k < e);
    while (__popc(left) > kSweepLanes) {
      if (k < e) {
        const int b = k & ~7;
        int32_t c[8];
        if (wide) {
          asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
              : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
              : "l"(t_col + b));
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) c[i] = b + i >= k && b + i < e ? __ldg(t_col + b + i) : 0;
        }
        bool hit[8];
#pragma unroll
        for (int i = 0; i < 8; i++) hit[i] = b + i >= k && b + i < e && frontier_bit(fin, c[i]);
#pragma unroll
        for (int i = 0; i < 8; i++) found |= hit[i];
        k = found ? e : b + 8;
      }
      left = __ballot_sync(kFull, k < e);
    }
    while (left) {
      const int l = __ffs(left) - 1;
      left &= left - 1;
      const int e1 = __shfl_sync(kFull, e, l);
      bool any = false;
      for (int k0 = __shfl_sync(kFull, k, l); k0 < e1 && !any; k0 += 128) {
        int32_t c[4];
#pragma unroll
        for (int i = 0; i < 4; i++) c[i] = k0 + 32 * i + lane < e1 ? __ldg(t_col + k0 + 32 * i + lane) : -1;
        bool hit[4];
#pragma unroll
        for (int i = 0; i < 4; i++) hit[i] = c[i] >= 0 && frontier_bit(fin, c[i]);
        any = __any_sync(kFull, hit[0] || hit[1] || hit[2] || hit[3]);
      }
      if (lane == l) found = any;
    }
    const uint32_t fm = __ballot_sync(kFull, found);
    if (fm) {
      if (lane == 0) {
        vbm[w] = vis | fm;
        fout[w] = fm;
      }
      int deg = 0, rs = 0;
      if (found) {
        rs = row_ptr == t_row_ptr ? k0 : __ldg(row_ptr + u);
        deg = (row_ptr == t_row_ptr ? e : __ldg(row_ptr + u + 1)) - rs;
        dist[u] = L;
        my_mf += (unsigned long long)deg;
      }
      if (kSegs) {
        emit_routed(found, u, deg, rs, wq, sout, lpack);
      } else {
        wq.push(found && deg < kLongRow, u);
        wl.push(found && deg >= kLongRow, u);
      }
    }
  }
  end_level(sm, wq, kSegs ? nullptr : &wl, my_mf, &ctl->mf[pout]);
}

// One warp (all 32 lanes).  Ends the loop when the frontier is empty,
// otherwise picks the next level's direction: the forced variant if one is
// set, else the learned selector if weights are loaded (direction-
// optimising calls only), else Beamer's alpha/beta rule.  The control block
// is read through volatile loads: when this runs at the end of the level
// kernel itself, counters other CTAs just raised may sit stale in this
// SM's L1.
// kStaySmall: small levels follow one another without a new decision while
// the frontier stays small, as inside bfs_small.
template <bool kStaySmall>
__device__ __forceinline__ Decision decide_level(SsCtl* __restrict__ ctl, int32_t n, const float* __restrict__ sel_w,
                                                 cudaGraphConditionalHandle loop, int in_graph) {
  const int lane = lane_id();
  if (sel_w) sel_prefetch(sel_w);
  const volatile SsCtl* vc = ctl;
  // every lane reads the control block before lane 0 changes it
  const int done = vc->done;
  const int L = vc->level, pout = L & 1;
  const int qn = vc->qsize[pout];
  const unsigned long long lp = vc->lpack[pout];
  const int nf = qn + long_vertices(lp);
  const unsigned long long mf = vc->mf[pout];
  const long long mu = vc->mu - (long long)mf;
  const int cur_mode = vc->mode, prev_nf = vc->prev_nf, policy = vc->policy, force = vc->force;
  const bool sel = vc->use_sel && sel_w;
  const long long m = vc->m;
  const int small = vc->small;
  const int nlong = long_vertices(lp);
  const float margin = vc->sel_margin;
  __syncwarp();
  if (done) {
    if (lane == 0 && in_graph) cudaGraphSetConditional(loop, 0);
    return {1, 0, L, 0, 0};
  }
  if (lane == 0) {
    ctl->reached += mf;
    ctl->mu = mu;
    if (cur_mode == kModePull) ctl->n_pull++; else ctl->n_push++;
  }
  if (nf == 0 || L >= n) {
    if (lane == 0) {
      ctl->done = 1;
      if (in_graph) cudaGraphSetConditional(loop, 0);
    }
    return {1, 0, L, 0, 0};
  }
  int mode = cur_mode == kModePull ? kModePull : kModePush;  // cluster levels are push levels
  if (policy == DAWN_VARIANT_DO) {
    if (mode == kModePush) {
      if ((long long)mf * kAlpha > mu && nf > prev_nf) mode = kModePull;
    } else {
      if ((long long)nf * kBeta < (long long)n && nf < prev_nf) mode = kModePush;
    }
  }
  if (force) {
    mode = force - 1 == kVarPull ? kModePull : kModePush;
  } else if (policy == DAWN_VARIANT_DO && sel) {
    float x[kSelIn];
    sel_features(x, (float)n, (float)m, (float)nf, (float)mf, (float)mu, (float)(L + 1), (float)prev_nf, 1.0f);
    const int h = mode == kModePull ? kVarPull : kVarPush;
    mode = sel_pick(sel_w, x, (1u << kVarPush) | (1u << kVarPull), h, margin) == kVarPull ? kModePull
                                                                                         : kModePush;
  }
  // small levels start from frontiers without long rows: a long row's
  // neighbourhood tends to hold more, which end the cluster levels at once
  const bool fits = small && !force && policy == DAWN_VARIANT_DO && nf <= kSmallFrontier &&
                    (long long)mf <= kSmallEdges && nlong == 0;
  if (fits && (mode == kModePush || (kStaySmall && cur_mode == kModeSmall))) mode = kModeSmall;
  if (lane == 0) {
    ctl->qsize[pout ^ 1] = 0;
    ctl->lpack[pout ^ 1] = 0;
    ctl->mf[pout ^ 1] = 0;
    ctl->prev_nf = nf;
    ctl->mode = mode;
    ctl->level = L + 1;
  }
  return {0, mode, L + 1, nf, qn};
}

__global__ void bfs_decide(SsCtl* __restrict__ ctl, int32_t n, const float* __restrict__ sel_w,
                           cudaGraphConditionalHandle loop, int in_graph) {
  decide_level(ctl, n, sel_w, loop, in_graph);
}

// One launch per push or pull level: the level's work, then its end-of-
// level bookkeeping by the last CTA to finish (an arrival count in the
// control block, reset by that CTA), so a level costs one kernel instead of
// a work kernel and a decide kernel.  Returns at once at cluster levels.
__global__ void __launch_bounds__(kBlock, 5) bfs_step(const int32_t* __restrict__ row_ptr,
                                                   const int32_t* __restrict__ col,
                                                   const int32_t* __restrict__ t_row_ptr,
                                                   const int32_t* __restrict__ t_col, SsCtl* __restrict__ ctl,
                                                   int32_t* __restrict__ q, Seg* __restrict__ segs, size_t segcap,
                                                   uint32_t* __restrict__ vbm, uint32_t* __restrict__ fbm,
                                                   int32_t n, int32_t nwords, const float* __restrict__ sel_w,
                                                   cudaGraphConditionalHandle loop, int in_graph) {
  __shared__ LevelSmem<kStepWarps> sm;
  __shared__ int s_last;
  if (ctl->done) {
    // a traversal that ended before its first level (an isolated source)
    // or at a cluster level: the loop still has to be told
    if (in_graph && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(loop, 0);
    return;
  }
  const int mode = ctl->mode;
  const Team tm{(int)blockIdx.x, (int)gridDim.x};
  int32_t* const dist = ctl->dist_base + (size_t)ctl->src_idx * n;
  const int L = ctl->level, pin = (L - 1) & 1;
  if (mode == kModePush)
    push_level<true>(tm, row_ptr, col, ctl, dist, L, ctl->qsize[pin], seg_count(ctl->lpack[pin]), q, segs, segcap,
                     nullptr, 0, vbm, fbm, n, nwords, sm);
  else if (mode == kModePull)
    pull_level<true>(tm, row_ptr, t_row_ptr, t_col, ctl, dist, L, q, segs, segcap, nullptr, 0, vbm, fbm, n, nwords, sm);
  else
    return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&ctl->arrive, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x < 32) {
    __threadfence();
    if (threadIdx.x == 0) ctl->arrive = 0;
    decide_level(ctl, n, sel_w, loop, in_graph);
  }
}

// --- the persistent launch ----------------------------------------------------------

// One source in one cooperative launch: fill, levels, counters.  In a
// conditional graph a level is two kernels of which one returns at once, about
// 10 us before any work; here it ends with one arrival per CTA and a decision
// in the last one, which names as many CTAs for the next step as it has work
// for (about 5 us a step, 1.1 us a level in CTA 0).  A small frontier without long rows is CTA 0's, level after level, with
// the lists in shared memory: a chain of two round trips to L2 (targets; their
// claims together with their row bounds) and a barrier, against cluster
// barriers and remote shared memory in bfs_small.  Push levels leave the
// frontier bitmaps alone: a pull that follows one sets them from the queue.
// Per call, level kernels -> this:
//   RMAT-12 (edge factor 8), distances to the host   134 ->   91 us
//   RMAT-20                                          141 ->   86
//   RMAT-22                                          261 ->  200
//   grid 300 x 300                                  1580 ->  818
//   grid 1000 x 1049                                6511 -> 4297
constexpr int kBfEntries = 4096;             // vertices and entries per CTA of a small graph
// Frontiers that go to CTA 0 and that stay there.  One SM makes about one access
// to L1 or L2 a clock: a row of four entries costs it a dozen (8 us for 1,000
// rows), with a record and the bitmap in shared memory two.
constexpr int kSoloStart = 192, kSoloKeep = 256, kSoloCap = 1024;  // the last: vertices that its lists hold
constexpr uint32_t kSoloEdges = 2048;
constexpr int kSoloRow = 8;                  // longest row that one lane walks there
constexpr int kMeshStart = 2048, kMeshKeep = 2560, kMeshCap = 3072;
constexpr int kRecMax = 32;                  // longest row with a record
constexpr int32_t kMeshMax = 1600000;        // vertices whose bitmap fits beside the lists
constexpr int32_t kMeshWide = 32768;

enum : int32_t { kBfStart = 0, kBfWipe, kBfBits, kBfCut, kBfPush, kBfPull, kBfSolo };

// What a wait that gives up adds to the arrivals: more than a launch's CTAs, so that
// no later arrival counts as a step's last.
constexpr uint32_t kBfBroken = 1u << 30;
struct BfsSync {
  struct __align__(128) {
    unsigned long long word[4];
  } step;  // BfsStep, tagged with the generation in the top 16 bits of each word
  struct __align__(128) {
    uint32_t n;
  } arrive;
};
struct BfsStep {
  int32_t ctas, phase, dirty;  // dirty: a pull has written frontier bitmaps
  int32_t L, qn, ln;           // the level, its queued vertices and long rows (push: their segments)
  uint32_t arrived;            // arrivals before the phase
};

struct BfsArgs {
  const int32_t *row_ptr, *col, *t_row_ptr, *t_col;
  SsCtl* ctl;
  BfsSync* sync;
  int32_t* dist;
  int32_t* q;
  Seg* segs;
  int32_t* lq;             // long rows, by level parity
  size_t segcap, lcap;
  uint32_t *vbm, *fbm;
  long long m;
  const float* sel_w;
  const int32_t* rec;  // n rows of rec_len neighbours, -1 behind the last (NULL: none)
  int32_t rec_len;
  int32_t n, nwords, source, first;  // first: of the call's sources
  int32_t policy, use_sel, force, small;
  float sel_margin;
  uint32_t polls;      // of one wait
  int32_t* err;        // pinned host word
};

struct SoloList {
  int32_t u[kSoloCap], rs[kSoloCap], deg[kSoloCap];
};
struct MeshLists {
  int32_t u[2][kMeshCap];
  uint32_t visited[4];  // and the rest of the n bits
};
template <int kWarps>
struct BfsSmem {
  BfsStep st;
  int32_t cnt[3];
  uint32_t mf[3], deg[3];  // solo: out-edges and longest row of the list
  union {
    LevelSmem<kWarps> lv;
    SoloList solo[2];
    MeshLists mesh;
  };
};

// The frontier's bits, from its lists.
__device__ __forceinline__ void set_bits(const Team& tm, const BfsArgs& a, const BfsStep& st) {
  const int pin = (st.L - 1) & 1;
  uint32_t* const f = rot(a.fbm, st.L - 1, a.nwords);
  const int32_t *const qin = a.q + (size_t)pin * a.n, *const lin = a.lq + (size_t)pin * a.lcap;
  for (size_t i = tm.thread(); i < (size_t)st.qn + st.ln; i += tm.threads()) {
    const int32_t v = __ldcg(i < (size_t)st.qn ? qin + i : lin + (i - st.qn));
    atomicOr(f + (v >> 5), 1u << (v & 31));
  }
}

// The segments of the frontier's long rows.
__device__ __forceinline__ void cut_rows(const Team& tm, const BfsArgs& a, const BfsStep& st) {
  const int pin = (st.L - 1) & 1, lane = lane_id();
  const int32_t* const lin = a.lq + (size_t)pin * a.lcap;
  for (int b = tm.warp() * 32; b < st.ln; b += tm.warps() * 32) {
    const bool ok = b + lane < st.ln;
    const int32_t v = ok ? __ldcg(lin + b + lane) : 0;
    const int rs = ok ? __ldg(a.row_ptr + v) : 0;
    const int nseg = ok ? (__ldg(a.row_ptr + v + 1) - rs + kSeg - 1) / kSeg : 0;
    const int incl = warp_incl_scan(nseg);
    unsigned long long base = 0;
    if (lane == 31) base = atomicAdd(&a.ctl->lpack[pin], (unsigned long long)incl);
    const uint32_t first = (uint32_t)__shfl_sync(kFull, base, 31) + incl - nseg;
    write_segments(__ballot_sync(kFull, ok), v, rs, nseg, first, a.segs + (size_t)pin * a.segcap);
  }
}

// A vertex of level L from CTA 0 into its list.
__device__ __forceinline__ void queue_vertex(const BfsArgs& a, int L, bool is, int32_t v, int deg) {
  SsCtl* const ctl = a.ctl;
  const int p = L & 1;
  const int at = warp_append(is && deg < kLongRow, &ctl->qsize[p]);
  if (is && deg < kLongRow) a.q[(size_t)p * a.n + at] = v;
  if (is && deg >= kLongRow)
    a.lq[(size_t)p * a.lcap + (uint32_t)(atomicAdd(&ctl->lpack[p], 1ull << 32) >> 32)] = v;
}

// Small levels, by CTA 0 alone.  The last one is left in the queue, with its
// counters, for the decision at the end of the phase.
template <int kWarps>
__device__ __forceinline__ void solo_levels(const BfsArgs& a, const BfsStep& st, BfsSmem<kWarps>& sm) {
  constexpr int kThreads = 32 * kWarps;
  SsCtl* const ctl = a.ctl;
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  int L = st.L;
  const int last = min(a.n, L + kSoloSteps);
  {
    const int32_t* qin = a.q + (size_t)((L - 1) & 1) * a.n;
    if (threadIdx.x < 3) sm.cnt[threadIdx.x] = sm.mf[threadIdx.x] = sm.deg[threadIdx.x] = 0;
    __syncthreads();
    uint32_t longest = 0;
    for (int i = threadIdx.x; i < st.qn; i += kThreads) {
      const int32_t u = __ldcg(qin + i);
      const int rs = __ldg(a.row_ptr + u), deg = __ldg(a.row_ptr + u + 1) - rs;
      sm.solo[0].rs[i] = rs;
      sm.solo[0].deg[i] = deg;
      longest = max(longest, (uint32_t)deg);
    }
    longest = __reduce_max_sync(kFull, longest);
    if (lane == 0) atomicMax(&sm.deg[0], longest);
    if (threadIdx.x == 0) {
      sm.cnt[0] = st.qn;
      for (int p = 0; p < 2; p++) {
        ctl->qsize[p] = 0;
        ctl->lpack[p] = 0;
        ctl->mf[p] = 0;
      }
    }
    __syncthreads();
  }
  unsigned long long sum_mf = 0;
  int it = 0, last_nf = 0;
  for (;; it++, L++) {
    const int cnt = sm.cnt[it % 3], o = (it + 1) % 3;
    const SoloList& in = sm.solo[it & 1];
    SoloList& nx = sm.solo[(it & 1) ^ 1];
    if (threadIdx.x < 1) sm.cnt[(it + 2) % 3] = sm.mf[(it + 2) % 3] = sm.deg[(it + 2) % 3] = 0;
    uint32_t my_mf = 0, longest = 0;
    // claims the targets of up to four entries per lane
    auto claim = [&](const int (&k)[4], const bool (&ok)[4]) {
      int32_t u[4];
      int rs[4], re[4];
      uint32_t old[4];
#pragma unroll
      for (int i = 0; i < 4; i++) u[i] = ok[i] ? __ldg(a.col + k[i]) : 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        rs[i] = re[i] = 0;
        old[i] = ~0u;
        if (ok[i]) {
          old[i] = atomicOr(a.vbm + (u[i] >> 5), 1u << (u[i] & 31));
          rs[i] = __ldg(a.row_ptr + u[i]);
          re[i] = __ldg(a.row_ptr + u[i] + 1);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool found = !((old[i] >> (u[i] & 31)) & 1u);
        const uint32_t m = __ballot_sync(kFull, found);
        if (m == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(&sm.cnt[o], __popc(m));
        const int slot = __shfl_sync(kFull, base, 0) + __popc(m & lanemask_lt());
        const int deg = re[i] - rs[i];
        if (found) {
          a.dist[u[i]] = L;
          my_mf += (uint32_t)deg;
          longest = max(longest, (uint32_t)deg);
          if (slot < kSoloCap) {
            nx.u[slot] = u[i];
            nx.rs[slot] = rs[i];
            nx.deg[slot] = deg;
          }
        }
        const bool spill = found && slot >= kSoloCap;
        if (__any_sync(kFull, spill))
          queue_vertex(a, L, spill, u[i], deg);
      }
    };
    if (sm.deg[it % 3] <= (uint32_t)kSoloRow) {  // a row per lane
      int per = 32;
      while (per > 1 && (per >> 1) * kWarps >= cnt) per >>= 1;
      for (int b = wib * per; b < cnt; b += kWarps * per) {
        const bool in_row = lane < per && b + lane < cnt;
        const int rs = in_row ? in.rs[b + lane] : 0, deg = in_row ? in.deg[b + lane] : 0;
#pragma unroll
        for (int j = 0; j < kSoloRow; j += 4) {
          if (!__any_sync(kFull, deg > j)) break;
          const int k[4] = {rs + j, rs + j + 1, rs + j + 2, rs + j + 3};
          const bool ok[4] = {deg > j, deg > j + 1, deg > j + 2, deg > j + 3};
          claim(k, ok);
        }
      }
    } else {
      int per = 32;
      while (per > 1 && (per >> 1) * kWarps >= cnt) per >>= 1;
      for (int b = wib * per; b < cnt; b += kWarps * per) {
        const bool in_row = lane < per && b + lane < cnt;
        const int rs = in_row ? in.rs[b + lane] : 0, deg = in_row ? in.deg[b + lane] : 0;
        const int incl = warp_incl_scan(deg), excl = incl - deg;
        const int total = __shfl_sync(kFull, incl, 31);
        for (int e0 = 0; e0 < total; e0 += 128) {
          int k[4];
          bool ok[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int e = e0 + 32 * j + lane;
            int lo = 0;  // last lane whose offset is <= e
#pragma unroll
            for (int step = 16; step; step >>= 1)
              if (__shfl_sync(kFull, excl, lo + step) <= e) lo += step;
            k[j] = __shfl_sync(kFull, rs, lo) + (e - __shfl_sync(kFull, excl, lo));
            ok[j] = e < total;
          }
          claim(k, ok);
        }
      }
    }
    my_mf = __reduce_add_sync(kFull, my_mf);
    longest = __reduce_max_sync(kFull, longest);
    if (lane == 0) {
      if (my_mf) atomicAdd(&sm.mf[o], my_mf);
      if (longest) atomicMax(&sm.deg[o], longest);
    }
    __syncthreads();
    const int nf = sm.cnt[o];
    if (nf == 0 || nf > kSoloKeep || sm.mf[o] > kSoloEdges || sm.deg[o] >= (uint32_t)kLongRow || L + 1 >= last) break;
    sum_mf += sm.mf[o];
    last_nf = nf;
  }
  const SoloList& out = sm.solo[(it & 1) ^ 1];
  const int o = (it + 1) % 3, p = L & 1, kept = min(sm.cnt[o], kSoloCap);
  for (int b = wib * 32; b < kept; b += kThreads) {
    const int i = b + lane;
    const bool ok = i < kept;
    queue_vertex(a, L, ok, ok ? out.u[i] : 0, ok ? out.deg[i] : 0);
  }
  if (threadIdx.x == 0) {
    ctl->mf[p] = sm.mf[o];
    ctl->reached += sum_mf;
    ctl->mu -= (long long)sum_mf;
    ctl->n_push += it;
    if (it) ctl->prev_nf = last_nf;
    ctl->level = L;
  }
}

// Likewise, its out-edges read and counted.
__device__ __forceinline__ void mesh_queue(const BfsArgs& a, int L, bool is, int32_t v) {
  uint32_t deg = is ? (uint32_t)(__ldg(a.row_ptr + v + 1) - __ldg(a.row_ptr + v)) : 0u;
  queue_vertex(a, L, is, v, (int)deg);
  deg = __reduce_add_sync(kFull, deg);
  if (lane_id() == 0 && deg) atomicAdd(&a.ctl->mf[L & 1], (unsigned long long)deg);
}

// Small levels of a graph with records (rows of at most kRecMax entries), by CTA
// 0 alone, with the visited bitmap in its shared memory: a level is one round
// trip, for the rows' records, and a store per vertex that no one waits for.
template <int kWarps>
__device__ __forceinline__ void mesh_levels(const BfsArgs& a, const BfsStep& st, BfsSmem<kWarps>& sm) {
  constexpr int kThreads = 32 * kWarps;
  SsCtl* const ctl = a.ctl;
  uint32_t* const vis = sm.mesh.visited;
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  int L = st.L;
  const int32_t* qin = a.q + (size_t)((L - 1) & 1) * a.n;
  for (int i = threadIdx.x; i < a.nwords; i += kThreads) vis[i] = __ldcg(a.vbm + i);
  for (int i = threadIdx.x; i < st.qn; i += kThreads) sm.mesh.u[0][i] = __ldcg(qin + i);
  if (threadIdx.x == 0) {
    sm.cnt[0] = st.qn;
    sm.cnt[1] = sm.cnt[2] = 0;
    for (int p = 0; p < 2; p++) {
      ctl->qsize[p] = 0;
      ctl->lpack[p] = 0;
      ctl->mf[p] = 0;
    }
  }
  __syncthreads();
  uint32_t my_deg = 0;  // entries of the rows walked, but for the first level's
  int it = 0, last_nf = 0;
  for (;; it++, L++) {
    const int cnt = sm.cnt[it % 3], o = (it + 1) % 3;
    const int32_t* const in = sm.mesh.u[it & 1];
    int32_t* const out = sm.mesh.u[(it & 1) ^ 1];
    if (threadIdx.x == 0) sm.cnt[(it + 2) % 3] = 0;
    int per = 32;
    while (per > 1 && (per >> 1) * kWarps >= cnt) per >>= 1;
    for (int b = wib * per; b < cnt; b += kWarps * per) {
      const bool in_row = lane < per && b + lane < cnt;
      const int32_t* rec = a.rec + (size_t)(in_row ? in[b + lane] : 0) * a.rec_len;
      bool go = in_row;
      for (int j = 0; __any_sync(kFull, go); j += 8) {
        int32_t c[8];
#pragma unroll
        for (int i = 0; i < 8; i++) c[i] = -1;
        if (go)
          asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
              : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
              : "l"(rec + j));
        go = c[7] >= 0 && j + 8 < a.rec_len;
        unsigned is_new = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
          if (c[i] >= 0) {
            my_deg += it > 0;
            is_new |= (~vis[c[i] >> 5] >> (c[i] & 31) & 1u) << i;
          }
#pragma unroll
        for (int i = 0; i < 8; i++)
          if ((is_new >> i) & 1u) {
            const uint32_t bit = 1u << (c[i] & 31);
            if (atomicOr(vis + (c[i] >> 5), bit) & bit) is_new &= ~(1u << i);
          }
        const int mine = __popc(is_new), incl = warp_incl_scan(mine);
        const int tot = __shfl_sync(kFull, incl, 31);
        if (tot == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(&sm.cnt[o], tot);
        base = __shfl_sync(kFull, base, 0);
        int slot = base + incl - mine;
#pragma unroll
        for (int i = 0; i < 8; i++)
          if ((is_new >> i) & 1u) {
            a.dist[c[i]] = L;
            if (slot < kMeshCap) {
              out[slot] = c[i];
              is_new &= ~(1u << i);
            }
            slot++;
          }
        if (base + tot > kMeshCap) {
#pragma unroll
          for (int i = 0; i < 8; i++) mesh_queue(a, L, (is_new >> i) & 1u, c[i]);
        }
      }
    }
    __syncthreads();
    const int nf = sm.cnt[o];
    if (nf == 0 || nf > kMeshKeep || L + 1 >= a.n) break;  // (kMeshMax levels at most: a few seconds)
    last_nf = nf;
  }
  for (int i = threadIdx.x; i < a.nwords; i += kThreads) a.vbm[i] = vis[i];
  const int32_t* const out = sm.mesh.u[(it & 1) ^ 1];
  const int kept = min(sm.cnt[(it + 1) % 3], kMeshCap);
  for (int b = wib * 32; b < kept; b += kThreads) mesh_queue(a, L, b + lane < kept, b + lane < kept ? out[b + lane] : 0);
  my_deg = __reduce_add_sync(kFull, my_deg);
  if (lane == 0 && my_deg) {
    atomicAdd(&ctl->reached, (unsigned long long)my_deg);
    atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->mu), -(unsigned long long)my_deg);
  }
  if (threadIdx.x == 0) {
    ctl->n_push += it;
    if (it) ctl->prev_nf = last_nf;
    ctl->level = L;
  }
}

// CTAs for `work` warp tasks.
template <int kWarps>
__device__ __forceinline__ int bf_ctas(int work) {
  const int c = (work + kWarps - 1) / kWarps;
  return c < 1 ? 1 : min(c, (int)gridDim.x);
}

// One warp of the last CTA to finish phase st: the next one.  Returns false
// when the traversal is done.  Not inlined: its registers would be the
// levels' spills.
template <int kWarps>
__device__ __noinline__ bool next_phase(const BfsArgs& a, BfsStep& step) {
  BfsStep st = step;
  SsCtl* const ctl = a.ctl;
  int phase = kBfPush;
  if (st.phase == kBfWipe) {
    phase = kBfBits;
  } else if (st.phase == kBfBits) {
    phase = kBfPull;
  } else if (st.phase == kBfCut) {
    st.ln = seg_count(static_cast<const volatile SsCtl*>(ctl)->lpack[(st.L - 1) & 1]);
  } else if (st.phase == kBfStart) {
    int done = 0, mode = 0, qn = 0, ln = 0;
    if (lane_id() == 0) {
      SsCtl c = {};
      c.policy = a.policy;
      c.use_sel = a.use_sel;
      c.sel_margin = a.sel_margin;
      c.force = a.force;
      c.small = a.small;
      c.m = a.m;
      c.source = a.source;
      if (!a.first) {
        const volatile SsCtl* vc = ctl;
        c.total_reached = vc->total_reached;
        c.total_levels = vc->total_levels;
        c.total_push = vc->total_push;
        c.total_pull = vc->total_pull;
      }
      *ctl = c;
      seed(ctl, a.source, a.dist, a.row_ptr, a.q, a.segs, a.lq, a.vbm, a.n, a.m);
      done = ctl->done;
      mode = ctl->mode;
      qn = ctl->qsize[0];
      ln = long_vertices(ctl->lpack[0]);
    }
    st.L = 1;
    st.qn = __shfl_sync(kFull, qn, 0);
    st.ln = __shfl_sync(kFull, ln, 0);
    mode = __shfl_sync(kFull, mode, 0);
    if (__shfl_sync(kFull, done, 0)) return false;
    phase = mode == kModePull ? kBfPull : st.ln ? kBfCut : kBfPush;
  } else {
    const Decision d = decide_level<true>(ctl, a.n, a.sel_w, 0, 0);
    if (d.done) return false;
    st.L = d.level;
    st.qn = d.qn;
    st.ln = d.nf - d.qn;
    if (st.ln) phase = kBfCut;
    if (d.mode == kModePull)
      phase = st.phase == kBfPull ? kBfPull : (st.dirty ? kBfWipe : kBfBits);
    else if (d.mode == kModeSmall && d.nf <= (a.rec ? kMeshStart : kSoloStart))
      phase = kBfSolo;
  }
  if (phase == kBfPull) st.dirty = 1;
  if (phase == kBfWipe) st.dirty = 0;
  st.ctas = phase == kBfSolo ? 1
            : phase == kBfPush ? bf_ctas<kWarps>(st.qn / 4 + st.ln * (kSeg / 32) + 1)
            : phase == kBfBits ? bf_ctas<kWarps>((st.qn + st.ln) / 32 + 1)
            : phase == kBfCut  ? bf_ctas<kWarps>(st.ln / 32 + 1)
                               : (int)gridDim.x;
  st.phase = phase;
  step = st;
  return true;
}

// kMesh: with records, 1,024 threads and one CTA per SM (the bitmap takes its
// shared memory); else two CTAs of 640 threads at 48 registers.
template <bool kMesh>
__global__ void __launch_bounds__(kMesh ? 1024 : 640, kMesh ? 1 : 2) bfs_traverse(const __grid_constant__ BfsArgs a) {
  constexpr int kWarps = kMesh ? 32 : 20;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t s_polls;  // of one wait
  auto& sm = *reinterpret_cast<BfsSmem<kWarps>*>(smem);
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  // no phase can open before every CTA has arrived, so all read the same
  uint32_t gen = (uint32_t)(*static_cast<const volatile unsigned long long*>(&a.sync->step.word[0]) >> 48);
  const BfsStep& st = sm.st;
  if (threadIdx.x == 0) {
    sm.st = BfsStep{};
    sm.st.phase = kBfStart;
    sm.st.ctas = (int)gridDim.x;
    sm.st.arrived = (uint32_t)*static_cast<const volatile unsigned long long*>(&a.sync->step.word[3]);
    // after a launch that gave up, none of the next ones' steps completes (its
    // arrivals are missing): they wait once and end
    const uint32_t now = *static_cast<const volatile uint32_t*>(&a.sync->arrive.n);
    s_polls = now - sm.st.arrived >= kBfBroken ? 1 : a.polls;
  }
  __syncthreads();
  for (;;) {
    const Team tm{(int)blockIdx.x, st.ctas};
    switch (st.phase) {
      case kBfStart: fill_row(tm, a.dist, a.vbm, a.n, 4 * (size_t)a.nwords); break;
      case kBfWipe:
        for (size_t i = tm.thread(); i < (size_t)3 * a.nwords; i += tm.threads()) a.fbm[i] = 0;
        break;
      case kBfBits: set_bits(tm, a, st); break;
      case kBfCut: cut_rows(tm, a, st); break;
      case kBfPush:
        push_level<false>(tm, a.row_ptr, a.col, a.ctl, a.dist, st.L, st.qn, st.ln, a.q, a.segs, a.segcap, a.lq, a.lcap,
                          a.vbm, a.fbm, a.n, a.nwords, sm.lv);
        break;
      case kBfPull:
        pull_level<false>(tm, a.row_ptr, a.t_row_ptr, a.t_col, a.ctl, a.dist, st.L, a.q, a.segs, a.segcap, a.lq, a.lcap,
                          a.vbm, a.fbm, a.n, a.nwords, sm.lv);
        break;
      default:
        if (kMesh)
          mesh_levels(a, st, sm);
        else
          solo_levels(a, st, sm);
    }
    __syncthreads();
    if (wib == 0) {
      int last = 0;
      if (lane == 0) {
        __threadfence();
        last = atomicAdd(&a.sync->arrive.n, 1u) + 1 == st.arrived + (uint32_t)st.ctas;
      }
      if (__shfl_sync(kFull, last, 0)) {
        __threadfence();
        BfsStep nx = st;
        nx.arrived = st.arrived + (uint32_t)st.ctas;
        const bool more = next_phase<kWarps>(a, nx);
        if (!more && lane == 0) {
          SsCtl* const c = a.ctl;
          c->total_reached += c->reached;
          c->total_levels += c->level;
          c->total_push += c->n_push;
          c->total_pull += c->n_pull;
        }
        __syncwarp();
        __threadfence();
        if (lane < 4) {
          const uint32_t lo = lane == 0 ? (uint32_t)nx.qn : lane == 1 ? (uint32_t)nx.ln : lane == 2 ? (uint32_t)nx.L : nx.arrived;
          const uint32_t hi = lane == 0 ? (more ? (uint32_t)nx.ctas : 0u) : lane == 1 ? (uint32_t)(nx.phase | nx.dirty << 8) : 0u;
          *static_cast<volatile unsigned long long*>(&a.sync->step.word[lane]) =
              (unsigned long long)((gen + 1) & 0xffffu) << 48 | (unsigned long long)hi << 32 | lo;
        }
      }
      __syncwarp();
      bool idle = false;
      for (uint32_t polls = 0;; polls++) {
        unsigned long long w;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(&a.sync->step.word[lane & 3]) : "memory");
        const uint32_t tag = (uint32_t)(w >> 48), tag0 = __shfl_sync(kFull, tag, 0);
        if (__all_sync(kFull, tag == tag0) && tag != gen) {
          gen = tag;
          polls = 0;
          const uint32_t hi = (uint32_t)(w >> 32) & 0xffffu, lo = (uint32_t)w;
          const uint32_t ctas = __shfl_sync(kFull, hi, 0), ph = __shfl_sync(kFull, hi, 1);
          const uint32_t qn = __shfl_sync(kFull, lo, 0), ln = __shfl_sync(kFull, lo, 1);
          const uint32_t L = __shfl_sync(kFull, lo, 2), arrived = __shfl_sync(kFull, lo, 3);
          if (ctas == 0 || blockIdx.x < ctas) {
            if (lane == 0) sm.st = BfsStep{(int)ctas, (int)(ph & 0xff), (int)(ph >> 8), (int)L, (int)qn, (int)ln, arrived};
            break;
          }
          idle = true;
        }
        if (polls == s_polls) {
          const uint32_t base = __shfl_sync(kFull, (uint32_t)w, 3);
          if (lane == 0) {
            atomicExch(&a.sync->arrive.n, base + kBfBroken);
            *a.err = DAWN_ERR_TIMEOUT;
            sm.st.ctas = 0;
          }
          break;
        }
        if (idle) __nanosleep(64);
      }
    }
    __syncthreads();
    if (st.ctas == 0) return;
  }
}

__global__ void __launch_bounds__(kBlock) fill_records(const int32_t* __restrict__ row_ptr,
                                                       const int32_t* __restrict__ col, int32_t n, int32_t len,
                                                       int32_t* __restrict__ rec) {
  const size_t words = (size_t)n * len, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < words; i += stride) {
    const int32_t v = (int32_t)(i / len), k = row_ptr[v] + (int32_t)(i % len);
    rec[i] = k < row_ptr[v + 1] ? col[k] : -1;
  }
}

// The records of a graph of low degree, once per handle: a row in whole sectors,
// so that a level's rows are one load away from its vertices.  Graphs of up to 12
// entries a row, none above kRecMax: meshes, street networks, kNN graphs, whose
// traversals take hundreds of small levels.  Beyond kMeshMax vertices, and with
// rows of more than eight entries beyond kMeshWide, these keep the level kernels
// and the cluster levels (kLevelKernels; records / level kernels, us a call: kNN of
// 9,000 points 280 / 291, 20,000 455 / 471, 32,000 545 / 575, of 200,000 1.54 / 1.23 ms).
// Random graphs of low degree have a few wide levels instead, which one SM with
// records is slow at: from kRandomFrom vertices on they go by their growth.  Records /
// level kernels / neither, us a call on Erdos-Renyi graphs of mean degree 11, 9,000
// vertices 101 / 89 / 74, 20,000 107 / 90 / 76, 32,000 126 / 97 / 82; of 7, 20,000
// 102 / 100 / 87; of 4 (growth 4.2 to 4.6) 9,000 88 / 90 / 101, 20,000 109 / 100 / 105,
// 32,000 113 / 122 / 111, 50,000 - / 131 / 108; of 2.5 20,000 117 / 115 / 136, 32,000 128 / 126 /
// 141, 50,000 - / 160 / 152; of 5, 3 M - / 365 / 297.
constexpr int32_t kLevelKernels = -2;
constexpr int32_t kRandomFrom = 6000, kRandomSlow = 26000, kRandomWide = 45000;
constexpr double kGrowsFast = 4.8, kGrowsWell = 3.5;
dawn_status records(dawn_graph* g) {
  if (g->rec_len != -1) return DAWN_OK;
  const int32_t n = g->n;
  int32_t len = 0;
  if (g->m <= 12 * (int64_t)n && n > kSoloKeep) {
    DAWN_CHECK(longest_row(g));
    const int32_t deg = g->max_row;
    len = std::max(8, (deg + 7) / 8 * 8);
    double growth = 0.0;
    if (deg <= kRecMax && n >= kRandomFrom) {
      DAWN_CHECK(read_growth(g));
      growth = g->growth;
    }
    if (deg > kRecMax || growth >= kGrowsFast || (growth >= kGrows && n > kRandomWide)) {
      len = 0;
    } else if (n > kMeshMax || (len > 8 && n > kMeshWide) || (growth >= kGrowsWell && n < kRandomSlow)) {
      len = kLevelKernels;
    } else {
      const dawn_status s = ensure(g->bfs_rec, sizeof(int32_t) * (size_t)n * len, g->stream);
      if (s == DAWN_ERR_OOM) {  // not decided: the next call tries again
        cudaGetLastError();
        clear_error();
        return DAWN_OK;
      }
      DAWN_CHECK(s);
      fill_records<<<g->geo.sms * 8, kBlock, 0, g->stream>>>(g->row_ptr, g->col, n, len, g->bfs_rec.as<int32_t>());
      DAWN_CUDA(cudaGetLastError());
    }
  }
  g->rec_len = len;
  return DAWN_OK;
}

// What the persistent launch needs beside the level kernels' buffers.
dawn_status persistent_buffers(dawn_graph* g, size_t lcap) {
  DAWN_CHECK(ensure(g->bfs_long, sizeof(int32_t) * 2 * lcap, g->stream));
  if (g->bfs_sync.p) return DAWN_OK;
  DAWN_CHECK(ensure(g->bfs_sync, sizeof(BfsSync), g->stream));
  DAWN_CUDA(cudaMemsetAsync(g->bfs_sync.p, 0, sizeof(BfsSync), g->stream));
  return DAWN_OK;
}

__global__ void ss_next(SsCtl* __restrict__ ctl) {
  if (threadIdx.x != 0) return;
  ctl->total_reached += ctl->reached;
  ctl->total_levels += ctl->level;
  ctl->total_push += ctl->n_push;
  ctl->total_pull += ctl->n_pull;
  ctl->src_idx += 1;
}

void probe_ss(const void* p, LevelProbe* out) {
  const SsCtl* c = static_cast<const SsCtl*>(p);
  const int pin = (c->level - 1) & 1;
  out->level = c->level;
  out->mode = c->mode;
  out->done = c->done;
  out->frontier = c->qsize[pin] + (int64_t)(c->lpack[pin] >> 32);
  out->frontier_edges = (int64_t)c->mf[pin];
  out->unvisited_edges = c->mu;
}

}  // namespace

dawn_status bfs_single(dawn_graph* g, const int32_t* sources, int32_t nsrc, int32_t* d_dist,
                       int32_t policy) {
  const int32_t n = g->n;
  int32_t nwords = (n + 31) / 32;
  long long m = g->m;
  DAWN_CHECK(ensure(g->ss_queues, sizeof(int32_t) * 2 * (size_t)n, g->stream));
  size_t segcap = seg_capacity(n, m);
  DAWN_CHECK(ensure(g->ss_segs, sizeof(Seg) * 2 * segcap, g->stream));
  DAWN_CHECK(ensure(g->ss_bitmaps, sizeof(uint32_t) * 4 * (size_t)nwords, g->stream));
  DAWN_CHECK(ensure(g->ss_ctl, sizeof(SsCtl), g->stream));
  const int32_t force = g->force_variant == 3 ? 1 + kVarPush : g->force_variant;
  if (g->small_levels) DAWN_CHECK(records(g));
  const size_t lcap = (size_t)(m / kLongRow) + 1;
  bool persistent = !g->trace && !(g->small_levels && g->rec_len == kLevelKernels);
  if (persistent) {
    const dawn_status s = persistent_buffers(g, lcap);
    if (s == DAWN_ERR_OOM) {  // the level kernels need neither
      cudaGetLastError();
      clear_error();
      persistent = false;
    } else {
      DAWN_CHECK(s);
    }
  }
  if (persistent) {
    BfsArgs a = {};
    a.row_ptr = g->row_ptr;
    a.col = g->col;
    a.t_row_ptr = g->t_row_ptr;
    a.t_col = g->t_col;
    a.ctl = g->ss_call = g->ss_ctl.as<SsCtl>();
    a.sync = g->bfs_sync.as<BfsSync>();
    a.q = g->ss_queues.as<int32_t>();
    a.segs = g->ss_segs.as<Seg>();
    a.segcap = segcap;
    a.lcap = lcap;
    a.lq = g->bfs_long.as<int32_t>();
    a.vbm = g->ss_bitmaps.as<uint32_t>();
    a.fbm = a.vbm + nwords;
    a.m = m;
    a.sel_w = g->sel_slot.as<float>();
    a.n = n;
    a.nwords = nwords;
    a.policy = policy;
    a.use_sel = g->sel_call;
    a.sel_margin = g->sel_margin;
    a.force = force;
    a.small = g->small_levels;
    a.polls = g->wait_polls;
    a.err = g->h_err;
    const bool mesh = g->small_levels && g->rec_len > 0;
    a.rec_len = mesh ? g->rec_len : 0;
    a.rec = mesh ? g->bfs_rec.as<int32_t>() : nullptr;
    const void* const fn = mesh ? (const void*)bfs_traverse<true> : (const void*)bfs_traverse<false>;
    const int threads = mesh ? 1024 : 640;
    constexpr size_t kMeshBytes = offsetof(BfsSmem<32>, mesh) + sizeof(MeshLists);
    static_assert(kMeshBytes + kMeshMax / 8 >= sizeof(BfsSmem<32>), "the largest size is the bitmap's");
    const size_t smem = mesh ? std::max(sizeof(BfsSmem<32>), kMeshBytes + sizeof(uint32_t) * (size_t)nwords)
                             : sizeof(BfsSmem<20>);
    if (g->bfs_fn != fn || g->bfs_cap != g->blocks_per_sm) {  // 8 us of every call otherwise
      DAWN_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     mesh ? (int)(kMeshBytes + kMeshMax / 8) : (int)smem));
      g->bfs_ctas = persistent_blocks(fn, threads, smem, g->blocks_per_sm);
      g->bfs_fn = fn;
      g->bfs_cap = g->blocks_per_sm;
    }
    // a small graph takes few CTAs: each adds to the arrivals of its phases
    const int64_t want = (n + m) / kBfEntries + 1;
    const int ctas = want < g->bfs_ctas ? (int)want : g->bfs_ctas;
    void* args[] = {&a};
    for (int32_t i = 0; i < nsrc; i++) {
      a.source = sources[i];
      a.first = i == 0;
      a.dist = d_dist + (size_t)i * n;
      DAWN_CUDA(cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(threads), args, smem, g->stream));
    }
    return DAWN_OK;
  }
  // level kernels: traced calls, and large graphs of low degree
  DAWN_CHECK(ensure(g->ss_sources, sizeof(int32_t) * (size_t)nsrc, g->stream));
  DAWN_CUDA(cudaMemcpyAsync(g->ss_sources.p, sources, sizeof(int32_t) * nsrc, cudaMemcpyHostToDevice,
                            g->stream));
  SsCtl c = {};
  c.policy = policy;
  c.nsrc = nsrc;
  c.dist_base = d_dist;
  c.sources = g->ss_sources.as<int32_t>();
  c.use_sel = g->sel_call;
  c.sel_margin = g->sel_margin;
  c.force = force;
  c.small = g->small_levels && cluster_fits((const void*)bfs_small, kSmallCtas, kSmallBlock) ? 1 : 0;
  c.m = m;
  DAWN_CHECK(upload_ctl(g, c));

  struct {
    SsCtl* ctl;
    const int32_t *row_ptr, *col, *t_row_ptr, *t_col;
    int32_t* q;
    Seg* segs;
    size_t segcap;
    uint32_t *bitmaps, *vbm, *fbm;
    int32_t n, nwords;
    long long m;
    cudaGraphConditionalHandle handle;
    int in_graph;
    const float* sel_w;
  } a;
  a.sel_w = g->sel_slot.as<float>();
  a.ctl = g->ss_ctl.as<SsCtl>();
  a.row_ptr = g->row_ptr;
  a.col = g->col;
  a.t_row_ptr = g->t_row_ptr;
  a.t_col = g->t_col;
  a.q = g->ss_queues.as<int32_t>();
  a.segs = g->ss_segs.as<Seg>();
  a.segcap = segcap;
  a.bitmaps = g->ss_bitmaps.as<uint32_t>();
  a.vbm = a.bitmaps;
  a.fbm = a.bitmaps + nwords;
  a.n = n;
  a.nwords = nwords;
  a.m = m;
  a.handle = 0;
  a.in_graph = 0;
  void* start_args[] = {&a.ctl, &a.row_ptr, &a.q, &a.segs, &a.bitmaps, &a.n, &a.nwords, &a.m};
  void* step_args[] = {&a.row_ptr, &a.col, &a.t_row_ptr, &a.t_col, &a.ctl, &a.q, &a.segs, &a.segcap, &a.vbm,
                       &a.fbm, &a.n, &a.nwords, &a.sel_w, &a.handle, &a.in_graph};
  void* small_args[] = {&a.row_ptr, &a.col, &a.ctl, &a.q, &a.segs, &a.segcap, &a.vbm, &a.fbm, &a.n, &a.nwords,
                        &a.sel_w, &a.handle, &a.in_graph};
  void* next_args[] = {&a.ctl};

  const int sms = g->geo.sms;
  SsFamily fam;
  fam.npre = 1;
  fam.pre[0] = {(const void*)bfs_start, start_args, dim3(sms * 8), dim3(kBlock), "bfs_start"};
  // Two kernels per loop iteration, each ending its level with the
  // bookkeeping (no separate decide launch): the push/pull level kernel and
  // the cluster levels; the one whose mode does not match returns at once.
  fam.nbody = 2;
  fam.decide_in_body = true;
  fam.body[0] = {(const void*)bfs_step, step_args,
                 dim3(persistent_blocks((const void*)bfs_step, kBlock, 0, g->blocks_per_sm)), dim3(kBlock),
                 "bfs_step", kModeStep};
  fam.body[1] = {(const void*)bfs_small, small_args, dim3(kSmallCtas), dim3(kSmallBlock), "bfs_small", kModeSmall};
  fam.npost = 1;
  fam.post[0] = {(const void*)ss_next, next_args, dim3(1), dim3(32), "ss_next"};
  fam.ctl = a.ctl;
  fam.ctl_bytes = sizeof(SsCtl);
  fam.probe = probe_ss;
  fam.handle = &a.handle;
  fam.in_graph = &a.in_graph;
  fam.done_flag = &a.ctl->done;
  return ss_run(g, fam, nsrc, &g->bfs_exec);
}

// --- single-source BFS with static scratch (dawn_bfs_static) ---------------
//
// Some callers may not allocate device memory at the moment they traverse:
// a serving loop whose device memory is entirely reserved by another
// allocator, or one that must never wait on the allocator (an allocation
// can synchronise the device, or fail under fragmentation, at a point where
// neither is acceptable).  For them the push traversal above runs over a
// fixed block of device memory that the library declares at file scope, so
// the call allocates nothing: the caller owns the CSR and the distance row,
// and every other word the traversal touches lives in `g_static_scratch`.
//
// The block holds a graph of at most kStaticMaxVertices vertices and
// kStaticMaxEdges edges (about 12.5 MiB).  It exists on a GPU once the
// library's kernels are loaded there (with lazy module loading, at the
// first launch of one of them on that device) and stays until the process
// exits.  There is one block per device,
// so calls that overlap on one device (from two host threads, or on two
// streams) race on it: the caller serialises them.

constexpr int32_t kStaticMaxVertices = DAWN_STATIC_MAX_VERTICES;
constexpr long long kStaticMaxEdges = DAWN_STATIC_MAX_EDGES;
constexpr size_t kStaticSegCap = 2 * (size_t)(kStaticMaxEdges / kSeg) + 64;  // seg_capacity at the maxima
constexpr size_t kStaticWords = (size_t)(kStaticMaxVertices + 31) / 32;
// layout (byte offsets, each 256-aligned): control block | source | flags |
// 4 bitmaps | 2 vertex queues | 2 segment lists
constexpr size_t kStaticCtlOff = 0;
constexpr size_t kStaticSrcOff = 512;
constexpr size_t kStaticFlagOff = 768;
constexpr size_t kStaticBitmapOff = 1024;
constexpr size_t kStaticQueueOff = kStaticBitmapOff + 4 * kStaticWords * sizeof(uint32_t);
constexpr size_t kStaticSegOff = kStaticQueueOff + 2 * (size_t)kStaticMaxVertices * sizeof(int32_t);
constexpr size_t kStaticBytes = kStaticSegOff + 2 * kStaticSegCap * sizeof(Seg);
static_assert(sizeof(SsCtl) <= kStaticSrcOff, "control block overlaps the source slot");
static_assert(kStaticQueueOff % 256 == 0 && kStaticSegOff % 256 == 0, "scratch regions must stay 256-aligned");

static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

namespace {

constexpr int kStaticPollLevels = 8;  // levels launched between two reads of the done flag
constexpr int kStaticMaxDevices = 64;

struct StaticDevice {
  std::once_flag once;
  cudaError_t err = cudaSuccess;
  unsigned char* scratch = nullptr;
  int clear_blocks = 0, push_blocks = 0, check_blocks = 0;
};
StaticDevice g_static_dev[kStaticMaxDevices];

// Set-up of one device, run once with that device current: the address of
// its copy of the scratch block and the launch shapes.
void static_setup(StaticDevice& d) {
  d.err = cudaGetSymbolAddress(reinterpret_cast<void**>(&d.scratch), g_static_scratch);
  if (d.err != cudaSuccess) return;
  int dev = 0, sms = 0, per_sm = 0;
  if ((d.err = cudaGetDevice(&dev)) != cudaSuccess) return;
  if ((d.err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return;
  if ((d.err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_push, kBlock, 0)) != cudaSuccess) return;
  d.push_blocks = sms * (per_sm > 0 ? per_sm : 1);
  d.clear_blocks = sms * 4;
  d.check_blocks = sms * 8;
}

// CSR checks of the static path: same invariants as the upload-time
// validation, with scalar loads (the caller's arrays carry no alignment
// promise beyond 4 bytes).  Flags: 1 row_ptr[0] != 0, 2 row_ptr[n] != m,
// 4 row_ptr decreases, 8 column outside [0, n).
__global__ void __launch_bounds__(kBlock) static_check_csr(const int32_t* __restrict__ rp,
                                                           const int32_t* __restrict__ col, int32_t n, long long m,
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
  for (size_t k = tid; k < (size_t)m; k += stride) {
    const int32_t c = __ldg(col + k);
    if (c < 0 || c >= n) f |= 8;
  }
  if (f) atomicOr(flags, f);
}

// Writes the control block of a one-source push traversal into the
// scratch (every field, so nothing is left from an earlier call) and clears
// the flag word.
__global__ void static_begin(SsCtl* __restrict__ ctl, int32_t* __restrict__ src_slot, int* __restrict__ flags,
                             int32_t source, int32_t* dist) {
  if (threadIdx.x != 0) return;
  SsCtl c = {};
  c.policy = DAWN_VARIANT_PUSH;
  c.nsrc = 1;
  c.dist_base = dist;
  c.sources = src_slot;
  *ctl = c;
  *src_slot = source;
  *flags = 0;
}

}  // namespace

dawn_status bfs_static(const int32_t* row_ptr, const int32_t* col, int32_t n, int64_t m, int32_t source,
                       int32_t* dist, uint32_t flags, cudaStream_t stream) {
  if (!row_ptr || !dist || (m > 0 && !col)) {
    set_error("dawn_bfs_static: row_ptr, col and dist must be device pointers (col may be NULL only when m = 0)");
    return DAWN_ERR_INVALID_ARG;
  }
  if (n < 1 || n > kStaticMaxVertices) {
    set_error("dawn_bfs_static: n = %d outside [1, %d], the vertex limit of the static scratch block", n,
              kStaticMaxVertices);
    return DAWN_ERR_INVALID_ARG;
  }
  if (m < 0 || m > kStaticMaxEdges) {
    set_error("dawn_bfs_static: m = %lld outside [0, %lld], the edge limit of the static scratch block",
              (long long)m, kStaticMaxEdges);
    return DAWN_ERR_INVALID_ARG;
  }
  if (source < 0 || source >= n) {
    set_error("dawn_bfs_static: source %d outside [0, %d)", source, n);
    return DAWN_ERR_INVALID_ARG;
  }
  int dev = 0;
  DAWN_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices) {
    set_error("dawn_bfs_static: device %d beyond the %d devices the library tracks", dev, kStaticMaxDevices);
    return DAWN_ERR_UNSUPPORTED;
  }
  const void* ptrs[3] = {row_ptr, col, dist};
  for (const void* p : ptrs) {
    if (!p) continue;
    cudaPointerAttributes at;
    DAWN_CUDA(cudaPointerGetAttributes(&at, p));
    if ((at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged) || at.device != dev) {
      set_error("dawn_bfs_static: row_ptr, col and dist must be memory of the current device (%d)", dev);
      return DAWN_ERR_INVALID_ARG;
    }
  }
  StaticDevice& d = g_static_dev[dev];
  std::call_once(d.once, static_setup, std::ref(d));
  DAWN_CUDA(d.err);

  SsCtl* ctl = reinterpret_cast<SsCtl*>(d.scratch + kStaticCtlOff);
  int32_t* src_slot = reinterpret_cast<int32_t*>(d.scratch + kStaticSrcOff);
  int* d_flags = reinterpret_cast<int*>(d.scratch + kStaticFlagOff);
  uint32_t* bitmaps = reinterpret_cast<uint32_t*>(d.scratch + kStaticBitmapOff);
  int32_t* q = reinterpret_cast<int32_t*>(d.scratch + kStaticQueueOff);
  Seg* segs = reinterpret_cast<Seg*>(d.scratch + kStaticSegOff);
  const int32_t nwords = (n + 31) / 32;
  uint32_t* vbm = bitmaps;
  uint32_t* fbm = bitmaps + nwords;

  static_begin<<<1, 32, 0, stream>>>(ctl, src_slot, d_flags, source, dist);
  DAWN_CUDA(cudaGetLastError());
  if (!(flags & DAWN_GRAPH_NO_VALIDATE)) {
    static_check_csr<<<d.check_blocks, kBlock, 0, stream>>>(row_ptr, col, n, (long long)m, d_flags);
    DAWN_CUDA(cudaGetLastError());
    int f = 0;
    DAWN_CUDA(cudaMemcpyAsync(&f, d_flags, sizeof(int), cudaMemcpyDeviceToHost, stream));
    DAWN_CUDA(cudaStreamSynchronize(stream));
    if (f) {
      set_error("dawn_bfs_static: invalid CSR:%s%s%s%s", (f & 1) ? " row_ptr[0] != 0;" : "",
                (f & 2) ? " row_ptr[n] != m;" : "", (f & 4) ? " row_ptr decreases;" : "",
                (f & 8) ? " col index outside [0, n);" : "");
      return DAWN_ERR_INVALID_ARG;
    }
  }
  // bfs_clear fills the distance row with -1 and zeroes the visited and
  // frontier bitmaps; bfs_init seeds the source.  Queues and segment lists
  // are read only up to the sizes the control block records.
  bfs_clear<<<d.clear_blocks, kBlock, 0, stream>>>(ctl, bitmaps, n, nwords);
  DAWN_CUDA(cudaGetLastError());
  bfs_init<<<1, 32, 0, stream>>>(ctl, row_ptr, q, segs, vbm, n, (long long)m);
  DAWN_CUDA(cudaGetLastError());
  // Levels after the last one return at once (done is set), so the host
  // reads the flag only every kStaticPollLevels levels.  Each level sets
  // done once its frontier is empty or the level count reaches n.
  for (;;) {
    for (int j = 0; j < kStaticPollLevels; j++) {
      bfs_push<<<d.push_blocks, kBlock, 0, stream>>>(row_ptr, col, ctl, q, segs, kStaticSegCap, vbm, fbm, n,
                                                      nwords);
      bfs_decide<<<1, 32, 0, stream>>>(ctl, n, nullptr, 0, 0);
    }
    DAWN_CUDA(cudaGetLastError());
    int32_t done = 0;
    DAWN_CUDA(cudaMemcpyAsync(&done, &ctl->done, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    DAWN_CUDA(cudaStreamSynchronize(stream));
    if (done) break;
  }
  return DAWN_OK;
}

}  // namespace dawn
