// Many independent graphs in one persistent launch, on sm_103a.
//
// The reference traverses one graph per process call: MSSP_GPU::run
// (src/algorithm/gpu/mssp.cu:9-51) copies a CSR, loops over its sources and
// frees it.  A workload of hundreds of small graphs then pays a CSR upload,
// per-level launches and host syncs for every (graph, source).  Here the
// graphs are the parts of one disjoint-union CSR (part p owns the vertex
// range [off[p], off[p+1]) and no edge leaves its part), and one persistent
// kernel runs every (part, batch of sources) task.  Tasks come in two forms,
// chosen per call (parts_bfs): single CTAs with the part's words in shared
// memory (parts_small, below), and, for parts too large for that, for few
// large parts and for traced calls, 64 sources on a cluster:
//
//   * a thread-block cluster (kPartCluster CTAs on as many SMs) takes the
//     next task from a device counter (tasks sorted by estimated cost,
//     longest first, so the long ones start early) and runs the whole
//     multi-source bitset traversal of that part, its CTAs splitting every
//     vertex and row sweep, with cluster barriers between phases and the
//     level counters summed through distributed shared memory: no launch
//     per level, no host sync, and no wait on another cluster;
//   * its working words live in a per-cluster slot of global memory
//     (visited, two frontier words, a push accumulator and bit-sliced
//     levels, one uint64 per vertex each); the part's words stay in L2
//     while the cluster works on them;
//   * each level is a push (frontier rows scattered with atomicOr into the
//     accumulator, then a sweep folding it in) or a pull (each unfinished
//     vertex ORs its in-neighbours' frontier words, stopping once no
//     missing bit is left), chosen by the same frontier-edge rule as the
//     single-graph bitset traversal;
//   * the distances of a task are emitted once, at its end, from the level
//     slices, with coalesced stores, and the emit pass zeroes every word the
//     task used, so the slot is clean for the next task without a separate
//     clearing pass.
//
// Hop distances are those of a separate BFS of each part from each source:
// bit b of a vertex's word appears at level L exactly when source b first
// reaches it at L, whatever the direction of each level.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "dawn_device.cuh"

namespace dawn {
namespace {

using u64 = unsigned long long;
constexpr int kPartBlock = 1024;
constexpr int kPartSlices = 8;  // level slices kept in registers by the emit pass
constexpr int kPartLaneMax = 64;  // rows below this many entries are walked by one lane
constexpr int kPartCluster = 8;   // CTAs (SMs) per task: a thread-block cluster (1 where 8 do not fit)

struct PartsCtl {
  int32_t next_task;    // task counter of the persistent grid
  int32_t ntasks;
  int32_t push_ratio;   // push while ratio * frontier edges < unfinished in-edges
  int32_t pad0;
  const PartTask* tasks;
  const int32_t* sources;  // part-local source ids, in task order
  int32_t* dist;           // output base
  unsigned long long reached;  // TEPS numerator, all tasks
  unsigned long long levels, push_levels, pull_levels;
  unsigned long long* task_log;  // tracing: 4 words per task, else NULL
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned sm_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

__device__ __forceinline__ u64 block_reduce_add(u64 x, u64* s_slot) {
  x = warp_sum(x);
  if (lane_id() == 0 && x) atomicAdd(s_slot, x);
  return x;
}

// Cluster tasks: distances of one vertex for the task's nb sources from its visited word
// and level slices; NB slices are read into registers, the rest (levels of
// 256 and above) from memory.
template <int NB>
__device__ __forceinline__ void emit_part_vertex(int32_t* __restrict__ dist, int32_t np, int nb, int u, u64 vis,
                                                 u64* __restrict__ slices, int32_t maxn, int nbits) {
  u64 w[NB > 0 ? NB : 1];
#pragma unroll
  for (int k = 0; k < NB; k++) {
    w[k] = slices[(size_t)k * maxn + u];
    slices[(size_t)k * maxn + u] = 0ull;
  }
  for (int b = 0; b < nb; b++) {
    int32_t v = -1;
    if ((vis >> b) & 1ull) {
      v = 0;
#pragma unroll
      for (int k = 0; k < NB; k++) v |= (int32_t)((w[k] >> b) & 1ull) << k;
      for (int k = NB; k < nbits; k++) v |= (int32_t)((slices[(size_t)k * maxn + u] >> b) & 1ull) << k;
    }
    dist[(size_t)b * np + u] = v;
  }
  for (int k = NB; k < nbits; k++) slices[(size_t)k * maxn + u] = 0ull;
}

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kPartBlock, 1)
    parts_traverse(PartsCtl* __restrict__ ctl,
                                                           const int32_t* __restrict__ row_ptr,
                                                           const int32_t* __restrict__ col,
                                                           const int32_t* __restrict__ t_row_ptr,
                                                           const int32_t* __restrict__ t_col,
                                                           const int32_t* __restrict__ voff,
                                                           u64* __restrict__ scratch, size_t slot_words,
                                                           int32_t maxn) {
  // Per level (by parity): frontier out-edges, in-edges of the vertices
  // finished, vertices reached.  Each CTA counts its own; the cluster's
  // totals are read through distributed shared memory after the level's
  // barrier, and a CTA resets its counters of the other parity then (every
  // reader of those passed the barrier).
  __shared__ int s_task;
  __shared__ u64 s_cnt[2][3];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  const int ctid = crank * kPartBlock + tid;  // thread index within the cluster
  constexpr int kThreads = C * kPartBlock;
  const int lane = lane_id(), wib = tid >> 5;
  const int cwarp = crank * (kPartBlock / 32) + wib;
  u64* const visit = scratch + (size_t)(blockIdx.x / C) * slot_words;
  u64* const fa = visit + maxn;
  u64* const fb = fa + maxn;
  u64* const acc = fb + maxn;
  u64* const slices = acc + maxn;
  const int ratio = ctl->push_ratio;
  u64 my_reached = 0;
  u64 t_levels = 0, t_push = 0, t_pull = 0;

  auto totals = [&](int par, u64& mf_t, u64& dec_t, u64& nf_t) {
    mf_t = dec_t = nf_t = 0;
#pragma unroll
    for (int r = 0; r < C; r++) {
      const u64* c = cluster.map_shared_rank(&s_cnt[par][0], r);
      mf_t += c[0];
      dec_t += c[1];
      nf_t += c[2];
    }
  };
  for (;;) {
    if (crank == 0 && tid == 0) s_task = atomicAdd(&ctl->next_task, 1);
    if (tid < 6) (&s_cnt[0][0])[tid] = 0;
    cluster.sync();
    const int t = *cluster.map_shared_rank(&s_task, 0);
    if (t >= ctl->ntasks) break;
    const PartTask task = ctl->tasks[t];
    const int32_t v0 = voff[task.part];
    const int32_t np = voff[task.part + 1] - v0;
    const int nb = task.nsrc;
    const u64 full = nb == 64 ? ~0ull : ((1ull << nb) - 1ull);
    const int32_t* src = ctl->sources + task.src0;
    const long long mp = (long long)row_ptr[v0 + np] - row_ptr[v0];
    unsigned long long t_start = 0, push0 = t_push;
    if (ctid == 0 && ctl->task_log) t_start = global_ns();
    // Seed: source b sets bit b at its vertex (the cluster's first CTA;
    // its level-0 counters take the seeds' rows).
    if (ctid < nb) {
      const int32_t s = src[ctid];
      atomicOr(visit + s, 1ull << ctid);
      atomicOr(fa + s, 1ull << ctid);
    }
    __syncthreads();
    if (ctid < nb) {
      const int32_t s = src[ctid];
      const int32_t gs = v0 + s;
      const u64 deg = (u64)(row_ptr[gs + 1] - row_ptr[gs]);
      my_reached += deg;
      // the thread of the lowest bit at a vertex counts the vertex once
      if ((fa[s] & ((1ull << ctid) - 1ull)) == 0ull) {
        atomicAdd(&s_cnt[0][0], deg);
        if (visit[s] == full) atomicAdd(&s_cnt[0][1], (u64)(t_row_ptr[gs + 1] - t_row_ptr[gs]));
      }
    }
    cluster.sync();
    long long mf, mu;
    {
      u64 a0, a1, a2;
      totals(0, a0, a1, a2);
      mf = (long long)a0;
      mu = mp - (long long)a1;
    }
    u64* cur = fa;
    u64* nxt = fb;
    int L = 1;
    for (;;) {
      const bool push = mf * ratio < mu;
      const int par = L & 1;  // this level's counters; level 0 used the other parity
      if (push) {
        // scatter: the frontier rows of 32 consecutive vertices per warp
        // task; rows of >= kPartLaneMax entries swept by the whole warp,
        // shorter ones walked by one lane each (no shared-memory search per
        // edge: these loops are bound by their L1/TEX traffic)
        for (int base = cwarp * 32; base < np; base += kThreads) {
          const int v = base + lane;
          const u64 f = v < np ? cur[v] : 0ull;
          int rs = 0, re = 0;
          if (f) {
            rs = row_ptr[v0 + v];
            re = row_ptr[v0 + v + 1];
          }
          const int deg = re - rs;
          if (__ballot_sync(kFull, deg > 0) == 0u) continue;
          uint32_t big = __ballot_sync(kFull, deg >= kPartLaneMax);
          while (big) {
            const int leader = __ffs(big) - 1;
            big &= big - 1;
            const u64 lf = __shfl_sync(kFull, f, leader);
            const int ks = __shfl_sync(kFull, rs, leader), ke = __shfl_sync(kFull, re, leader);
            for (int k = ks + lane; k < ke; k += 32) {
              const int u = __ldg(col + k) - v0;
              const u64 bits = lf & ~visit[u];
              if (bits) atomicOr(acc + u, bits);
            }
          }
          // short rows: one lane each, four targets in flight
          if (deg > 0 && deg < kPartLaneMax) {
            for (int k = rs; k < re; k += 4) {
              int u[4];
#pragma unroll
              for (int j = 0; j < 4; j++) u[j] = k + j < re ? __ldg(col + k + j) - v0 : -1;
              u64 bits[4];
#pragma unroll
              for (int j = 0; j < 4; j++) bits[j] = u[j] >= 0 ? f & ~visit[u[j]] : 0ull;
#pragma unroll
              for (int j = 0; j < 4; j++)
                if (bits[j]) atomicOr(acc + u[j], bits[j]);
            }
          }
        }
      }
      if (push) cluster.sync();  // the scatter's ORs are in before the sweep reads them
      u64 lmf = 0, ldec = 0, lnf = 0;
      for (int base = cwarp * 32; base < np; base += kThreads) {
        const int u = base + lane;
        const bool in = u < np;
        const int gu = v0 + u;
        // every load of the vertex's own words and row bounds is issued at
        // once, ahead of the gathers that need them
        u64 vis = full, x = 0ull;
        int rp0 = 0, rp1 = 0, tr0 = 0, tr1 = 0;
        if (in) {
          vis = visit[u];
          rp0 = row_ptr[gu];
          rp1 = row_ptr[gu + 1];
          tr0 = t_row_ptr[gu];
          tr1 = t_row_ptr[gu + 1];
          if (push) x = acc[u];
        }
        u64 nw = 0ull;
        if (push) {
          if (x) {
            acc[u] = 0ull;
            nw = x & ~vis;
          }
        } else {
          // pull: unfinished vertices OR their in-neighbours' frontier
          // words; long rows by the whole warp, short rows by one lane
          // each, both stopping once no missing bit is left
          const bool active = vis != full;
          const int rs = active ? tr0 : 0, re = active ? tr1 : 0;
          const int deg = re - rs;
          u64 got = 0ull;
          uint32_t big = __ballot_sync(kFull, deg >= kPartLaneMax);
          while (big) {
            const int leader = __ffs(big) - 1;
            big &= big - 1;
            const u64 lvis = __shfl_sync(kFull, vis, leader);
            const int ks = __shfl_sync(kFull, rs, leader), ke = __shfl_sync(kFull, re, leader);
            u64 w = 0ull;
            for (int k0 = ks; k0 < ke; k0 += 128) {
              const int k = k0 + lane;
              const int32_t c0 = k < ke ? __ldg(t_col + k) : -1;
              const int32_t c1 = k + 32 < ke ? __ldg(t_col + k + 32) : -1;
              const int32_t c2 = k + 64 < ke ? __ldg(t_col + k + 64) : -1;
              const int32_t c3 = k + 96 < ke ? __ldg(t_col + k + 96) : -1;
              if (c0 >= 0) w |= cur[c0 - v0];
              if (c1 >= 0) w |= cur[c1 - v0];
              if (c2 >= 0) w |= cur[c2 - v0];
              if (c3 >= 0) w |= cur[c3 - v0];
              if ((warp_or(w) | lvis) == full) break;
            }
            w = warp_or(w);
            if (lane == leader) got = w;
          }
          // short rows: one lane each, four in-neighbours in flight,
          // stopping once the missing bits are all found
          if (active && deg < kPartLaneMax) {
            u64 w = 0ull;
            for (int k = rs; k < re; k += 4) {
              int32_t c[4];
#pragma unroll
              for (int j = 0; j < 4; j++) c[j] = k + j < re ? __ldg(t_col + k + j) : -1;
#pragma unroll
              for (int j = 0; j < 4; j++)
                if (c[j] >= 0) w |= cur[c[j] - v0];
              if ((w | vis) == full) break;
            }
            got = w;
          }
          nw = got & ~vis;
        }
        if (!in) continue;
        nxt[u] = nw;
        if (nw) {
          visit[u] = vis | nw;
          // the bits are new to every slice, so an OR without a return
          // (no load on the thread's path) records them
          for (unsigned l = (unsigned)L; l; l &= l - 1) atomicOr(slices + (size_t)(__ffs(l) - 1) * maxn + u, nw);
          const u64 od = (u64)(rp1 - rp0);
          lmf += od;
          my_reached += od * (u64)__popcll(nw);
          lnf++;
          if ((vis | nw) == full) ldec += (u64)(tr1 - tr0);
        }
      }
      block_reduce_add(lmf, &s_cnt[par][0]);
      block_reduce_add(ldec, &s_cnt[par][1]);
      block_reduce_add(lnf, &s_cnt[par][2]);
      if (push) t_push++; else t_pull++;
      cluster.sync();
      u64 mf_t, dec_t, nf_t;
      totals(par, mf_t, dec_t, nf_t);
      // every reader of the other parity's counters is past the barrier,
      // and this CTA's next-level sums wait for the reset
      if (tid < 3) s_cnt[par ^ 1][tid] = 0;
      __syncthreads();
      if (nf_t == 0 || L >= np) break;
      mf = (long long)mf_t;
      mu -= (long long)dec_t;
      u64* tmp = cur;
      cur = nxt;
      nxt = tmp;
      L++;
    }
    t_levels += (u64)L;
    // Emit: the last level found nothing, so the deepest level is L - 1.
    const int deepest = L - 1;
    const int nbits = deepest > 0 ? 32 - __clz(deepest) : 0;
    int32_t* dist = ctl->dist + task.out0;
    for (int u = ctid; u < np; u += kThreads) {
      const u64 vis = visit[u];
      visit[u] = 0ull;
      fa[u] = 0ull;
      fb[u] = 0ull;
      switch (nbits < kPartSlices ? nbits : kPartSlices) {
        case 0: emit_part_vertex<0>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 1: emit_part_vertex<1>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 2: emit_part_vertex<2>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 3: emit_part_vertex<3>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 4: emit_part_vertex<4>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 5: emit_part_vertex<5>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 6: emit_part_vertex<6>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        case 7: emit_part_vertex<7>(dist, np, nb, u, vis, slices, maxn, nbits); break;
        default: emit_part_vertex<kPartSlices>(dist, np, nb, u, vis, slices, maxn, nbits); break;
      }
    }
    cluster.sync();  // the slot is clean before the next task seeds it
    if (ctid == 0 && ctl->task_log) {
      unsigned long long* r = ctl->task_log + 4 * (size_t)t;
      r[0] = t_start;
      r[1] = global_ns();
      r[2] = ((unsigned long long)L << 32) | (unsigned)(t_push - push0);
      r[3] = sm_id();
    }
  }
  cluster.sync();  // no CTA exits while another may still read its task slot
  my_reached = warp_sum(my_reached);
  if (lane_id() == 0 && my_reached) atomicAdd(&ctl->reached, my_reached);
  if (ctid == 0 && t_levels) {
    atomicAdd(&ctl->levels, t_levels);
    atomicAdd(&ctl->push_levels, t_push);
    atomicAdd(&ctl->pull_levels, t_pull);
  }
}

// --- parts whose words fit shared memory: one CTA per task -------------------
//
// The cluster kernel above gathers an in-neighbour's word from L2 for every
// entry, one L1/TEX sector per SM clock at best, with its CTAs waiting on
// each other at every phase.  A part of np vertices fits the 227 KB of one
// SM with 16 or 32 bits per vertex, and shared memory serves about nine
// random gathers per clock, so here a task is one CTA's: up to 16 or 32
// sources of one part (a longer source list is cut into more tasks), the
// visited words in shared memory, and block barriers only.
//   * A level reads the visited words `V` as they were at its start and
//     writes every vertex's new bits to that level's word array; after a
//     barrier each thread folds the vertices it owns into V.  Visited words
//     serve as frontier words: bits older than the last level are already at
//     every out-neighbour.
//   * Push and pull follow the same rule as everywhere, with a heavier weight
//     on the push: its atomics go to L2.  A push walks the list of vertices
//     that gained bits; a pull streams the in-edge columns of the unfinished
//     vertices past L1.  The columns are kept as 16-bit part-local ids in rows
//     padded to eight (made when the parts are declared; the padding names a
//     word that is always 0), so a 16-byte load brings eight of them, a row of
//     average length comes in one round trip and no entry is checked against
//     the row's bounds.
//   * The word arrays of levels 1 .. kPartDeep - 1 are expanded into the
//     distance rows at the end, in full lines; deeper levels are stored at
//     once (and share the last array).
// 300 directed ER graphs (1,024 to 65,536 vertices, degrees 4 to 32, 8 to 64
// sources): 5.08 ms as cluster tasks, 1.64 ms here (3.44 with global-memory
// accumulators and 32-bit columns, 2.21 with a word array per level).  What bounds
// it is latency at the 32 warps an SM holds beside a part's words: 512 such graphs
// issue 1.6 instructions a clock with L1 and shared memory at 44% and HBM at 2.55 TB/s
// (2.76 ms), about 1 ns per vertex and level.
constexpr int kPartDeep = 15;
constexpr int kPartPush = 4;  // times the handle's push ratio
constexpr int kPartLanePieces = 8;  // in-rows of this many pieces are swept by the warp

// Eight in-edge columns (part-local, 16 bits each), past L1; 16-byte aligned.
__device__ __forceinline__ uint4 part_cols(const uint16_t* p) {
  uint4 c;
  asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(c.x), "=r"(c.y), "=r"(c.z), "=r"(c.w)
               : "l"(p));
  return c;
}
// The visited words of a single-CTA task.  Referenced by name, so that the
// gathers compile to scaled shared-memory loads.
extern __shared__ __align__(16) unsigned char s_part_words[];

// OR of the words that eight columns name.
template <class T>
__device__ __forceinline__ unsigned or_cols(const uint4& c) {
  const T* V = reinterpret_cast<const T*>(s_part_words);
  const unsigned a = (unsigned)V[c.x & 0xffffu] | V[c.x >> 16], b = (unsigned)V[c.y & 0xffffu] | V[c.y >> 16];
  const unsigned d = (unsigned)V[c.z & 0xffffu] | V[c.z >> 16], e = (unsigned)V[c.w & 0xffffu] | V[c.w >> 16];
  return a | b | d | e;
}

// OR into word u of a T array through the 32-bit word holding it.
template <class T>
__device__ __forceinline__ void or_word(T* a, int u, unsigned bits) {
  if constexpr (sizeof(T) == 4)
    atomicOr(reinterpret_cast<unsigned*>(a) + u, bits);
  else
    atomicOr(reinterpret_cast<unsigned*>(a) + (u >> 1), bits << (16 * (u & 1)));
}

struct PartShared {
  int nf;    // vertices that gained bits
  int done;  // vertices that hold every bit
  int task;
};

// Distances of vertex u for the task's sources: slice k holds bit k of its
// levels; all four bits set (no level here) is an unreached pair, or one
// reached at kPartDeep or later, which is already written (deep).
__device__ __forceinline__ void emit_small_vertex(int32_t* __restrict__ dist, int np, int nb, unsigned vis,
                                                  const unsigned (&w)[4], bool deep) {
  int32_t* out = dist;
  for (int c = 0; c < nb; c += 8) {
    // byte c / 8 of the four slices in one word: the level of source c + b is
    // bits b, 8 + b, 16 + b, 24 + b, gathered by one multiplication (each
    // partial product lands on a bit of its own)
    const unsigned x = ((w[0] >> c) & 0xffu) | ((w[1] >> c) & 0xffu) << 8 | ((w[2] >> c) & 0xffu) << 16 |
                       ((w[3] >> c) & 0xffu) << 24;
    const int lim = min(8, nb - c);
#pragma unroll
    for (int b = 0; b < 8; b++, out += np) {
      if (b >= lim) break;
      const unsigned level = (((x >> b) & 0x01010101u) * 0x01020408u) >> 24;
      if (level == 15u && deep && ((vis >> (c + b)) & 1u)) continue;
      *out = level == 15u ? -1 : (int32_t)level;
    }
  }
}

template <class T, int kThreads>
__device__ __forceinline__ void small_task(const PartsCtl* __restrict__ ctl, const PartTask& task, PartShared& sh,
                                           T* __restrict__ words, size_t pitch,
                                           int32_t* __restrict__ list, const int32_t* __restrict__ row_ptr,
                                           const int32_t* __restrict__ col, const int32_t* __restrict__ t_off,
                                           const uint16_t* __restrict__ t_col, int32_t v0, int np, u64& my_reached,
                                           u64& t_levels, u64& t_push, u64& t_pull) {
  T* const V = reinterpret_cast<T*>(s_part_words);
  const int tid = threadIdx.x, lane = lane_id(), wib = tid >> 5;
  constexpr int kWarps = kThreads / 32;
  const int nb = task.nsrc;
  const unsigned full = nb == 32 ? 0xffffffffu : (1u << nb) - 1u;
  const int32_t* src = ctl->sources + task.src0;
  int32_t* dist = ctl->dist + task.out0;
  const long long ratio = (long long)ctl->push_ratio * kPartPush;
  const int listed = np / 8 + 64;  // longer frontiers are not listed: the next level pulls
  for (int u = tid; u <= np; u += kThreads) V[u] = 0;  // V[np] stays 0: the padding of the in-rows
  if (tid == 0) sh.nf = sh.done = 0;
  __syncthreads();
  if (tid < nb) or_word(V, src[tid], 1u << tid);
  __syncthreads();
  if (tid < nb) {
    const int s = src[tid];
    // the thread of the lowest bit at a vertex counts and lists it once
    if ((V[s] & ((1u << tid) - 1u)) == 0) {
      if (V[s] == full) atomicAdd(&sh.done, 1);
      list[atomicAdd(&sh.nf, 1)] = s;
    }
  }
  __syncthreads();
  int L = 1;
  for (;; L++) {
    const int nf = sh.nf;
    if (nf == 0 || L > np) break;
    // push while the frontier, weighed, is smaller than what is unfinished
    // (vertices stand for their edges: reading every row's bounds at every
    // level costs more than the better estimate saves)
    const bool push = nf <= listed && nf * ratio < np - sh.done;
    T* const N = words + (size_t)min(L, kPartDeep) * pitch;
    if (push)
      for (int u = tid; u < np; u += kThreads) N[u] = 0;
    __syncthreads();
    if (tid == 0) sh.nf = 0;
    if (push) {
      // a short list is dealt over all warps, each row swept by its warp
      const bool few = nf <= 4 * kWarps;
      const int per = few ? (nf + kWarps - 1) / kWarps : 32, sweep = few ? 1 : kWarpRow;
      for (int b = wib * per; b < nf; b += kWarps * per) {
        const int i = b + lane;
        int v = -1, rs = 0, re = 0;
        unsigned f = 0;
        if (lane < per && i < nf) {
          v = list[i];
          f = V[v];
          rs = row_ptr[v0 + v];
          re = row_ptr[v0 + v + 1];
        }
        const int deg = re - rs;
        uint32_t big = __ballot_sync(kFull, deg >= sweep);
        while (big) {
          const int l = __ffs(big) - 1;
          big &= big - 1;
          const unsigned lf = __shfl_sync(kFull, f, l);
          const int ks = __shfl_sync(kFull, rs, l), ke = __shfl_sync(kFull, re, l);
          for (int k = ks + lane; k < ke; k += 32) {
            const int u = __ldg(col + k) - v0;
            const unsigned bits = lf & ~(unsigned)V[u];
            if (bits) or_word(N, u, bits);
          }
        }
        if (deg < sweep)
          for (int k = rs; k < re; k += 4) {
            int u[4];
#pragma unroll
            for (int j = 0; j < 4; j++) u[j] = k + j < re ? __ldg(col + k + j) - v0 : -1;
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const unsigned bits = u[j] >= 0 ? f & ~(unsigned)V[u[j]] : 0u;
              if (bits) or_word(N, u[j], bits);
            }
          }
      }
    } else {
      // the bounds of the next 32 rows are loaded while these are walked
      unsigned vis = full;
      int rs = 0, re = 0;
      auto bounds = [&](int u) {
        vis = u < np ? (unsigned)V[u] : full;
        rs = re = 0;
        if (vis != full) {
          rs = __ldg(t_off + v0 + u);
          re = __ldg(t_off + v0 + u + 1);
        }
      };
      bounds(wib * 32 + lane);
      for (int base = wib * 32; base < np; base += kThreads) {
        const unsigned my = vis;
        const int ks0 = rs, ke0 = re;  // in pieces of eight columns
        bounds(base + kThreads + lane);
        unsigned got = 0;
        uint32_t big = __ballot_sync(kFull, ke0 - ks0 >= kPartLanePieces);
        while (big) {
          const int l = __ffs(big) - 1;
          big &= big - 1;
          const unsigned lvis = __shfl_sync(kFull, my, l);
          const int ks = __shfl_sync(kFull, ks0, l), ke = __shfl_sync(kFull, ke0, l);
          unsigned w = 0;
          for (int k = ks; k < ke; k += 32) {
            if (k + lane < ke) w |= or_cols<T>(part_cols(t_col + 8 * (size_t)(k + lane)));
            w = __reduce_or_sync(kFull, w);
            if ((w | lvis) == full) break;
          }
          if (lane == l) got = w;
        }
        if (ke0 > ks0 && ke0 - ks0 < kPartLanePieces) {
          // a lane's row, four pieces in flight
          unsigned w = 0;
          const uint16_t* p = t_col + 8 * (size_t)ks0;
          uint4 c[4];
          int k = ks0;
#pragma unroll
          for (int j = 0; j < 4; j++) c[j] = part_cols(p + 8 * (k + j < ke0 ? j : 0));
          for (;;) {
            w |= or_cols<T>(c[0]) | or_cols<T>(c[1]);
            if (k + 2 >= ke0 || (w | my) == full) break;
            if (k + 4 < ke0) {
              c[0] = part_cols(p + 32);
              c[1] = part_cols(p + (k + 5 < ke0 ? 40 : 32));
            }
            w |= or_cols<T>(c[2]) | or_cols<T>(c[3]);
            if (k + 4 >= ke0 || (w | my) == full) break;
            if (k + 6 < ke0) {
              c[2] = part_cols(p + 48);
              c[3] = part_cols(p + (k + 7 < ke0 ? 56 : 48));
            }
            k += 4;
            p += 32;
          }
          got = w;
        }
        if (base + lane < np) N[base + lane] = (T)(got & ~my);
      }
    }
    __syncthreads();
    // fold: each thread the vertices it owns, four at a time
    int ldone = 0;
    for (int base = wib * 32; base < np; base += 4 * kThreads) {
      unsigned nw[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int u = base + j * kThreads + lane;
        // written by atomics after a push: not through L1
        nw[j] = u < np ? (unsigned)*static_cast<const volatile T*>(N + u) : 0u;
      }
      uint32_t m[4];
      int tot = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int u = base + j * kThreads + lane;
        if (nw[j]) {
          const unsigned all = V[u] | nw[j];
          V[u] = (T)all;
          ldone += all == full;
          if (L >= kPartDeep)
            for (unsigned x = nw[j]; x; x &= x - 1) dist[(size_t)(__ffs(x) - 1) * np + u] = L;
        }
        m[j] = __ballot_sync(kFull, nw[j] != 0);
        tot += __popc(m[j]);
      }
      if (tot == 0) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&sh.nf, tot);
      at = __shfl_sync(kFull, at, 0);
      if (at >= listed) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int p = at + __popc(m[j] & lanemask_lt());
        if (nw[j] && p < listed) list[p] = base + j * kThreads + lane;
        at += __popc(m[j]);
      }
    }
    ldone = __reduce_add_sync(kFull, ldone);
    if (lane == 0 && ldone) atomicAdd(&sh.done, ldone);
    if (push) t_push++; else t_pull++;
    __syncthreads();
  }
  t_levels += (u64)(L - 1);
  const int deepest = L - 2;  // the last level run found nothing
  const int last = min(deepest, kPartDeep - 1);
  const bool deep = deepest >= kPartDeep;
  for (int u = tid; u < np; u += kThreads) {
    const unsigned vis = V[u];
    const int od = __ldg(row_ptr + v0 + u + 1) - __ldg(row_ptr + v0 + u);
    unsigned w[4] = {0u, 0u, 0u, 0u}, any = 0u;
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      if (h > last) break;
      unsigned x[8];  // the words of eight levels, loaded together
#pragma unroll
      for (int l = 0; l < 8; l++) x[l] = h + l >= 1 && h + l <= last ? (unsigned)words[(size_t)(h + l) * pitch + u] : 0u;
#pragma unroll
      for (int l = 0; l < 8; l++) {
        any |= x[l];
        if (l & 1) w[0] |= x[l];
        if (l & 2) w[1] |= x[l];
        if (l & 4) w[2] |= x[l];
        if (h) w[3] |= x[l];
      }
    }
    const unsigned here = deep ? any : vis;  // pairs to write a level for
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] |= ~here;
    my_reached += (u64)od * (u64)__popc(vis);
    emit_small_vertex(dist + u, np, nb, vis, w, deep);
  }
  // a source's own pair is in no word: with deep levels the loop left it out
  if (deep && tid < nb) dist[(size_t)tid * np + src[tid]] = 0;
}

// slot: this CTA's global scratch: kPartDeep + 1 word arrays of word_bytes
// each (the first unused), then the vertex list.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads)
    parts_small(PartsCtl* __restrict__ ctl, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                const int32_t* __restrict__ t_off, const uint16_t* __restrict__ t_col,
                const int32_t* __restrict__ voff, unsigned char* __restrict__ scratch, size_t slot_bytes,
                size_t word_bytes) {
  __shared__ PartShared sh;
  unsigned char* const slot = scratch + (size_t)blockIdx.x * slot_bytes;
  int32_t* const list = reinterpret_cast<int32_t*>(slot + (1 + kPartDeep) * word_bytes);
  u64 my_reached = 0, t_levels = 0, t_push = 0, t_pull = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sh.task = atomicAdd(&ctl->next_task, 1);
    __syncthreads();
    const int t = sh.task;
    if (t >= ctl->ntasks) break;
    const PartTask task = ctl->tasks[t];
    const int32_t v0 = voff[task.part];
    const int np = voff[task.part + 1] - v0;
    if (task.bits == 32)
      small_task<uint32_t, kThreads>(ctl, task, sh, reinterpret_cast<uint32_t*>(slot), word_bytes / 4, list, row_ptr, col, t_off,
                                     t_col, v0, np, my_reached, t_levels, t_push, t_pull);
    else
      small_task<uint16_t, kThreads>(ctl, task, sh, reinterpret_cast<uint16_t*>(slot), word_bytes / 2, list, row_ptr, col, t_off,
                                     t_col, v0, np, my_reached, t_levels, t_push, t_pull);
  }
  my_reached = warp_sum(my_reached);
  if (lane_id() == 0 && my_reached) atomicAdd(&ctl->reached, my_reached);
  if (threadIdx.x == 0 && t_levels) {
    atomicAdd(&ctl->levels, t_levels);
    atomicAdd(&ctl->push_levels, t_push);
    atomicAdd(&ctl->pull_levels, t_pull);
  }
}

// Block-diagonal check: every column of a part's rows lies in that part.
__global__ void __launch_bounds__(kBlock) parts_check(const int32_t* __restrict__ row_ptr,
                                                      const int32_t* __restrict__ col,
                                                      const int32_t* __restrict__ voff, int32_t nparts,
                                                      int* __restrict__ flag) {
  const int32_t p = blockIdx.y * gridDim.x + blockIdx.x;
  if (p >= nparts) return;
  const int32_t lo = voff[p], hi = voff[p + 1];
  const int k0 = row_ptr[lo], k1 = row_ptr[hi];
  int bad = 0;
  for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
    const int32_t c = col[k];
    bad |= c < lo || c >= hi;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

// Pieces of eight per in-row, for the scan that places the padded rows.
__global__ void __launch_bounds__(kBlock) parts_pieces(const int32_t* __restrict__ t_row_ptr, int32_t n,
                                                       int64_t* __restrict__ out) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v <= (size_t)n; v += stride)
    out[v] = v < (size_t)n ? (t_row_ptr[v + 1] - t_row_ptr[v] + 7) / 8 : 0;
}

// In-rows as part-local 16-bit ids, padded to pieces of eight with the id one
// past the part's vertices (ids of larger parts are cut off and never read).
// Eight lanes per row.
__global__ void __launch_bounds__(kBlock) parts_local_cols(const int32_t* __restrict__ t_row_ptr,
                                                           const int32_t* __restrict__ t_col,
                                                           const int32_t* __restrict__ voff, int32_t nparts,
                                                           const int64_t* __restrict__ off,
                                                           int32_t* __restrict__ t_off, uint16_t* __restrict__ out) {
  const int32_t p = blockIdx.y * gridDim.x + blockIdx.x;
  if (p >= nparts) return;
  const int32_t lo = voff[p], hi = voff[p + 1];
  const int sub = threadIdx.x & 7;
  for (int32_t v = lo + (int32_t)((threadIdx.x + blockIdx.z * blockDim.x) >> 3); v < hi;
       v += (int32_t)((blockDim.x * gridDim.z) >> 3)) {
    const int rs = t_row_ptr[v], deg = t_row_ptr[v + 1] - rs;
    const int64_t o = off[v];
    if (sub == 0) t_off[v] = (int32_t)o;
    for (int k = sub; k < ((deg + 7) & ~7); k += 8)
      out[8 * o + k] = (uint16_t)((k < deg ? t_col[rs + k] : hi) - lo);
    if (v + 1 == hi && p + 1 == nparts && sub == 0) t_off[hi] = (int32_t)off[hi];
  }
}

// Row-pointer values at the part boundaries (edge positions of each part).
__global__ void parts_bounds(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ voff, int32_t count,
                             long long* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) out[i] = row_ptr[voff[i]];
}

// Per (part, source) row: sum of the hop distances of the reached vertices
// other than the source, and their count.  One CTA per row.
__global__ void __launch_bounds__(kBlock) parts_row_sums(const int32_t* __restrict__ dist,
                                                         const PartRow* __restrict__ rows, int32_t nrows,
                                                         long long* __restrict__ sum,
                                                         long long* __restrict__ cnt) {
  __shared__ long long s_sum, s_cnt;
  for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
    if (threadIdx.x == 0) {
      s_sum = 0;
      s_cnt = 0;
    }
    __syncthreads();
    const PartRow row = rows[r];
    const int32_t* d = dist + row.off;
    long long ls = 0, lc = 0;
    for (int v = threadIdx.x; v < row.len; v += blockDim.x) {
      const int32_t x = d[v];
      if (x > 0) {
        ls += x;
        lc++;
      }
    }
    ls = (long long)warp_sum((u64)ls);
    lc = (long long)warp_sum((u64)lc);
    if (lane_id() == 0 && lc) {
      atomicAdd(reinterpret_cast<u64*>(&s_sum), (u64)ls);
      atomicAdd(reinterpret_cast<u64*>(&s_cnt), (u64)lc);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      sum[r] = s_sum;
      cnt[r] = s_cnt;
    }
    __syncthreads();
  }
}

}  // namespace

namespace {

const void* small_kernel(int threads) {
  return threads == 256 ? (const void*)parts_small<256>
                        : (threads == 512 ? (const void*)parts_small<512> : (const void*)parts_small<1024>);
}

// Widest words (32 or 16 bits) with which a part of np vertices fits
// `bytes` of shared memory; 0: none, or its ids need more than 16 bits.
int small_bits(int64_t np, size_t bytes) {
  if (np > 65535) return 0;
  for (int bits = 32; bits >= 16; bits /= 2)
    if (((size_t)np + 1) * (size_t)(bits / 8) + 16 <= bytes) return bits;
  return 0;
}

// Launch shape, columns and scratch of the single-CTA tasks.  Small parts run as
// smaller CTAs, more of them per SM, with the SM's memory shared out.  Until it
// has succeeded, no part counts as small (pt_small_smem is 0).
dawn_status small_slots(dawn_graph* g) {
  g->pt_small_smem = 0;
  int optin = 0;
  DAWN_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device));
  const size_t all = ((size_t)optin - 1024) & ~(size_t)127;
  const size_t widest = sizeof(uint32_t) * ((size_t)g->pt_maxn + 1) + 16;
  int threads = 1024;
  size_t smem = all;
  if (widest <= all / 4 - 1024) {
    threads = 256;
    smem = (all / 4 - 1024) & ~(size_t)127;
  } else if (widest <= all / 2 - 1024) {
    threads = 512;
    smem = (all / 2 - 1024) & ~(size_t)127;
  }
  size_t word_bytes = 16;
  int32_t listed = 1;
  for (size_t p = 0; p + 1 < g->pt_off.size(); p++) {
    const int32_t np = g->pt_off[p + 1] - g->pt_off[p];
    const int bits = small_bits(np, smem);
    if (!bits) continue;
    word_bytes = std::max(word_bytes, ((size_t)np * (size_t)(bits / 8) + 15) & ~(size_t)15);
    listed = std::max(listed, np);
  }
  const void* fn = small_kernel(threads);
  DAWN_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)all));
  DAWN_CUDA(cudaFuncSetAttribute(small_kernel(1024), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)all));
  g->pt_small_threads = threads;
  g->pt_small_ctas = persistent_blocks(fn, threads, smem);
  g->pt_small_words = word_bytes;
  g->pt_small_slot = ((1 + kPartDeep) * word_bytes + sizeof(int32_t) * ((size_t)listed / 8 + 64) + 127) & ~(size_t)127;
  DAWN_CHECK(ensure(g->pt_small, g->pt_small_slot * (size_t)g->pt_small_ctas, g->stream));
  const int32_t nparts = (int32_t)g->pt_off.size() - 1;
  const size_t n1 = (size_t)g->n + 1;
  // a row of d entries takes at most d / 8 + 1 pieces
  DAWN_CHECK(ensure(g->pt_tcol, sizeof(uint16_t) * ((size_t)g->m + 8 * n1), g->stream));
  DAWN_CHECK(ensure(g->pt_toff, sizeof(int32_t) * n1, g->stream));
  int64_t* tmp = nullptr;
  DAWN_CHECK(pool_alloc((void**)&tmp, sizeof(int64_t) * 2 * n1, g->stream));
  parts_pieces<<<g->geo.sms * 8, kBlock, 0, g->stream>>>(g->t_row_ptr, g->n, tmp);
  dawn_status s = exclusive_scan_i64(tmp, tmp + n1, (int64_t)n1, g->stream);
  if (s == DAWN_OK) {
    const int gx = std::min(nparts, 65535);
    parts_local_cols<<<dim3(gx, (nparts + gx - 1) / gx, 8), kBlock, 0, g->stream>>>(
        g->t_row_ptr, g->t_col, g->pt_voff.as<int32_t>(), nparts, tmp + n1, g->pt_toff.as<int32_t>(),
        g->pt_tcol.as<uint16_t>());
  }
  pool_free(tmp, g->stream);
  DAWN_CHECK(s);
  DAWN_CUDA(cudaGetLastError());
  g->pt_small_smem = smem;
  return DAWN_OK;
}

// Launch shape and scratch of the cluster tasks, on their first use.
dawn_status cluster_slots(dawn_graph* g) {
  if (g->pt_cluster_ready) return DAWN_OK;
  const int32_t maxn = g->pt_maxn;
  // Per-cluster slots: visited, two frontiers, accumulator and one slice
  // per level bit (levels never exceed the part's vertex count).  The grid
  // is as many clusters as the device holds at once.
  const int nbits = 32 - __builtin_clz((unsigned)maxn);
  const size_t slot_words = (size_t)(4 + nbits) * (size_t)maxn;
  int cluster = kPartCluster, clusters = 0;
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kPartCluster);
    cfg.blockDim = dim3(kPartBlock);
    if (cudaOccupancyMaxActiveClusters(&clusters, (const void*)parts_traverse<kPartCluster>, &cfg) != cudaSuccess ||
        clusters < 1) {
      // no room for clusters of kPartCluster CTAs (a small partition of the
      // device): one CTA per task, one per SM
      cudaGetLastError();
      cluster = 1;
      clusters = g->geo.sms;
    }
  }
  const int slots = clusters * cluster;  // CTAs of the grid
  const size_t bytes = sizeof(u64) * slot_words * (size_t)clusters;
  if (g->pt_scratch.bytes < bytes) {
    DAWN_CHECK(ensure(g->pt_scratch, bytes, g->stream));
    if (g->pt_exec) {
      cudaGraphExecDestroy(g->pt_exec);
      g->pt_exec = nullptr;
    }
  }
  // Slots are clean between calls: each task zeroes what it used.
  DAWN_CUDA(cudaMemsetAsync(g->pt_scratch.p, 0, bytes, g->stream));
  if (g->pt_exec && (g->pt_slots != slots || g->pt_slot_words != slot_words || g->pt_exec_maxn != maxn ||
                     g->pt_cluster != cluster)) {
    cudaGraphExecDestroy(g->pt_exec);
    g->pt_exec = nullptr;
  }
  g->pt_slots = slots;
  g->pt_cluster = cluster;
  g->pt_slot_words = slot_words;
  g->pt_exec_maxn = maxn;
  g->pt_cluster_ready = true;
  return DAWN_OK;
}

// Uploads offsets, reads the edge positions there and checks that no edge leaves
// its part.  Waits for the stream.
dawn_status read_parts(dawn_graph* g, int32_t nparts, const int32_t* offsets, DevBuf& voff,
                       std::vector<long long>& pos) {
  const size_t count = (size_t)nparts + 1;
  DAWN_CHECK(ensure(voff, sizeof(int32_t) * count, g->stream));
  DAWN_CUDA(cudaMemcpyAsync(voff.p, offsets, sizeof(int32_t) * count, cudaMemcpyHostToDevice, g->stream));
  long long* d_pos = nullptr;  // and the flag behind them
  DAWN_CHECK(pool_alloc((void**)&d_pos, sizeof(long long) * (count + 1), g->stream));
  pos.assign(count + 1, 0);
  int* const d_flag = reinterpret_cast<int*>(d_pos + count);
  cudaError_t e = cudaMemsetAsync(d_flag, 0, sizeof(long long), g->stream);
  parts_bounds<<<((int)count + kBlock - 1) / kBlock, kBlock, 0, g->stream>>>(g->row_ptr, voff.as<int32_t>(), (int)count,
                                                                            d_pos);
  if (!(g->flags & DAWN_GRAPH_NO_VALIDATE)) {
    const int gx = std::min(nparts, 65535);
    const int gy = (nparts + gx - 1) / gx;
    parts_check<<<dim3(gx, gy), kBlock, 0, g->stream>>>(g->row_ptr, g->col, voff.as<int32_t>(), nparts, d_flag);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(pos.data(), d_pos, sizeof(long long) * (count + 1), cudaMemcpyDeviceToHost, g->stream);
  pool_free(d_pos, g->stream);
  DAWN_CUDA(e);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  const bool leaves = pos.back() != 0;
  pos.pop_back();
  if (leaves) {
    set_error("parts: an edge leaves its part (the graph is not the disjoint union the offsets describe)");
    return DAWN_ERR_INVALID_ARG;
  }
  return DAWN_OK;
}

}  // namespace

dawn_status parts_set(dawn_graph* g, int32_t nparts, const int32_t* offsets) {
  if (nparts < 1 || !offsets) {
    set_error("parts: need nparts >= 1 and an offsets array of nparts + 1 entries");
    return DAWN_ERR_INVALID_ARG;
  }
  if (offsets[0] != 0 || offsets[nparts] != g->n) {
    set_error("parts: offsets must start at 0 and end at n = %d", g->n);
    return DAWN_ERR_INVALID_ARG;
  }
  int32_t maxn = 0;
  for (int32_t p = 0; p < nparts; p++) {
    const int32_t np = offsets[p + 1] - offsets[p];
    if (np < 1) {
      set_error("parts: part %d is empty or the offsets decrease", p);
      return DAWN_ERR_INVALID_ARG;
    }
    maxn = std::max(maxn, np);
  }
  if (maxn > kPartMaxVertices) {
    set_error("parts: a part of %d vertices exceeds the per-part limit of %d; traverse it as its own graph",
              maxn, kPartMaxVertices);
    return DAWN_ERR_INVALID_ARG;
  }
  // The parts that a handle has stay as they are until the new ones are known to
  // hold.
  DevBuf voff;
  std::vector<long long> pos;
  const dawn_status read = read_parts(g, nparts, offsets, voff, pos);
  if (read != DAWN_OK) {
    release(voff);
    return read;
  }
  release(g->pt_voff);
  g->pt_voff = voff;
  g->pt_pos.swap(pos);
  g->pt_off.assign(offsets, offsets + nparts + 1);
  g->pt_maxn = maxn;
  g->pt_cluster_ready = false;
  if (g->pt_exec) {  // it holds the earlier parts' addresses and sizes
    cudaGraphExecDestroy(g->pt_exec);
    g->pt_exec = nullptr;
  }
  const dawn_status small = small_slots(g);
  if (small == DAWN_ERR_OOM) {  // then every part is a cluster's
    cudaGetLastError();
    clear_error();
    for (DevBuf* b : {&g->pt_small, &g->pt_tcol, &g->pt_toff}) release(*b);
  } else {
    DAWN_CHECK(small);
  }
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  return DAWN_OK;
}

namespace {

// The cluster tasks of the uploaded control block, one persistent launch.
dawn_status run_clusters(dawn_graph* g) {
  DAWN_CHECK(cluster_slots(g));
  PartsCtl* ctl = g->pt_ctl.as<PartsCtl>();
  const int32_t* voff = g->pt_voff.as<int32_t>();
  u64* scratch = g->pt_scratch.as<u64>();
  size_t slot_words = g->pt_slot_words;
  int32_t maxn = g->pt_maxn;
  const bool capturable = g->stream != nullptr && g->stream != cudaStreamLegacy && g->stream != cudaStreamPerThread;
  if (!g->pt_exec && g->graphs_ok && capturable) {
    // One persistent launch, captured once per handle and replayed: every
    // per-call value travels in the control block.
    cudaGraph_t graph = nullptr;
    cudaStream_t cs = g->stream;
    DAWN_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    (g->pt_cluster == kPartCluster ? parts_traverse<kPartCluster> : parts_traverse<1>)<<<g->pt_slots, kPartBlock, 0, cs>>>(ctl, g->row_ptr, g->col, g->t_row_ptr, g->t_col, voff, scratch,
                                                  slot_words, maxn);
    const cudaError_t le = cudaGetLastError();
    const cudaError_t ce = cudaStreamEndCapture(cs, &graph);
    if (le != cudaSuccess || ce != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      set_error("parts: capture failed: %s", cudaGetErrorString(le != cudaSuccess ? le : ce));
      return DAWN_ERR_CUDA;
    }
    const cudaError_t ie = cudaGraphInstantiate(&g->pt_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
      g->pt_exec = nullptr;
      set_error("parts: graph instantiation failed: %s", cudaGetErrorString(ie));
      return DAWN_ERR_CUDA;
    }
  }
  if (g->pt_exec) {
    DAWN_CUDA(cudaGraphLaunch(g->pt_exec, g->stream));
  } else {
    (g->pt_cluster == kPartCluster ? parts_traverse<kPartCluster> : parts_traverse<1>)<<<g->pt_slots, kPartBlock, 0, g->stream>>>(ctl, g->row_ptr, g->col, g->t_row_ptr, g->t_col, voff,
                                                         scratch, slot_words, maxn);
    DAWN_CUDA(cudaGetLastError());
  }
  return DAWN_OK;
}

}  // namespace

dawn_status parts_bfs(dawn_graph* g, const int32_t* source_offset, const int32_t* sources, int32_t* d_dist,
                      std::vector<PartRow>* rows_out, dawn_stats* st) {
  const int32_t nparts = (int32_t)g->pt_off.size() - 1;
  if (nparts < 1) {
    set_error("parts: the graph has no parts (dawn_graph_set_parts)");
    return DAWN_ERR_INVALID_ARG;
  }
  if (!source_offset || source_offset[0] != 0) {
    set_error("parts: source_offset must have nparts + 1 entries starting at 0");
    return DAWN_ERR_INVALID_ARG;
  }
  const std::vector<int32_t>& off = g->pt_off;
  long long out = 0;
  std::vector<long long> out0(nparts);
  int32_t batches = 0;
  for (int32_t p = 0; p < nparts; p++) {
    const int32_t s0 = source_offset[p], s1 = source_offset[p + 1];
    const int32_t np = off[p + 1] - off[p];
    if (s1 < s0) {
      set_error("parts: source_offset decreases at part %d", p);
      return DAWN_ERR_INVALID_ARG;
    }
    for (int32_t i = s0; i < s1; i++)
      if (sources[i] < 0 || sources[i] >= np) {
        set_error("parts: source %d of part %d is outside [0, %d)", sources[i], p, np);
        return DAWN_ERR_INVALID_ARG;
      }
    if (rows_out)
      for (int32_t i = s0; i < s1; i++) rows_out->push_back(PartRow{out + (long long)(i - s0) * np, np, p});
    out0[p] = out;
    out += (long long)(s1 - s0) * np;
    batches += (s1 - s0 + 63) / 64;
  }
  if (st) std::memset(st, 0, sizeof(*st));
  if (batches == 0) return DAWN_OK;
  // Tasks.  A part whose words fit one SM's shared memory is cut into tasks of
  // as many sources as its widest words hold, or of fewer where the tasks
  // would not cover the CTAs; larger parts, and every part of a traced call,
  // go 64 sources per cluster task.
  const std::vector<long long>& pos = g->pt_pos;
  std::vector<PartTask> small, tasks;
  auto cut = [&](int32_t most) {
    small.clear();
    tasks.clear();
    for (int32_t p = 0; p < nparts; p++) {
      const int32_t s0 = source_offset[p], ns = source_offset[p + 1] - s0, np = off[p + 1] - off[p];
      const int bits = g->trace || most == 0 ? 0 : small_bits(np, g->pt_small_smem);
      const int32_t c = bits ? std::min(bits, most) : 64;
      const int32_t k = (ns + c - 1) / c;
      for (int32_t j = 0; j < k; j++) {
        // single-CTA tasks share the sources evenly
        const int32_t i = bits ? (int32_t)((long long)ns * j / k) : j * c;
        const int32_t e = bits ? (int32_t)((long long)ns * (j + 1) / k) : std::min(ns, i + c);
        PartTask t;
        t.part = p;
        t.src0 = s0 + i;
        t.nsrc = e - i;
        t.bits = bits ? std::min(bits, t.nsrc <= 16 ? 16 : 32) : 0;
        t.out0 = out0[p] + (long long)i * np;
        (bits ? small : tasks).push_back(t);
      }
    }
  };
  // Microseconds of a cut's tasks on the whole device.  Fitted: a single-CTA
  // task (491 of them) 37 + 6.0 per 1,000 vertices + 0.12 per 1,000 entries
  // + 0.19 per 1,000 distances, a cluster task 70 + 0.25 per 1,000 entries,
  // 16 at a time.  Few large parts are the clusters' (8 parts of 1,000 to
  // 65,536 vertices: 300 us against 477), many or small ones single CTAs'
  // (300 such parts: 1,635 against 5,083).
  auto estimate = [&]() {
    double sum = 0, most = 0, csum = 0, cmost = 0;
    for (const PartTask& t : small) {
      const double np = off[t.part + 1] - off[t.part], mp = (double)(pos[t.part + 1] - pos[t.part]);
      const double us = 37 + 6.0e-3 * np + 0.12e-3 * mp + 0.19e-3 * np * t.nsrc;
      sum += us;
      most = std::max(most, us);
    }
    for (const PartTask& t : tasks) {
      const double us = 70 + 0.25e-3 * (double)(pos[t.part + 1] - pos[t.part]);
      csum += us;
      cmost = std::max(cmost, us);
    }
    const double s_us = (int)small.size() <= g->geo.sms ? most : sum / g->geo.sms + 0.3 * most;
    return s_us + std::max(cmost, csum / 16);
  };
  cut(32);
  if (!small.empty() && small.size() < 4 * (size_t)g->geo.sms) {
    int32_t best = 32;
    double us = estimate();
    for (int32_t most : {16, 8, 0}) {
      cut(most);
      const double x = estimate();
      if (x < us) {
        us = x;
        best = most;
      }
    }
    cut(best);
  }
  // Longest tasks first, so they start while the grid is full.  Measured
  // on 512 random parts (the per-task trace), a cluster task takes about
  // levels x (n + m / 60) time units: the per-level sweep of the part's
  // vertices costs far more than its edges.  A random part of n vertices
  // and average degree d is about ln n / ln d + 3 ln n / d levels deep
  // (correlation 0.98 with the traced depths).  Single-CTA tasks follow the
  // same rule (fitted over 491 of them: 8.5 us per 1,000 vertices, 0.04 per
  // 1,000 entries).
  std::vector<double> cost(nparts);
  for (int32_t p = 0; p < nparts; p++) {
    const double np = (double)(off[p + 1] - off[p]), mp = (double)(pos[p + 1] - pos[p]);
    const double d = np > 0 ? std::max(2.0, mp / np) : 2.0;
    const double ln = std::log(std::max(np, 2.0));
    cost[p] = (np + mp / 60.0) * std::max(1.0, ln / std::log(d) + 3.0 * ln / d);
  }
  auto longest = [&](const PartTask& a, const PartTask& b) { return cost[a.part] > cost[b.part]; };
  std::stable_sort(tasks.begin(), tasks.end(), longest);
  std::stable_sort(small.begin(), small.end(), longest);
  // One upload: the two control blocks, the tasks, the sources.
  const int32_t nsrc = source_offset[nparts];
  const size_t o_tasks = 2 * sizeof(PartsCtl);
  const size_t o_src = o_tasks + sizeof(PartTask) * (small.size() + tasks.size());
  const size_t up_bytes = o_src + sizeof(int32_t) * (size_t)nsrc;
  const void* const ctl_before = g->pt_ctl.p;
  DAWN_CHECK(ensure(g->pt_ctl, up_bytes, g->stream));
  if (g->pt_exec && g->pt_ctl.p != ctl_before) {  // the captured launch holds the old address
    cudaGraphExecDestroy(g->pt_exec);
    g->pt_exec = nullptr;
  }
  unsigned char* const dev = g->pt_ctl.as<unsigned char>();
  PartsCtl c = {};
  c.push_ratio = g->bs_push_ratio;
  c.sources = reinterpret_cast<const int32_t*>(dev + o_src);
  c.dist = d_dist;
  unsigned long long* d_log = nullptr;
  if (g->trace) {
    DAWN_CHECK(pool_alloc((void**)&d_log, sizeof(unsigned long long) * 4 * tasks.size(), g->stream));
    c.task_log = d_log;
  }
  std::vector<unsigned char> up(up_bytes);
  c.ntasks = (int32_t)tasks.size();
  c.tasks = reinterpret_cast<const PartTask*>(dev + o_tasks) + small.size();
  std::memcpy(up.data(), &c, sizeof(c));
  c.ntasks = (int32_t)small.size();
  c.tasks = reinterpret_cast<const PartTask*>(dev + o_tasks);
  std::memcpy(up.data() + sizeof(c), &c, sizeof(c));
  if (!small.empty()) std::memcpy(up.data() + o_tasks, small.data(), sizeof(PartTask) * small.size());
  if (!tasks.empty())
    std::memcpy(up.data() + o_tasks + sizeof(PartTask) * small.size(), tasks.data(), sizeof(PartTask) * tasks.size());
  std::memcpy(up.data() + o_src, sources, sizeof(int32_t) * (size_t)nsrc);
  // pageable: staged before the call returns
  DAWN_CUDA(cudaMemcpyAsync(dev, up.data(), up_bytes, cudaMemcpyHostToDevice, g->stream));

  if (!small.empty()) {
    PartsCtl* sctl = g->pt_ctl.as<PartsCtl>() + 1;
    const int32_t *rp = g->row_ptr, *cl = g->col, *trp = g->pt_toff.as<int32_t>(), *vo = g->pt_voff.as<int32_t>();
    const uint16_t* tcl = g->pt_tcol.as<uint16_t>();
    unsigned char* scr = g->pt_small.as<unsigned char>();
    void* args[] = {&sctl, &rp, &cl, &trp, &tcl, &vo, &scr, &g->pt_small_slot, &g->pt_small_words};
    // tasks that have an SM to themselves take all of its threads
    const int threads = (int)small.size() <= g->geo.sms ? 1024 : g->pt_small_threads;
    DAWN_CUDA(cudaLaunchKernel(small_kernel(threads), dim3(std::min(g->pt_small_ctas, (int)small.size())),
                               dim3(threads), args, g->pt_small_smem, g->stream));
  }
  if (!tasks.empty()) DAWN_CHECK(run_clusters(g));
  if (d_log) {
    // one trace record per task: device-clock start and duration
    std::vector<unsigned long long> h(4 * tasks.size());
    DAWN_CUDA(cudaMemcpyAsync(h.data(), d_log, sizeof(unsigned long long) * h.size(), cudaMemcpyDeviceToHost,
                              g->stream));
    pool_free(d_log, g->stream);
    DAWN_CUDA(cudaStreamSynchronize(g->stream));
    unsigned long long t0 = ~0ull;
    for (size_t i = 0; i < tasks.size(); i++) t0 = std::min(t0, h[4 * i]);
    for (size_t i = 0; i < tasks.size(); i++) {
      dawn_trace_rec r = {};
      std::snprintf(r.kernel, sizeof(r.kernel), "parts_task");
      const int p = tasks[i].part;
      r.run = p;
      r.level = (int32_t)(h[4 * i + 2] >> 32);
      r.mode = (int32_t)(h[4 * i + 2] & 0xffffffffu);
      r.pad = (int32_t)h[4 * i + 3];
      r.frontier = tasks[i].nsrc;
      r.frontier_edges = g->pt_pos[p + 1] - g->pt_pos[p];
      r.unvisited_edges = (int64_t)(h[4 * i] - t0);
      r.ms = (float)((double)(h[4 * i + 1] - h[4 * i]) * 1e-6);
      g->trace_log.push_back(r);
    }
  }
  if (st) {
    PartsCtl h[2];
    DAWN_CUDA(cudaMemcpyAsync(h, g->pt_ctl.p, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
    DAWN_CUDA(cudaStreamSynchronize(g->stream));
    st->edges_traversed = (int64_t)(h[0].reached + h[1].reached);
    st->levels = (int32_t)(h[0].levels + h[1].levels);
    st->push_levels = (int32_t)(h[0].push_levels + h[1].push_levels);
    st->pull_levels = (int32_t)(h[0].pull_levels + h[1].pull_levels);
    st->batches = batches;
  }
  return DAWN_OK;
}

dawn_status parts_row_reduce(dawn_graph* g, const int32_t* d_dist, const std::vector<PartRow>& rows,
                             long long* h_sum, long long* h_cnt) {
  if (rows.empty()) return DAWN_OK;
  const size_t nr = rows.size();
  DAWN_CHECK(ensure(g->pt_rows, sizeof(PartRow) * nr, g->stream));
  DAWN_CHECK(ensure(g->cc_out, 2 * sizeof(long long) * nr, g->stream));
  DAWN_CUDA(cudaMemcpyAsync(g->pt_rows.p, rows.data(), sizeof(PartRow) * nr, cudaMemcpyHostToDevice, g->stream));
  long long* d_sum = g->cc_out.as<long long>();
  long long* d_cnt = d_sum + nr;
  const int grid = (int)std::min<size_t>(nr, (size_t)g->geo.sms * 8);
  parts_row_sums<<<grid, kBlock, 0, g->stream>>>(d_dist, g->pt_rows.as<PartRow>(), (int32_t)nr, d_sum, d_cnt);
  DAWN_CUDA(cudaGetLastError());
  DAWN_CUDA(cudaMemcpyAsync(h_sum, d_sum, sizeof(long long) * nr, cudaMemcpyDeviceToHost, g->stream));
  DAWN_CUDA(cudaMemcpyAsync(h_cnt, d_cnt, sizeof(long long) * nr, cudaMemcpyDeviceToHost, g->stream));
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  return DAWN_OK;
}

}  // namespace dawn
