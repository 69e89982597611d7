// Ordered min-plus relaxation (near-far) in one persistent launch, on
// sm_103a: weighted distances of one source, or of a batch of up to 64.
//
// The level-by-level traversals (govm.cu, msssp.cu) relax a vertex again
// every time its distance improves: on a mesh of 200,000 points a (vertex,
// source) pair improves 15 times on average, and one source on RMAT scale
// 22 relaxes 2.5 m entries.  Here a pair is relaxed only once its distance
// is at most a threshold T; pairs beyond it wait in a far list.  When the
// near list runs empty, T rises by a step and the far list is scanned: pairs
// whose distance is now within T move to the near list, pairs that were
// relaxed meanwhile are dropped.  Any relaxation order reaches the same
// fixed point, so the distances are those of the level-by-level forms.
//
// Everything between the first fill and the last relaxation is one
// cooperative launch, because a mesh takes 500 to 1,500 steps of a few
// thousand pairs, and a step of two or three launches in a conditional graph
// costs 12 us and more before it does any work.  A phase (fill, mark, seed,
// near, far) ends when its participating CTAs have checked in; the last one
// decides the next phase and how many CTAs it takes, and publishes both in
// words that all CTAs poll.  A short near list is then a matter of a few
// CTAs and a short arrival count, while the others only watch the words; a
// near list of a few hundred pairs is one CTA's, phase after phase, with the
// lists in shared memory.
//
// What bounds it: on meshes the chain of dependent L2 round trips of a phase
// (list entry, row bounds, targets, their distances, list reservation,
// arrival: 6 to 7 us, 1.6 us within one CTA); on RMAT the gather of a
// target's distance per entry, 100 to 140 G entries/s in the large phases
// against the 230 G/s of the L1/TEX sector rate.  Times per call, before
// (level by level) and now, float32, on one GPU in turn, from the fastest to the
// slowest of three sources (source lists):
//   kNN mesh, 200,003 points, 50 sources     55.9-57.2 -> 10.2-10.5 ms
//   RMAT scale 22, one source                1.90-2.32 -> 1.87-2.00 ms (real-valued lengths 2.55 -> 2.0-2.2)
//   grid 1000 x 1049, one source             24.0-29.1 -> 9.9-12.4 ms
//   kNN mesh, 20,000 points, one source      1.41-1.64 -> 0.88-1.04 ms
//   RMAT scale 12 (edge factor 8), one       143-163 -> 131-141 us
// Slower than cluster levels were (one launch for many small levels): one source on
// meshes of 20,000 to 90,000 vertices whose levels hold 500 to 1,500 pairs, a phase of
// 6.8 us each (grid 200 x 200 by a tenth, a street network of 62,500 by a quarter).
#include <algorithm>
#include <cstring>

#include "dawn_device.cuh"

namespace dawn {

namespace {

// 16 warps, two CTAs per SM: 64 registers leave room for the loads of three
// or four entries per lane in flight (768 threads at 40 registers, one entry
// at a time: RMAT scale 22 2.12 ms against 1.94).
constexpr int kNfBlock = 512;
constexpr int kShortUnroll = 3;  // groups of 32 entries of short rows in flight per warp
constexpr int kNfWarps = kNfBlock / 32;
constexpr int kNfEntries = 256;  // vertices and entries per CTA of a small graph (512 the same, 1024: kNN of 2,127 8% slower)

enum : int32_t { kPhFill = 0, kPhMark, kPhSeed, kPhNear, kPhFar };

// What the CTAs poll: four words of one 32-byte sector, each tagged with the
// phase's generation in its top 16 bits, so that one load per lane brings
// everything a phase needs to start and a torn read shows in the tags.
//   word 0: CTAs of the phase (16 bits; 0: finished) << 32 | near or far entries read
//   word 1: phase << 40 | near list read << 33 | far list appended to << 32 | near segments read
//   word 2: the near threshold T
//   word 3: the threshold before (far scans)
constexpr int kTag = 48;
constexpr unsigned long long kTallyMask = (1ull << 40) - 1;

struct __align__(128) NfCtl {
  unsigned long long word[4];
  unsigned pad0[24];
  // Counters of the phase with generation g at index g & 3; the last CTA of
  // phase g clears those of g + 2.
  struct __align__(128) {
    unsigned long long tally;  // CTAs that finished << 40 | near entries written
    unsigned long long lpack;  // near long rows written: (rows << 32) | segments
  } cnt[4];
  struct __align__(128) {
    int32_t n[2];              // entries of the two far lists
    uint32_t min_far;          // smallest distance left by the running far scan
    uint32_t delta;            // threshold step (float bits for float weights)
    uint32_t iters;            // near phases of this launch
    uint32_t bucket_iters;     // near phases since T last rose, and the pairs they read
    unsigned long long bucket_pairs;
  } far;
};

// Near list of a single-CTA phase.
constexpr int kSoloMax = 640, kSoloCap = 1024;
// At the graph's mean degree: one SM relaxes about 1,900 entries in the time of a
// phase on the grid (grid 120 x 150: 640 pairs 1005 us, 480 899, 160 1044; kNN of
// 2,127 points: 310 pairs 451 us, 190 405, 60 416).
constexpr double kSoloEntries = 1920.0;
struct Solo {
  uint32_t p[kSoloCap];
  int32_t rs[kSoloCap], deg[kSoloCap];
};

struct NfArgs {
  const int32_t *row_ptr, *col, *w;
  int32_t* D;              // distances: n << shift
  NfCtl* ctl;
  int32_t* queue;          // near lists 0, 1, far lists 0, 1: cap entries each
  Seg* segs;               // near long-row segments 0, 1: segcap entries each
  uint32_t* masks;         // near bits 0, 1, far bits: nwords words each
  size_t cap, segcap, nwords;
  const int32_t* sources;  // the batch's first source
  int32_t nb;              // sources (1..64)
  int32_t n, shift;
  uint32_t inf, delta, delta_min, delta_max;
  int32_t has_long;        // some row has at least kLongRow entries
  uint32_t solo_max;       // pairs of a single-CTA phase
  int32_t* levels_out;     // of the call's control block: levels, push levels
  int32_t* push_out;
  uint32_t polls;          // of one wait
  int32_t* err;            // pinned host word
};

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Distances and weights are non-negative, as int32 or as float bits; both
// order like unsigned words, and an int32 sum past INT32_MAX compares above
// every distance instead of wrapping below it.
template <bool kFloat>
__device__ __forceinline__ uint32_t nf_add(uint32_t a, uint32_t b) {
  if (kFloat) return __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
  return a + b;
}

template <bool kFloat>
__device__ __forceinline__ uint32_t nf_threshold(uint32_t t, uint32_t step, uint32_t inf) {
  const uint32_t x = nf_add<kFloat>(t, step);
  return x < inf ? x : inf - 1;  // a pair at `inf` is unreached and never queued
}

// The step follows the near lists: half as long again after a bucket whose
// phases read fewer than kNearLow pairs (all waiting, no work) or that took at
// most two phases (the step is short against the weights, so nothing is
// relaxed twice), three quarters of it after phases of more than kNearHigh
// pairs, where a pair relaxed twice costs more than a phase.
constexpr unsigned long long kNearLow = 4096, kNearHigh = 131072;

template <bool kFloat>
__device__ __forceinline__ uint32_t nf_scale(uint32_t d, bool up, uint32_t lo, uint32_t hi) {
  uint32_t x;
  if (kFloat)
    x = __float_as_uint(__uint_as_float(d) * (up ? 1.5f : 0.75f));
  else
    x = up ? d + (d + 1) / 2 : d - d / 4;
  return x < lo ? lo : (x > hi ? hi : x);
}

// CTAs for `entries`, at most per_cta each (near phases: two pairs per warp,
// so that a short list spreads over many warps but its arrivals stay few).
__device__ __forceinline__ uint32_t nf_ctas(uint32_t entries, uint32_t per_cta) {
  const uint32_t a = (entries + per_cta - 1) / per_cta;
  return a < 1 ? 1 : (a > gridDim.x ? gridDim.x : a);
}

// A phase as every CTA sees it.
struct Phase {
  uint32_t ctas, n;  // participating CTAs (0: finished), entries read
  uint32_t segs;     // near segments read
  uint32_t T, t_old;
  int32_t kind, in, fcur;
};

__device__ __forceinline__ Phase unpack(unsigned long long w0, unsigned long long w1, unsigned long long w2,
                                        unsigned long long w3) {
  Phase p;
  p.ctas = (uint32_t)(w0 >> 32) & 0xffffu;
  p.n = (uint32_t)w0;
  p.kind = (int32_t)(w1 >> 40) & 0xff;
  p.in = (int32_t)(w1 >> 33) & 1;
  p.fcur = (int32_t)(w1 >> 32) & 1;
  p.segs = (uint32_t)w1;
  p.T = (uint32_t)w2;
  p.t_old = (uint32_t)w3;
  return p;
}

// Run by one thread of the last CTA to finish phase p (generation g), which
// wrote `nn` near entries: every other participant has arrived and the rest
// only watch the words, so nothing else touches the control block.  Decides
// the next phase; returns false when the traversal is finished.
template <bool kFloat>
__device__ __forceinline__ bool nf_control(const NfArgs& a, uint32_t g, uint32_t nn, Phase& p) {
  NfCtl* c = a.ctl;
  const uint32_t ns = a.has_long ? (uint32_t)__ldcg(&c->cnt[g & 3].lpack) : 0u;
  if (p.kind == kPhFill || p.kind == kPhMark) {
    p.kind++;
    p.ctas = gridDim.x;
  } else if (nn | ns) {
    p.in = p.kind == kPhSeed ? 1 : p.in ^ 1;
    p.kind = kPhNear;
    p.n = nn;
    p.segs = ns;
    p.ctas = ns == 0 && nn <= a.solo_max ? 1 : nf_ctas(nn + 2 * ns, kNfWarps * 2);
    atomicAdd(&c->far.iters, 1u);
    atomicAdd(&c->far.bucket_iters, 1u);
    atomicAdd(&c->far.bucket_pairs, (unsigned long long)nn + 4ull * ns);
  } else {
    const uint32_t far_n = (uint32_t)__ldcg(&c->far.n[p.fcur]);
    if (far_n == 0) {
      const int32_t iters = (int32_t)__ldcg(&c->far.iters);
      *a.levels_out += iters;
      *a.push_out += iters;
      return false;
    }
    uint32_t delta = __ldcg(&c->far.delta);
    p.t_old = p.T;
    const bool scanned = p.kind == kPhFar;
    if (scanned) {
      // the scan moved nothing: step past the gap
      p.T = nf_threshold<kFloat>(__ldcg(&c->far.min_far), delta, a.inf);
    } else {
      const uint32_t iters = __ldcg(&c->far.bucket_iters);
      const unsigned long long pairs = __ldcg(&c->far.bucket_pairs);
      if (iters) {
        if (pairs < kNearLow * iters || iters <= 2) delta = nf_scale<kFloat>(delta, true, a.delta_min, a.delta_max);
        else if (pairs > kNearHigh * iters) delta = nf_scale<kFloat>(delta, false, a.delta_min, a.delta_max);
        c->far.delta = delta;
      }
      p.T = nf_threshold<kFloat>(p.T, delta, a.inf);
    }
    c->far.bucket_iters = 0;
    c->far.bucket_pairs = 0;
    c->far.n[p.fcur ^ 1] = 0;
    c->far.min_far = 0xffffffffu;
    p.in = p.kind == kPhSeed ? 0 : p.in;
    p.kind = kPhFar;
    p.fcur ^= 1;
    p.n = far_n;
    p.ctas = nf_ctas(far_n, kNfBlock);
    // Every pair that a scan leaves lies above T and below `inf`, so T rises past
    // it; a launch in which it does not would never end.  (After a near list T may
    // stay where it is: a step below its rounding.)
    if (scanned && p.T <= p.t_old) {
      *a.err = DAWN_ERR_TIMEOUT;
      p.ctas = 0;
    }
  }
  c->cnt[(g + 2) & 3].tally = 0;
  c->cnt[(g + 2) & 3].lpack = 0;
  return true;
}

// One bit per pair id, in flat bitmaps.
__device__ __forceinline__ bool set_pair(uint32_t* masks, uint32_t p) {
  const uint32_t bit = 1u << (p & 31);
  return !(atomicOr(masks + (p >> 5), bit) & bit);
}
__device__ __forceinline__ void clear_pair(uint32_t* masks, uint32_t p) {
  atomicAnd(masks + (p >> 5), ~(1u << (p & 31)));
}

// Per-warp staging of list appends (WarpQueueT with the list's length in a
// word whose upper bits hold something else).
template <class Count>
struct PairQueue {
  int32_t* buf;
  int32_t* out;
  Count* count;
  int n = 0;

  __device__ __forceinline__ PairQueue(int32_t* sbuf, int32_t* q, Count* cnt) : buf(sbuf), out(q), count(cnt) {}

  __device__ __forceinline__ void drain(uint32_t base) {
    for (int i = lane_id(); i < n; i += 32) out[(size_t)base + i] = buf[i];
    n = 0;
  }
  __device__ __forceinline__ void push(bool pred, int32_t v) {
    const uint32_t m = __ballot_sync(kFull, pred);
    if (m == 0) return;
    const int c = __popc(m);
    if (n + c > kWarpQueue) {
      uint32_t base = 0;
      if (lane_id() == 0) base = (uint32_t)(atomicAdd(count, (Count)n) & (Count)kTallyMask);
      base = __shfl_sync(kFull, base, 0);
      __syncwarp();
      drain(base);
      __syncwarp();
    }
    if (pred) buf[n + __popc(m & lanemask_lt())] = v;
    n += c;
  }
};

// A pair id is (vertex << shift) + source, and the index of its distance.
template <bool kFloat>
__global__ void __launch_bounds__(kNfBlock, 2) nf_traverse(const __grid_constant__ NfArgs a) {
  __shared__ int32_t s_near[kNfWarps][kWarpQueue], s_far[kNfWarps][kWarpQueue];
  __shared__ uint32_t s_nn[kNfWarps], s_nf[kNfWarps];
  __shared__ unsigned long long s_word[4];
  __shared__ Solo s_solo[2];
  __shared__ int2 s_cl[3];  // lists of three phases in a row: entries, and whether a long row is among them
  const int shift = a.shift;
  const uint32_t smask = (1u << shift) - 1u;
  NfCtl* const ctl = a.ctl;
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  const size_t tid = blockIdx.x * (size_t)kNfBlock + threadIdx.x, nthreads = (size_t)gridDim.x * kNfBlock;
  uint32_t* const far_mask = a.masks + 2 * a.nwords;

  // fill: every CTA, before its first arrival (the control block is zero)
  uint32_t gen = 0;
  if (tid == 0) ctl->far.delta = a.delta;
  {
    const size_t words = (size_t)a.n << shift;
    if ((reinterpret_cast<uintptr_t>(a.D) & 15) == 0 && (words & 3) == 0) {
      int4* d4 = reinterpret_cast<int4*>(a.D);
      const int x = (int)a.inf;
      for (size_t i = tid; i < words / 4; i += nthreads) d4[i] = make_int4(x, x, x, x);
    } else {
      for (size_t i = tid; i < words; i += nthreads) a.D[i] = (int)a.inf;
    }
    for (size_t i = tid; i < 3 * a.nwords; i += nthreads) a.masks[i] = 0u;
  }

  Phase ph = {};
  ph.ctas = gridDim.x;
  ph.kind = kPhFill;
  ph.T = nf_threshold<kFloat>(0u, a.delta, a.inf);
  for (;;) {
    // check in; the last participant opens the next phase
    __syncthreads();
    if (wib == 0) {
      if (lane == 0) {
        __threadfence();
        const unsigned long long t = atomicAdd(&ctl->cnt[gen & 3].tally, kTallyMask + 1);
        if ((uint32_t)(t >> 40) == ph.ctas - 1) {
          __threadfence();
          Phase nx = ph;
          const bool more = nf_control<kFloat>(a, gen, (uint32_t)(t & kTallyMask), nx);
          const unsigned long long tag = (unsigned long long)((gen + 1) & 0xffffu) << kTag;
          __threadfence();
          volatile unsigned long long* w = ctl->word;
          w[0] = tag | (unsigned long long)(more ? nx.ctas : 0u) << 32 | nx.n;
          w[1] = tag | (unsigned long long)nx.kind << 40 | (unsigned long long)nx.in << 33 |
                 (unsigned long long)nx.fcur << 32 | nx.segs;
          w[2] = tag | nx.T;
          w[3] = tag | nx.t_old;
        }
      }
      // wait for a phase that this CTA takes part in
      __syncwarp();
      bool idle = false;
      for (uint32_t polls = 0;; polls++) {
        const unsigned long long w = ld_acquire(&ctl->word[lane & 3]);
        const uint32_t tag = (uint32_t)(w >> kTag), tag0 = __shfl_sync(kFull, tag, 0);
        if (__all_sync(kFull, tag == tag0) && tag != gen) {
          gen = tag;
          polls = 0;
          const uint32_t ctas = (uint32_t)(__shfl_sync(kFull, w, 0) >> 32) & 0xffffu;
          if (ctas == 0 || blockIdx.x < ctas) {
            if (lane < 4) s_word[lane] = w;
            break;
          }
          idle = true;
        }
        if (polls == a.polls) {
          if (lane == 0) {
            *a.err = DAWN_ERR_TIMEOUT;
            s_word[0] = 0;
          }
          break;
        }
        if (idle) __nanosleep(64);
      }
    }
    __syncthreads();
    ph = unpack(s_word[0], s_word[1], s_word[2], s_word[3]);
    if (ph.ctas == 0) return;
    gen = (uint32_t)(s_word[0] >> kTag);
    const int phase = ph.kind;
    const uint32_t T = ph.T;
    const int slot = ph.in;  // the near list read
    const int out = phase == kPhNear || phase == kPhFar ? slot ^ 1 : 1;
    const int fcur = ph.fcur;
    uint32_t* const near_out = a.masks + (size_t)out * a.nwords;
    Seg* const seg_out = a.segs + (size_t)out * a.segcap;
    unsigned long long* const lpack = &ctl->cnt[gen & 3].lpack;
    PairQueue<unsigned long long> wn(s_near[wib], a.queue + (size_t)out * a.cap, &ctl->cnt[gen & 3].tally);
    PairQueue<int32_t> wf(s_far[wib], a.queue + (size_t)(2 + fcur) * a.cap, &ctl->far.n[fcur]);

    // queues a pair for the next near phase: long rows as segments
    auto emit_near = [&](bool is, uint32_t p) {
      if (!a.has_long) {
        wn.push(is, (int32_t)p);
        return;
      }
      int rs = 0, deg = 0;
      if (is) {
        rs = __ldg(a.row_ptr + (p >> shift));
        deg = __ldg(a.row_ptr + (p >> shift) + 1) - rs;
      }
      const bool is_long = is && deg >= kLongRow;
      wn.push(is && !is_long, (int32_t)p);
      const uint32_t lm = __ballot_sync(kFull, is_long);
      if (lm) {
        const int nseg = is_long ? (deg + kSeg - 1) / kSeg : 0;
        const int incl = warp_incl_scan(nseg);
        const int tot = __shfl_sync(kFull, incl, 31);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(lpack, ((unsigned long long)__popc(lm) << 32) | (unsigned)tot);
        write_segments(lm, (int32_t)p, rs, nseg, (uint32_t)__shfl_sync(kFull, base, 0) + incl - nseg, seg_out);
      }
    };
    // Relaxes CSR entry k[i] from distance d[i] for source s[i] (ok[i]), kU
    // entries per lane: the loads of each stage are issued for all of them
    // before the first is waited on.
    auto relax = [&](auto& k, auto& ok, auto& d, auto& src) {
      constexpr int kU = sizeof(k) / sizeof(k[0]);
      uint32_t pu[kU], c[kU];
#pragma unroll
      for (int i = 0; i < kU; i++) {
        pu[i] = ok[i] ? ((uint32_t)__ldg(a.col + k[i]) << shift) | src[i] : 0u;
        c[i] = ok[i] ? (uint32_t)__ldg(a.w + k[i]) : 0u;
      }
      uint32_t cur[kU];
#pragma unroll
      for (int i = 0; i < kU; i++) cur[i] = ok[i] ? (uint32_t)__ldcg(a.D + pu[i]) : 0u;
#pragma unroll
      for (int i = 0; i < kU; i++) {
        c[i] = nf_add<kFloat>(d[i], c[i]);
        const bool less = c[i] < cur[i];  // never without ok: cur is 0 there
        if (!__any_sync(kFull, less)) continue;
        bool near = false, far = false;
        if (less) {
          atomicMin(reinterpret_cast<uint32_t*>(a.D) + pu[i], c[i]);
          if (c[i] <= T)
            near = set_pair(near_out, pu[i]);
          else
            far = set_pair(far_mask, pu[i]);
        }
        emit_near(near, pu[i]);
        wf.push(far, (int32_t)pu[i]);
      }
    };
    // one row or segment of a pair, swept by the whole warp
    auto sweep = [&](int k0, int k1, uint32_t dist, uint32_t s, auto& op) {
      for (int kb = k0; kb < k1; kb += 128) {
        int k[4];
        bool ok[4];
        uint32_t d[4], src[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          k[i] = kb + 32 * i + lane;
          ok[i] = k[i] < k1;
          d[i] = dist;
          src[i] = s;
        }
        op(k, ok, d, src);
      }
    };
    // the rows of up to 32 pairs (lane i: pair p at distance d, row rs, deg;
    // deg = 0: none): rows of >= kWarpRow entries by the whole warp, shorter
    // ones concatenated and dealt 32 entries at a time
    auto expand = [&](uint32_t p, int rs, int deg, uint32_t d, auto& op) {
      uint32_t big = __ballot_sync(kFull, deg >= kWarpRow);
      while (big) {
        const int l = __ffs(big) - 1;
        big &= big - 1;
        const int s = __shfl_sync(kFull, rs, l), e = s + __shfl_sync(kFull, deg, l);
        const uint32_t ld = __shfl_sync(kFull, d, l), lp = __shfl_sync(kFull, p, l);
        sweep(s, e, ld, lp & smask, op);
      }
      const int sdeg = deg < kWarpRow ? deg : 0;
      const int incl = warp_incl_scan(sdeg);
      const int excl = incl - sdeg;
      const int total = __shfl_sync(kFull, incl, 31);
      for (int e0 = 0; e0 < total; e0 += 32 * kShortUnroll) {
        int k[kShortUnroll];
        bool ok[kShortUnroll];
        uint32_t ed[kShortUnroll], es[kShortUnroll];
#pragma unroll
        for (int j = 0; j < kShortUnroll; j++) {
          const int e = e0 + 32 * j + lane;
          int lo = 0;  // last lane whose offset is <= e
#pragma unroll
          for (int step = 16; step; step >>= 1) {
            const int ex = __shfl_sync(kFull, excl, lo + step);
            if (ex <= e) lo += step;
          }
          k[j] = __shfl_sync(kFull, rs, lo) + (e - __shfl_sync(kFull, excl, lo));
          ok[j] = e < total;
          ed[j] = __shfl_sync(kFull, d, lo);
          es[j] = __shfl_sync(kFull, p, lo) & smask;
        }
        op(k, ok, ed, es);
      }
    };

    if (phase == kPhNear && ph.ctas == 1 && ph.segs == 0 && ph.n <= a.solo_max) {
      // A few pairs: this CTA alone runs near phases one after another with
      // the lists in shared memory, one barrier per phase, until a list is
      // empty, too long, or holds a long row.  A pair pushed twice in a phase
      // is relaxed twice (no near bits here); the list left over is queued
      // as usual.
      uint32_t* const near_in = a.masks + (size_t)slot * a.nwords;
      const int32_t* qin = a.queue + (size_t)slot * a.cap;
      for (int i = threadIdx.x; i < (int)ph.n; i += kNfBlock) {
        const uint32_t p = (uint32_t)__ldcg(qin + i);
        const int rs = __ldg(a.row_ptr + (p >> shift));
        s_solo[0].p[i] = p;
        s_solo[0].rs[i] = rs;
        s_solo[0].deg[i] = __ldg(a.row_ptr + (p >> shift) + 1) - rs;
        clear_pair(near_in, p);
      }
      if (threadIdx.x == 0) {
        s_cl[0] = make_int2((int)ph.n, 0);
        s_cl[1] = s_cl[2] = make_int2(0, 0);
      }
      __syncthreads();
      int left = 0, it = 0;
      for (;; it++) {
        const int cnt = s_cl[it % 3].x;
        const Solo& in = s_solo[it & 1];
        Solo& nx = s_solo[(it & 1) ^ 1];
        int32_t* const nx_cnt = &s_cl[(it + 1) % 3].x;
        if (threadIdx.x == 0) s_cl[(it + 2) % 3] = make_int2(0, 0);
        auto push = [&](auto& k, auto& ok, auto& d, auto& src) {
          constexpr int kU = sizeof(k) / sizeof(k[0]);
          uint32_t pu[kU], c[kU];
#pragma unroll
          for (int i = 0; i < kU; i++) {
            pu[i] = ok[i] ? ((uint32_t)__ldg(a.col + k[i]) << shift) | src[i] : 0u;
            c[i] = ok[i] ? (uint32_t)__ldg(a.w + k[i]) : 0u;
          }
          uint32_t old[kU];
          int rs[kU], re[kU];
#pragma unroll
          for (int i = 0; i < kU; i++) {
            c[i] = nf_add<kFloat>(d[i], c[i]);
            old[i] = ok[i] ? atomicMin(reinterpret_cast<uint32_t*>(a.D) + pu[i], c[i]) : 0u;
            rs[i] = ok[i] ? __ldg(a.row_ptr + (pu[i] >> shift)) : 0;
            re[i] = ok[i] ? __ldg(a.row_ptr + (pu[i] >> shift) + 1) : 0;
          }
#pragma unroll
          for (int i = 0; i < kU; i++) {
            const bool less = c[i] < old[i];
            if (!__any_sync(kFull, less)) continue;
            const uint32_t m = __ballot_sync(kFull, less && c[i] <= T);
            int base = 0;
            if (m && lane == 0) base = atomicAdd(nx_cnt, __popc(m));
            base = __shfl_sync(kFull, base, 0) + __popc(m & lanemask_lt());
            const bool near = (m >> lane) & 1u;
            if (near && base < kSoloCap) {
              nx.p[base] = pu[i];
              nx.rs[base] = rs[i];
              nx.deg[base] = re[i] - rs[i];
              if (re[i] - rs[i] >= kLongRow) nx_cnt[1] = 1;
            }
            bool over = near && base >= kSoloCap;
            if (over) over = set_pair(near_out, pu[i]);
            emit_near(over, pu[i]);
            bool far = less && !near;
            if (far) far = set_pair(far_mask, pu[i]);
            wf.push(far, (int32_t)pu[i]);
          }
        };
        int per = 32;
        while (per > 1 && (per >> 1) * kNfWarps >= cnt) per >>= 1;
        for (int b = wib * per; b < cnt; b += kNfWarps * per) {
          const int i = b + lane;
          const bool ok = lane < per && i < cnt;
          const uint32_t p = ok ? in.p[i] : 0u;
          expand(p, ok ? in.rs[i] : 0, ok ? in.deg[i] : 0, ok ? (uint32_t)__ldcg(a.D + p) : 0u, push);
        }
        __syncthreads();
        // a warp that goes on writes the next phase's words, not these
        left = *nx_cnt;
        if (left == 0 || left > (int)a.solo_max || nx_cnt[1] || it + 1 == kSoloSteps) break;
      }
      if (threadIdx.x == 0 && it > 0) {
        atomicAdd(&ctl->far.iters, (uint32_t)it);
        atomicAdd(&ctl->far.bucket_iters, (uint32_t)it);
      }
      const Solo& rest = s_solo[(it & 1) ^ 1];
      const int n = min(left, kSoloCap);
      for (int b = wib * 32; b < n; b += kNfBlock) {
        const int i = b + lane;
        const uint32_t p = i < n ? rest.p[i] : 0u;
        const bool first = i < n && set_pair(near_out, p);
        emit_near(first, p);
      }
    } else if (phase == kPhNear) {
      uint32_t* const near_in = a.masks + (size_t)slot * a.nwords;
      const int nw = (int)ph.ctas * kNfWarps, gw = wib * (int)ph.ctas + (int)blockIdx.x;
      const Seg* sin = a.segs + (size_t)slot * a.segcap;
      const int ns = (int)ph.segs, nn = (int)ph.n;
      for (int i = gw; i < ns; i += nw) {
        const uint32_t p = (uint32_t)__ldcg(&sin[i].v);
        const int k0 = __ldcg(&sin[i].k0);
        const int rs = __ldg(a.row_ptr + (p >> shift)), re = __ldg(a.row_ptr + (p >> shift) + 1);
        const uint32_t d = (uint32_t)__ldcg(a.D + p);
        if (lane == 0 && k0 == rs) clear_pair(near_in, p);
        const int k1 = min(k0 + kSeg, re);
        sweep(k0, k1, d, p & smask, relax);
      }
      int per = 32;
      while (per > 1 && (long long)(per >> 1) * nw >= nn) per >>= 1;
      const int32_t* qin = a.queue + (size_t)slot * a.cap;
      for (int b = gw * per; b < nn; b += nw * per) {
        const int i = b + lane;
        uint32_t p = 0, d = 0;
        int rs = 0, deg = 0;
        if (lane < per && i < nn) {
          p = (uint32_t)__ldcg(qin + i);
          rs = __ldg(a.row_ptr + (p >> shift));
          deg = __ldg(a.row_ptr + (p >> shift) + 1) - rs;
          d = (uint32_t)__ldcg(a.D + p);
          clear_pair(near_in, p);
        }
        expand(p, rs, deg, d, relax);
      }
    } else if (phase == kPhFar) {
      // pairs within the raised threshold move to the near list; those at
      // or below the old one were relaxed since they were put here
      const uint32_t t_old = ph.t_old;
      const int fn = (int)ph.n;
      const int32_t* fin = a.queue + (size_t)(2 + (fcur ^ 1)) * a.cap;
      uint32_t least = 0xffffffffu;
      const int stride = (int)ph.ctas * kNfBlock;
      for (int b = (int)blockIdx.x * kNfBlock + wib * 32; b < fn; b += stride) {
        const int i = b + lane;
        bool near = false, keep = false;
        uint32_t p = 0;
        if (i < fn) {
          p = (uint32_t)__ldcg(fin + i);
          const uint32_t d = (uint32_t)__ldcg(a.D + p);
          keep = d > T;
          near = !keep && d > t_old;
          if (keep) {
            least = min(least, d);
          } else {
            clear_pair(far_mask, p);
            if (near) set_pair(near_out, p);
          }
        }
        emit_near(near, p);
        wf.push(keep, (int32_t)p);
      }
      least = __reduce_min_sync(kFull, least);
      if (lane == 0 && least != 0xffffffffu) atomicMin(&ctl->far.min_far, least);
    } else {
      // The source rows, as the reference CPU path reads them
      // (src/algorithm/cpu/sssp.cpp:41-46): each distinct neighbour takes the
      // weight of its last CSR entry.  Mark: entry k lowers the neighbour's
      // word to -(k + 1); seed: the surviving entry writes its weight and
      // queues the pair, the source itself gets 0 (and is queued only
      // through a self loop).  CTA c works on source c % nb.
      const int b = (int)blockIdx.x % a.nb, grp = (int)blockIdx.x / a.nb;
      const int ngrp = ((int)gridDim.x - b + a.nb - 1) / a.nb;
      for (int sb = b; sb < a.nb; sb += gridDim.x) {  // more than one round only on a grid smaller than nb
        const int32_t s = a.sources[sb];
        const int rs = __ldg(a.row_ptr + s), re = __ldg(a.row_ptr + s + 1);
        const int step = ngrp * kNfBlock;
        for (int k0 = rs + grp * kNfBlock + wib * 32; k0 < re; k0 += step) {
          const int k = k0 + lane;
          const int32_t u = k < re ? __ldg(a.col + k) : 0;
          const uint32_t p = ((uint32_t)u << shift) | (uint32_t)sb;
          if (phase == kPhMark) {
            if (k < re) atomicMin(a.D + p, -(k + 1));
            continue;
          }
          const bool win = k < re && __ldcg(a.D + p) == -(k + 1);
          bool near = false, far = false;
          if (win) {
            const uint32_t d = u == s ? 0u : min((uint32_t)__ldg(a.w + k), a.inf);
            a.D[p] = (int32_t)d;
            if (d <= T)
              near = set_pair(near_out, p);
            else if (d < a.inf)  // a weight of `inf` reaches nothing, and no T covers it
              far = set_pair(far_mask, p);
          }
          emit_near(near, p);
          wf.push(far, (int32_t)p);
        }
        if (phase == kPhSeed && grp == 0 && threadIdx.x == 0) {
          const uint32_t p = ((uint32_t)s << shift) | (uint32_t)sb;
          if ((uint32_t)__ldcg(a.D + p) == a.inf) a.D[p] = 0;  // no self loop: no entry marked it
        }
      }
    }
    // One reservation per CTA and list for what its warps still hold: a
    // reservation per warp is 7,000 same-address atomics on the whole grid
    // (25 us for a phase of 20,000 pairs).
    if (lane == 0) {
      s_nn[wib] = (uint32_t)wn.n;
      s_nf[wib] = (uint32_t)wf.n;
    }
    __syncthreads();
    if (wib == 0) {
      const int x = lane < kNfWarps ? (int)s_nn[lane] : 0, y = lane < kNfWarps ? (int)s_nf[lane] : 0;
      const int ix = warp_incl_scan(x), iy = warp_incl_scan(y);
      const int tx = __shfl_sync(kFull, ix, 31), ty = __shfl_sync(kFull, iy, 31);
      uint32_t bx = 0, by = 0;
      if (lane == 0) {
        if (tx) bx = (uint32_t)(atomicAdd(wn.count, (unsigned long long)tx) & kTallyMask);
        if (ty) by = (uint32_t)atomicAdd(wf.count, ty);
      }
      bx = __shfl_sync(kFull, bx, 0);
      by = __shfl_sync(kFull, by, 0);
      if (lane < kNfWarps) {
        s_nn[lane] = bx + (uint32_t)(ix - x);
        s_nf[lane] = by + (uint32_t)(iy - y);
      }
    }
    __syncthreads();
    wn.drain(s_nn[wib]);
    wf.drain(s_nf[wib]);
  }
}

// Longest row and sum of a sample of the weights (at most 65,536 entries,
// evenly spaced).
struct NfShape {
  double weights;
  unsigned long long segs;
  int32_t max_deg, pad;
};
__global__ void __launch_bounds__(kBlock) nf_shape(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ w,
                                                   int is_float, int32_t n, long long m, int samples,
                                                   NfShape* __restrict__ out) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  unsigned deg = 0;
  unsigned long long segs = 0;
  for (int32_t v = tid; v < n; v += stride) {
    const int d = row_ptr[v + 1] - row_ptr[v];
    deg = max(deg, (unsigned)d);
    if (d >= kLongRow) segs += (d + kSeg - 1) / kSeg;
  }
  double sum = 0.0;
  for (int i = tid; i < samples; i += stride) {
    const int32_t x = w[(long long)i * m / samples];
    sum += is_float ? (double)__int_as_float(x) : (double)x;
  }
  deg = __reduce_max_sync(kFull, deg);
  segs = warp_sum(segs);
#pragma unroll
  for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
  if (lane_id() == 0) {
    if (deg) atomicMax(&out->max_deg, (int)deg);
    if (segs) atomicAdd(&out->segs, segs);
    if (sum != 0.0) atomicAdd(&out->weights, sum);
  }
}

// The shape of the handle's graph, read once.
dawn_status shape_of(dawn_graph* g) {
  if (g->nf_max_deg >= 0) return DAWN_OK;
  NfShape* d = nullptr;
  DAWN_CHECK(pool_alloc((void**)&d, sizeof(NfShape), g->stream));
  DAWN_CUDA(cudaMemsetAsync(d, 0, sizeof(NfShape), g->stream));
  const int samples = (int)std::min<int64_t>(g->m, 65536);
  nf_shape<<<g->geo.sms * 4, kBlock, 0, g->stream>>>(g->row_ptr, static_cast<const int32_t*>(g->val),
                                                      g->wtype == DAWN_W_F32, g->n, g->m, samples, d);
  DAWN_CUDA(cudaGetLastError());
  NfShape h;
  DAWN_CUDA(cudaMemcpyAsync(&h, d, sizeof(NfShape), cudaMemcpyDeviceToHost, g->stream));
  pool_free(d, g->stream);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  g->nf_mean_weight = samples ? h.weights / samples : 0.0;
  g->nf_segs = (int64_t)h.segs;
  g->nf_max_deg = h.max_deg;
  return DAWN_OK;
}

}  // namespace

// Pair ids are 32-bit, and the lists take 16 bytes per pair.
constexpr int64_t kNfMaxPairs = (int64_t)1 << 28;

int nearfar_shift(int32_t nb) {
  int shift = 0;
  while ((1 << shift) < nb) shift++;
  return shift == 1 ? 2 : shift;  // rows of at least 16 bytes in a batch
}

// Where the pairs beat the rows of msssp.cu.  The pairs cost 13 to 60 ps per entry
// and source, the more the less of the block fits L2; the rows have a price per
// entry that 64 sources pay as well as two, so the line lies in the sources beyond a
// few times the entries.  Measured, ms ordered / by rows, int32 lengths 1 to 63 (m:
// million entries):
//   hub, light stage:  RMAT-14 (0.4 m) 32 sources 0.67 / 0.77, 48 1.34 / 0.81; RMAT-16 (1.0)
//     16 0.69 / 0.87, 24 1.26 / 0.89; RMAT-18 (7.6) 4 0.69 / 0.90, 6 1.16 / 0.96;
//     RMAT-20 (15.7) 2 1.09 / 1.61, 4 1.88 / 1.81; RMAT-22 (128) 2 3.7 / 5.3, 4 6.2 / 5.8
//   hub, equal lengths: RMAT-18 16 1.00 / 1.32, 24 1.51 / 1.35; RMAT-20 16 2.35 / 2.25
//   no hub: Erdos-Renyi 300,000 x 8 32 1.96 / 2.68, 48 3.14 / 2.91; 1 M x 4 32 5.7 / 6.9,
//     48 11.9 / 8.0; 1 M x 12 24 8.7 / 8.7; 1 M x 22 16 6.0 / 9.6, 24 12.1 / 10.3; 2 M x 6 16
//     8.2 / 13.2, 24 16.2 / 14.4; 4 M x 16 16 37.4 / 37.8
//   meshes: kNN of 100,000, 64 sources 6.9 / 30.9; grid 300 x 300 5.7 / 34.7: the rows take
//     hundreds of levels, at any number of sources
// A graph of low degree without long rows is a mesh if it does not grow like a random
// one.
constexpr int64_t kNfLine = 72000000, kNfLightLine = 13000000;

dawn_status nearfar_batch_fits(dawn_graph* g, int32_t nsrc, bool* fits) {
  *fits = false;
  const int32_t nb = nsrc < 64 ? nsrc : 64;
  if ((int64_t)g->n << nearfar_shift(nb) > kNfMaxPairs) return DAWN_OK;
  DAWN_CHECK(shape_of(g));
  if ((double)g->nf_max_deg * g->n >= kHubDegree * (double)g->m) {
    if ((nb - 3) * g->m > kNfLightLine) DAWN_CHECK(light_weights(g));
    *fits = (nb - 3) * g->m <= kNfLightLine || (!g->light_pays && (nb - 12) * g->m <= kNfLine);
    return DAWN_OK;
  }
  *fits = (nb - 16) * g->m <= kNfLine;
  if (!*fits && g->nf_max_deg < kLongRow && g->m < 10 * (int64_t)g->n) {
    DAWN_CHECK(read_growth(g));
    *fits = g->growth < kGrows;
  }
  return DAWN_OK;
}

namespace {

// Lists, segments and masks of a traversal of nb sources.
struct NfSizes {
  size_t cap, segcap, nwords;
  NfSizes(const dawn_graph* g, int32_t nb, int shift)
      : cap((size_t)g->n * (size_t)nb),
        segcap(g->nf_max_deg >= kLongRow ? (size_t)g->nf_segs * (size_t)nb + 64 : 64),
        nwords((((size_t)g->n << shift) + 31) / 32) {}
};

}  // namespace

dawn_status nearfar_reserve(dawn_graph* g, int32_t nb, int shift) {
  DAWN_CHECK(shape_of(g));
  const NfSizes z(g, nb, shift);
  DAWN_CHECK(ensure(g->nf_ctl, sizeof(NfCtl), g->stream));
  DAWN_CHECK(ensure(g->nf_queue, sizeof(int32_t) * 4 * z.cap, g->stream));
  DAWN_CHECK(ensure(g->nf_segbuf, sizeof(Seg) * 2 * z.segcap, g->stream));
  DAWN_CHECK(ensure(g->nf_masks, sizeof(uint32_t) * 3 * z.nwords, g->stream));
  return DAWN_OK;
}

dawn_status nearfar_run(dawn_graph* g, const int32_t* d_sources, int32_t nb, int shift, int32_t* D,
                        int32_t* levels_out, int32_t* push_out) {
  DAWN_CHECK(nearfar_reserve(g, nb, shift));
  const NfSizes z(g, nb, shift);
  const bool fl = g->wtype == DAWN_W_F32;
  NfArgs a = {};
  a.row_ptr = g->row_ptr;
  a.col = g->col;
  a.w = static_cast<const int32_t*>(g->val);
  a.D = D;
  a.n = g->n;
  a.shift = shift;
  a.nb = nb;
  a.sources = d_sources;
  a.cap = z.cap;
  a.nwords = z.nwords;
  a.has_long = g->nf_max_deg >= kLongRow;
  a.segcap = z.segcap;
  // the arrival counts start at zero, also after a launch that gave up
  DAWN_CUDA(cudaMemsetAsync(g->nf_ctl.p, 0, sizeof(NfCtl), g->stream));
  a.ctl = g->nf_ctl.as<NfCtl>();
  a.queue = g->nf_queue.as<int32_t>();
  a.segs = g->nf_segbuf.as<Seg>();
  a.masks = g->nf_masks.as<uint32_t>();
  a.inf = fl ? 0x7f7fffffu : 0x7fffffffu;
  a.levels_out = levels_out;
  a.push_out = push_out;
  a.polls = g->wait_polls;
  a.err = g->h_err;
  // First step, in mean weights per mean out-degree.  A short step relaxes
  // few entries twice but takes more phases; which of the two costs more
  // depends on the work there is.  4 / 8 / 32 / 128: RMAT scale 22 2.14 /
  // 1.83 / 2.75 / 2.85 ms, kNN x 50 sources 10.1 / 10.0 / 10.5 / 13.4 ms; ER
  // (16M entries) 614 / 637 / 529 / 913 us; RMAT scale 12 190 / 160 / 146 /
  // 130 us, ER (160K entries) 194 / 184 / 151 / 135 us.  128 / 512: kNN of 2,127
  // points 406 / 363 us, grid 120 x 150 913 / 945, 10 sources there 1531 / 1387.
  const double work = (double)g->m * nb;
  const double kStep = work < 1 << 16 || (nb > 1 && work < 1 << 20) ? 512.0
                       : work < 1 << 20                               ? 128.0
                                                                      : (work < 1 << 24 ? 32.0 : 8.0);
  const double deg = g->m > 0 ? (double)g->m / (double)g->n : 1.0;
  a.solo_max = (uint32_t)std::min((double)kSoloMax, kSoloEntries / std::max(1.0, deg));
  const double step = kStep * g->nf_mean_weight / std::max(1.0, deg);
  const double lo = step / 2, hi = step * 16;
  auto bits = [&](double x) -> uint32_t {
    if (fl) {
      const float f = (float)std::min(x, 1e37);
      uint32_t u;
      std::memcpy(&u, &f, sizeof(u));
      return u;
    }
    return (uint32_t)std::max(1.0, std::min(x, 1e9));
  };
  a.delta = bits(step);
  a.delta_min = bits(lo);
  a.delta_max = bits(hi);
  const void* fn = fl ? (const void*)nf_traverse<true> : (const void*)nf_traverse<false>;
  void* args[] = {&a};
  // a small graph takes few CTAs: each adds to the arrivals of its phases
  const int64_t want = (int64_t)((double)(g->n + g->m) * nb / kNfEntries) + 1;
  const int full = persistent_blocks(fn, kNfBlock, 0, g->blocks_per_sm);
  const int ctas = want < full ? (int)want : full;
  DAWN_CUDA(cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(kNfBlock), args, 0, g->stream));
  return DAWN_OK;
}

}  // namespace dawn
