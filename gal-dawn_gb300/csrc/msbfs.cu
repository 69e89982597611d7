// Batched boolean expand over bitset frontiers on sm_103a.
//
// The reference runs multi-source and all-pairs BFS as a serial loop of
// single-source traversals (src/algorithm/gpu/mssp.cu:26-43,
// src/algorithm/gpu/apsp.cu:81-100), re-reading the whole CSR once per
// source.  Here up to 64*W sources share one traversal: every vertex carries
// W uint64 words per state (visited, frontier, next), bit b of word i
// standing for source 64*i + b of the batch, so one pass over an adjacency
// row serves all of them.  The W words of a vertex are contiguous, so a
// gather of a neighbour's frontier is one 8W-byte load (one 32-byte sector
// for W = 4).  Hop distances come out identical to separate traversals: a
// source's bit appears at a vertex at level L exactly when that source
// first reaches it at L.
//
// A level runs in one of two directions, chosen on the device:
//   pull: each unfinished vertex (some source has not reached it) ORs the
//         frontier words of its in-neighbours, stopping early once every
//         missing bit is found; the vertex owns its words, so no atomics.
//         Heavy rows are cut into segments combined by the last finisher;
//   push: the active vertices' rows are dealt to warps; new bits are
//         atomicOr-ed into `next`, and an update pass folds `next` into
//         visited / frontier (over the touched list, or densely for large
//         frontiers).
// Below level kDeepLevel neither writes distances: the level at which a bit
// first appears is recorded in bit-sliced level words (slice k holds bit k
// of the level of every (source, vertex) pair), and a final pass expands
// them into the distance block with full-line coalesced stores, writing -1
// for pairs never reached.  From kDeepLevel on (high-diameter graphs, whose
// vertices gain their bits one source at a time over thousands of levels) a
// new bit is written out directly instead: one store per (source, vertex)
// pair rather than a read-modify-write of every set bit's slice, and the
// final pass leaves those entries alone.
#include <algorithm>
#include <cstring>
#include <vector>

#include "dawn_device.cuh"
#include "selector.cuh"

namespace dawn {
namespace {

using u64 = unsigned long long;
constexpr int kMaxW = 4;

struct BsCtl {
  int32_t aq_size[3];           // active (frontier) list sizes, rotating by level % 3
  int32_t pad0;
  unsigned long long alpack[3]; // active long rows: (vertices << 32) | segments
  int32_t tq_size;              // push: vertices touched this level
  int32_t ul_size[2];           // unfinished-vertex lists (pull work lists)
  int32_t ul_cur;               // list the next pull reads: -1 = the graph's static list
  int32_t level;                // with depth: read together by level-mode callers
  int32_t depth[kMaxW];         // level mode: the deepest level of each 64 sources
  int32_t mode, done, policy, batch, nsrc, n_push, n_pull;
  int32_t push_ratio;           // push while push_ratio * frontier edges < unfinished edges
  int32_t work;                 // dynamic work counter of the current level (light rows)
  int32_t hwork;                // dynamic work counter of the heavy-row segments
  int32_t hs_size[2];           // heavy-segment task lists: segments of rows still unfinished
  int32_t hs_cur;               // list the next pull reads: -1 = every segment of the graph
  int32_t dense;                // push level: fire-and-forget scatter + dense update sweep
  int32_t nbits;                // level slices available
  int32_t width;                // W: words per vertex and state
  unsigned long long mf[3];     // out-degree sums of the active lists
  long long mu;                 // in-degree sum of vertices not yet finished
  long long mu_dec;             // in-degree of vertices finished this level
  unsigned long long reached;   // TEPS numerator of the batch
  unsigned long long full[kMaxW];  // this batch's source bits, less those of sources without out-edges
  int32_t* dist_base;
  const int32_t* sources;
  int32_t* lv_block;            // level mode: per 64 sources, their level block (else NULL)
  int32_t* lv_range;            // level mode: per 64 sources, lowest and highest level of every vertex
  unsigned long long* cc_sum;   // closeness mode: per source, sum of hop distances (else NULL)
  unsigned long long* cc_cnt;   // closeness mode: per source, vertices reached besides itself
  int32_t use_sel;              // decide with the handle's selector weights
  float sel_margin;             // log2 margin by which the selector must beat the heuristic
  int32_t force;                // 0 = decide per level; 1 + variant = always that variant
  int32_t prev_nf;              // frontier size entering the current level
  long long m;                  // CSR entries (selector input)
  unsigned long long total_reached;
  int32_t total_levels, total_push, total_pull;
  // 1 = the level that wrote this slot's frontier words kept no active list
  // (a dense push update: the next level is then a pull, which needs none,
  // and the slot is cleared densely when it goes stale); aq_size holds the
  // count only
  int32_t unlisted[3];
  // persistent launch: the words that all CTAs poll (BsStep), and the
  // arrivals of all phases so far
  struct __align__(128) {
    unsigned long long word[15];
    uint32_t broken;  // a wait of an earlier batch gave up: its arrivals are missing
  } sync;
  struct __align__(128) {
    uint32_t n;
  } arrive;
};

// What a CTA has to know to work on a level, from the control block (one
// launch per step) or from the words of the persistent launch: nine of 48
// bits, each tagged with the phase's generation in its top 16, so that one
// load per lane brings them all and a torn read shows in the tags.
struct BsStep {
  int32_t ctas, phase;
  uint32_t arrived;                           // arrivals before the phase
  int32_t L, dense;
  int32_t qn, ln;                             // frontier: listed vertices, long-row segments
  int32_t stale, stale_segs, stale_unlisted;  // the slot to clear
  int32_t tn;                                 // update: vertices touched
  int32_t ul_cur, un, hs_cur, hn;             // pull: the lists and their sizes
  int32_t nf;                                 // frontier vertices
};

struct BsArgs {
  BsCtl* ctl;
  const int32_t *row_ptr, *col, *t_row_ptr, *t_col;
  const int32_t *ul_static, *hv_static, *hv_segoff;  // pull lists of the graph
  u64 *words, *visit, *fr, *nxt, *slices;
  u64* hv_acc;
  int2* hv_tasks;
  int32_t *aq, *tq, *ul;
  uint32_t* tbm;
  Seg* segs;
  size_t segcap, nwords;
  long long m;
  int32_t n, ul_static_size, hv_count, hv_segs, pull_seg;
  int32_t nbits, force;
  int32_t batch;                // -1: the control block's (one launch per step)
  // where levels from kDeepLevel on go, as in the control block
  int32_t *dist_base, *lv_block;
  unsigned long long* cc_sum;
  const float* sel_w;
  uint32_t polls;               // persistent launch: of one wait
  int32_t* err;                 // pinned host word
};

constexpr int kSlicesCleared = 4;  // slices zeroed per batch; higher ones on first use
// Pull rows below this many in-edges are walked by one lane each; longer
// ones are swept by the whole warp.  Packing short rows across the lanes
// (a warp scan, a shared-memory search and a shared-memory OR per edge)
// measured 4-10% slower: the pull is bound by its L1/TEX traffic, and the
// lane walk adds none beyond the column loads and the gathers.
constexpr int kPullLaneMax = 64;
constexpr int kShallowBits = 5;    // level slices kept: the bits of levels below kDeepLevel
static_assert(kDeepLevel == 1 << kShallowBits, "slices hold exactly the levels below kDeepLevel");
// Heavy pull rows: a row of at least 2 x seg in-edges (seg = the handle's
// pull segment, 1024 by default) is cut into seg-entry warp tasks.

// Words per heavy-row accumulator: W bits and a finished-segment counter,
// rounded up to an even count so the W words start 16-byte aligned for
// the vectorised loads.
__host__ __device__ constexpr int acc_stride(int w) { return (w + 2) & ~1; }

__device__ __forceinline__ u64 warp_or64(u64 x) {
  const unsigned lo = __reduce_or_sync(kFull, (unsigned)x);
  const unsigned hi = __reduce_or_sync(kFull, (unsigned)(x >> 32));
  return ((u64)hi << 32) | lo;
}

// 32 x 32 bit transpose across a warp: lane i holds row i on entry and
// column i on exit (bit j of lane i's result = bit i of lane j's input).
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x) {
  const int lane = lane_id();
  const uint32_t left[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int t = 0; t < 5; t++) {
    const int s = 16 >> t;
    const uint32_t y = __shfl_xor_sync(kFull, x, s);
    x = (lane & s) ? ((x & ~left[t]) | ((y & ~left[t]) >> s)) : ((x & left[t]) | ((y & left[t]) << s));
  }
  return x;
}

// *p |= x without waiting for the old value.  As a reduction by name: beside an
// atomicOr whose result is used, the compiler makes one returning atomic of both
// (the dense scatter of RMAT-22 then takes 224 us, not 164; a call for 500 sources
// on RMAT-18 763, not 720).
__device__ __forceinline__ void or_word(u64* p, u64 x) {
  asm volatile("red.relaxed.gpu.global.or.b64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}

// W words of one vertex.
template <int W>
struct Bits {
  u64 w[W];
  __device__ __forceinline__ static Bits zero() {
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = 0ull;
    return b;
  }
  __device__ __forceinline__ static Bits full_of(const BsCtl* ctl) {
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = ctl->full[i];
    return b;
  }
  // Vectorised loads: W = 2 is one 16-byte load, W = 4 one 32-byte load
  // (a gather then asks L1/TEX for its sector once, not twice).  The
  // vertex's words start on a 32-byte boundary: slots are n x 32 bytes
  // apart from an aligned base.
  // Not through the read-only path: in the persistent launch the words of a
  // level were written earlier in the same launch.
  __device__ __forceinline__ static Bits gather(const u64* p) {
    Bits b;
    if constexpr (W == 4) {
      asm volatile("ld.global.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(b.w[0]), "=l"(b.w[1]), "=l"(b.w[2]), "=l"(b.w[3])
                   : "l"(p));
    } else if constexpr (W == 1) {
      asm volatile("ld.global.u64 %0, [%1];" : "=l"(b.w[0]) : "l"(p));
    } else {
      asm volatile("ld.global.v2.u64 {%0,%1}, [%2];" : "=l"(b.w[0]), "=l"(b.w[1]) : "l"(p));
    }
    return b;
  }
  __device__ __forceinline__ static Bits ldcg(const u64* p) {
    Bits b;
    if (W == 1) {
      b.w[0] = __ldcg(p);
    } else {
#pragma unroll
      for (int i = 0; i < W; i += 2) {
        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p + i));
        b.w[i] = v.x;
        b.w[i + 1] = v.y;
      }
    }
    return b;
  }
  __device__ __forceinline__ static Bits ld(const u64* p) {
    Bits b;
    if (W == 1) {
      b.w[0] = *p;
    } else {
#pragma unroll
      for (int i = 0; i < W; i += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + i);
        b.w[i] = v.x;
        b.w[i + 1] = v.y;
      }
    }
    return b;
  }
  __device__ __forceinline__ void st(u64* p) const {
    if (W == 1) {
      *p = w[0];
    } else {
#pragma unroll
      for (int i = 0; i < W; i += 2) *reinterpret_cast<ulonglong2*>(p + i) = make_ulonglong2(w[i], w[i + 1]);
    }
  }
  __device__ __forceinline__ Bits operator|(const Bits& o) const {
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = w[i] | o.w[i];
    return b;
  }
  __device__ __forceinline__ Bits andnot(const Bits& o) const {  // this & ~o
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = w[i] & ~o.w[i];
    return b;
  }
  __device__ __forceinline__ bool operator==(const Bits& o) const {
    bool e = true;
#pragma unroll
    for (int i = 0; i < W; i++) e &= w[i] == o.w[i];
    return e;
  }
  __device__ __forceinline__ bool any() const {
    u64 x = 0;
#pragma unroll
    for (int i = 0; i < W; i++) x |= w[i];
    return x != 0ull;
  }
  __device__ __forceinline__ int popc() const {
    int c = 0;
#pragma unroll
    for (int i = 0; i < W; i++) c += __popcll(w[i]);
    return c;
  }
  __device__ __forceinline__ Bits warp_or() const {
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = warp_or64(w[i]);
    return b;
  }
  __device__ __forceinline__ Bits shfl(int src) const {
    Bits b;
#pragma unroll
    for (int i = 0; i < W; i++) b.w[i] = __shfl_sync(kFull, w[i], src);
    return b;
  }
};

// Records the level of newly reached (source, vertex) pairs.  Below
// kDeepLevel slice k of vertex u gains nw for every set bit k of the level.
// From kDeepLevel on the level is stored at once: in the batch's distance
// rows, or in u's level row (level mode); closeness mode sums it per source
// instead (add_deep_sums).  The caller owns u.
__device__ __forceinline__ int batch_of(const BsArgs& a) { return a.batch >= 0 ? a.batch : a.ctl->batch; }

template <int W>
__device__ __forceinline__ void record_level(const BsArgs& a, int32_t u, const Bits<W>& nw, int32_t level) {
  const int32_t n = a.n;
  if (level < kDeepLevel) {
    u64* const slices = a.slices;
    for (unsigned L = (unsigned)level; L; L &= L - 1) {
      u64* p = slices + ((size_t)(__ffs(L) - 1) * n + u) * W;
      (Bits<W>::ld(p) | nw).st(p);
    }
    return;
  }
  if (a.cc_sum) return;
  if (a.lv_block) {
#pragma unroll
    for (int i = 0; i < W; i++) {
      int32_t* row = a.lv_block + ((size_t)i * n + u) * 64;
      for (u64 b = nw.w[i]; b; b &= b - 1) row[__ffsll((long long)b) - 1] = level;
    }
    return;
  }
  int32_t* dist = a.dist_base + (size_t)batch_of(a) * 64 * W * n;
#pragma unroll
  for (int i = 0; i < W; i++)
    for (u64 b = nw.w[i]; b; b &= b - 1) dist[(size_t)(64 * i + __ffsll((long long)b) - 1) * n + u] = level;
}

// Closeness mode from kDeepLevel on: adds the levels of the warp's new bits
// to the CTA's per-source sums.  The warp's 32 new-bit words are transposed
// so lane j counts the bits of sources 64i + j and 64i + 32 + j with popc.
// All 32 lanes call it (nw zero where a lane has no vertex).
template <int W>
__device__ __forceinline__ void add_deep_sums(u64* sums, const Bits<W>& nw, int32_t level) {
  const int lane = lane_id();
#pragma unroll
  for (int i = 0; i < W; i++) {
    if (!__any_sync(kFull, nw.w[i] != 0ull)) continue;
    const unsigned lo = __popc(warp_transpose32((uint32_t)nw.w[i]));
    const unsigned hi = __popc(warp_transpose32((uint32_t)(nw.w[i] >> 32)));
    if (lo) atomicAdd(sums + 64 * i + lane, (unsigned long long)lo * (unsigned)level);
    if (hi) atomicAdd(sums + 64 * i + 32 + lane, (unsigned long long)hi * (unsigned)level);
  }
}
// The CTA's sums: cleared before a level, then added to the batch's rows.
template <int W>
__device__ __forceinline__ void clear_deep_sums(u64* sums) {
  for (int t = threadIdx.x; t < 64 * W; t += blockDim.x) sums[t] = 0;
  __syncthreads();
}
template <int W>
__device__ __forceinline__ void flush_deep_sums(const BsArgs& a, const u64* sums) {
  __syncthreads();
  u64* const rows = a.cc_sum + (size_t)batch_of(a) * 64 * W;
  for (int t = threadIdx.x; t < 64 * W; t += blockDim.x)
    if (sums[t]) atomicAdd(rows + t, sums[t]);
}

// Level L is the last one before slice log2(L + 1) is first used: clear it.
template <int W>
__device__ __forceinline__ void clear_next_slice(const Team& tm, u64* slices, int32_t n, int32_t level, int nbits) {
  const unsigned next = (unsigned)level + 1;
  if (next & (next - 1)) return;
  const int b = __ffs(next) - 1;
  if (b < kSlicesCleared || b >= nbits) return;
  u64* p = slices + (size_t)b * n * W;
  for (size_t i = tm.thread(); i < (size_t)n * W; i += tm.threads()) p[i] = 0ull;
}

// Column loads of the pull.  The in-edge columns stream through once per
// level, so they bypass L1 and are marked first to leave L2 (the frontier
// words they index are what L1 and L2 should keep).  A lane reads its short
// row 32 bytes at a time: one sector per load where two 16-byte loads
// cost two sector lookups in L1/TEX, whose sector throughput bounds the
// pull (one sector per in-edge for the gather of its frontier word).
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ int32_t ld_col(const int32_t* p, uint64_t pol) {
  int32_t v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
// p must be 32-byte aligned; the eight entries may run up to 28 bytes past
// the row (the column arrays carry 32 spare bytes).
__device__ __forceinline__ void ld_col8(const int32_t* p, uint64_t pol, int32_t (&c)[8]) {
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
      : "l"(p), "l"(pol));
}

// Zero the frontier words of a stale active list and its segment list.  A
// list that covers more than a quarter of the vertices is cleared as the
// whole slot instead: n coalesced word stores cost less than that many
// scattered partial-sector writes.
__device__ __forceinline__ bool clears_slot(int cnt, bool unlisted, int32_t n) {
  return unlisted || (long long)cnt * 4 > n;
}
template <int W>
__device__ __forceinline__ void clear_stale(const Team& tm, u64* fr, int32_t n, const int32_t* list, int cnt,
                                            const Seg* segs, int nsegs, bool unlisted) {
  const size_t t0 = tm.thread(), stride = tm.threads();
  if (!clears_slot(cnt, unlisted, n)) {
    for (size_t i = t0; i < (size_t)cnt; i += stride) Bits<W>::zero().st(fr + (size_t)list[i] * W);
    for (size_t i = t0; i < (size_t)nsegs; i += stride) Bits<W>::zero().st(fr + (size_t)segs[i].v * W);
    return;
  }
  // 8-byte stores: a slot starts on an 8-byte boundary only (n * W words
  // per slot, n odd possible), and a warp's 32 of them still fill two lines.
  for (size_t i = t0; i < (size_t)n * W; i += stride) fr[i] = 0ull;
}

__device__ __forceinline__ void clear_words(const Team& tm, u64* words, size_t count) {
  ulonglong2* w2 = reinterpret_cast<ulonglong2*>(words);
  for (size_t i = tm.thread(); i < count / 2; i += tm.threads()) w2[i] = make_ulonglong2(0ull, 0ull);
  if (tm.thread() == 0 && (count & 1)) words[count - 1] = 0;
}

// One CTA of at least 64 W threads: thread b seeds source b of the batch.
template <int W>
__device__ __forceinline__ void init_batch(const BsArgs& a) {
  __shared__ u64 s_mf, s_reached, s_dec;
  BsCtl* const ctl = a.ctl;
  const int32_t *row_ptr = a.row_ptr, *t_row_ptr = a.t_row_ptr;
  u64 *visit = a.visit, *fr0 = a.fr;
  int32_t* aq0 = a.aq;
  Seg* segs0 = a.segs;
  const long long m = a.m;
  const int b = threadIdx.x;
  const int batch = batch_of(a);
  const int per = 64 * W;
  const int nb = min(per, ctl->nsrc - batch * per);
  if (b == 0) {
    s_mf = 0;
    s_reached = 0;
    s_dec = 0;
    for (int i = 0; i < 3; i++) {
      ctl->aq_size[i] = 0;
      ctl->alpack[i] = 0;
    }
    ctl->tq_size = 0;
    ctl->ul_size[0] = 0;
    ctl->ul_size[1] = 0;
    ctl->ul_cur = -1;
    ctl->unlisted[0] = ctl->unlisted[1] = ctl->unlisted[2] = 0;
    ctl->hs_size[0] = 0;
    ctl->hs_size[1] = 0;
    ctl->hs_cur = -1;
    ctl->work = 0;
    ctl->hwork = 0;
    ctl->dense = 0;
    for (int i = 0; i < kMaxW; i++) {
      const int bits = min(64, max(0, nb - 64 * i));
      ctl->full[i] = i >= W ? 0ull : (bits == 64 ? ~0ull : ((1ull << bits) - 1ull));
    }
  }
  __syncthreads();
  int32_t s = -1;
  int rs = 0, deg = 0;
  if (b < nb) {
    s = ctl->sources[batch * per + b];
    const u64 bit = 1ull << (b & 63);
    atomicOr(visit + (size_t)s * W + (b >> 6), bit);
    atomicOr(fr0 + (size_t)s * W + (b >> 6), bit);
    rs = row_ptr[s];
    deg = row_ptr[s + 1] - rs;
    // A source without out-edges reaches no vertex but itself.  Its bit is
    // left out of `full`, so the other vertices still finish (and leave
    // the pull lists) once every other source has reached them; a batch
    // of all vertices as sources holds many such sources.
    if (deg == 0) atomicAnd(&ctl->full[b >> 6], ~bit);
  }
  // (64-bit sums in shared memory are compare-and-swap loops: one per warp)
  const u64 reached = warp_sum((u64)deg);
  if (lane_id() == 0 && reached) atomicAdd(&s_reached, reached);
  __syncthreads();
  // A vertex that is the source of several bits is queued once, by the
  // thread of its lowest bit.
  bool lowest = b < nb;
  if (lowest) {
    const Bits<W> f = Bits<W>::ldcg(fr0 + (size_t)s * W);
#pragma unroll
    for (int i = 0; i < W; i++) {
      const u64 below = i < (b >> 6) ? ~0ull : (i == (b >> 6) ? (1ull << (b & 63)) - 1ull : 0ull);
      lowest &= (f.w[i] & below) == 0ull;
    }
  }
  u64 dec = 0;
  if (lowest && Bits<W>::ldcg(visit + (size_t)s * W) == Bits<W>::full_of(ctl)) dec = (u64)(t_row_ptr[s + 1] - t_row_ptr[s]);
  const u64 mf = warp_sum(lowest ? (u64)deg : 0ull);
  dec = warp_sum(dec);
  if (lane_id() == 0) {
    if (mf) atomicAdd(&s_mf, mf);
    if (dec) atomicAdd(&s_dec, dec);
  }
  if (b < per) emit_routed(lowest, s, deg, rs, aq0, &ctl->aq_size[0], segs0, &ctl->alpack[0]);  // whole warps
  __syncthreads();
  if (b == 0) {
    for (int i = 0; i < 3; i++) ctl->mf[i] = 0;
    ctl->mf[0] = s_mf;
    ctl->reached = s_reached;
    ctl->mu = m - (long long)s_dec;
    ctl->mu_dec = 0;
    ctl->level = 1;
    ctl->mode = ctl->force - 1 == kVarPull ? kModePull : kModePush;
    ctl->dense = ctl->force - 1 == kVarDense;
    ctl->prev_nf = 0;
    ctl->done = 0;
    ctl->n_push = 0;
    ctl->n_pull = 0;
  }
}

// Shared memory of a level's work: per warp two staging queues (the push
// keeps its row dealing in the second one's place).
template <int kWarps>
struct BsSmem {
  int32_t q[kWarps][2 * kWarpQueueBig];
  u64 acc[3];
  u64 deep[64 * kMaxW];  // closeness: per-source sums of deep levels
  uint32_t n[2][kWarps];
  int32_t nf;
  u64 word[16];
  BsStep st, next;  // the running phase, and in its last CTA the one it opens
};
static_assert(3 * 32 <= kWarpQueueBig, "row dealing fits the second queue");

// Per-thread accumulators of a level.
struct LevelAcc {
  u64 mf = 0, reached = 0, dec = 0;
  __device__ __forceinline__ void add(u64 out_deg, u64 in_deg, int new_pairs, bool finished) {
    mf += out_deg;
    reached += out_deg * (u64)new_pairs;
    if (finished) dec += in_deg;
  }
};

// The end of a CTA's share of a level: what its warps still stage goes out
// with one reservation per queue, and its sums and counts with one atomic
// each.  A reservation and three sums per warp were 5,000 to 6,000 atomics on
// each of five words at every level: 10 us even where no vertex was left to
// visit.  b may be NULL; nf is added to *nf_count when given.
template <int kWarps>
__device__ __forceinline__ void end_level(BsSmem<kWarps>& sm, BsCtl* ctl, int slot, LevelAcc& acc, WarpQueueBig& a,
                                          WarpQueueBig* b, int nf, int32_t* nf_count) {
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  if (threadIdx.x < 3) sm.acc[threadIdx.x] = 0;
  if (threadIdx.x == 3) sm.nf = 0;
  if (lane == 0) {
    sm.n[0][wib] = (uint32_t)a.n;
    sm.n[1][wib] = b ? (uint32_t)b->n : 0u;
  }
  __syncthreads();
  const u64 mf = warp_sum(acc.mf), reached = warp_sum(acc.reached), dec = warp_sum(acc.dec);
  if (lane == 0) {
    if (mf) atomicAdd(&sm.acc[0], mf);
    if (reached) atomicAdd(&sm.acc[1], reached);
    if (dec) atomicAdd(&sm.acc[2], dec);
    if (nf) atomicAdd(&sm.nf, nf);
  }
  if (wib == 0) {
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int x = lane < kWarps ? (int)sm.n[q][lane] : 0;
      const int incl = warp_incl_scan(x);
      const int tot = __shfl_sync(kFull, incl, 31);
      int base = 0;
      if (tot && lane == 0) base = atomicAdd(q ? b->count : a.count, tot);
      base = __shfl_sync(kFull, base, 0);
      if (lane < kWarps) sm.n[q][lane] = (uint32_t)(base + incl - x);
    }
  }
  __syncthreads();
  for (int i = lane; i < a.n; i += 32) a.out[sm.n[0][wib] + i] = a.buf[i];
  if (b)
    for (int i = lane; i < b->n; i += 32) b->out[sm.n[1][wib] + i] = b->buf[i];
  if (threadIdx.x == 0) {
    if (sm.acc[0]) atomicAdd(&ctl->mf[slot], sm.acc[0]);
    if (sm.acc[1]) atomicAdd(&ctl->reached, sm.acc[1]);
    if (sm.acc[2]) atomicAdd(reinterpret_cast<u64*>(&ctl->mu_dec), sm.acc[2]);
    if (nf_count && sm.nf) atomicAdd(nf_count, sm.nf);
  }
}

// Pull: every vertex of the unfinished list ORs the frontier words of its
// in-neighbours.  Heavy rows (>= 2 x pull_seg in-edges) come first, one
// pull_seg-entry segment per warp task, OR-ed into the row's accumulator;
// the warp finishing a row's last segment folds the accumulator into the
// vertex, so only one warp writes a vertex's words and every segment sees
// the same visited words for the whole level.  Light rows follow, 32 list
// entries per warp task from a shared counter: rows of >= kPullLaneMax
// entries are swept by the whole warp (4 gathers in flight per lane, early
// exit once no missing bit is left), shorter ones are walked by one lane
// each.  The list is filtered into the next unfinished list as it goes.
template <int W, int kWarps>
__device__ __forceinline__ void pull_level(const BsArgs& a, const Team& tm, const BsStep& st, BsSmem<kWarps>& sm) {
  using B = Bits<W>;
  BsCtl* const ctl = a.ctl;
  const int32_t* __restrict__ row_ptr = a.row_ptr;
  const int32_t* __restrict__ t_row_ptr = a.t_row_ptr;
  const int32_t* __restrict__ t_col = a.t_col;
  const int32_t* __restrict__ hv_static = a.hv_static;
  const int32_t* __restrict__ hv_segoff = a.hv_segoff;
  u64 *const visit = a.visit, *const hv_acc = a.hv_acc;
  const int32_t n = a.n, pull_seg = a.pull_seg, hv_segs = a.hv_segs;
  const int L = st.L;
  const u64* fin = a.fr + (size_t)((L - 1) % 3) * n * W;
  u64* fout = a.fr + (size_t)(L % 3) * n * W;
  int32_t* aq_out = a.aq + (size_t)(L % 3) * n;
  Seg* seg_out = a.segs + (size_t)(L % 3) * a.segcap;
  int32_t* aq_count = &ctl->aq_size[L % 3];
  u64* al_pack = &ctl->alpack[L % 3];
  clear_stale<W>(tm, a.fr + (size_t)((L + 1) % 3) * n * W, n, a.aq + (size_t)((L + 1) % 3) * n,
                 st.stale, a.segs + (size_t)((L + 1) % 3) * a.segcap, st.stale_segs, st.stale_unlisted != 0);
  const uint64_t pol = evict_first_policy();
  clear_next_slice<W>(tm, a.slices, n, L, a.nbits);
  const int cur = st.ul_cur;
  const int32_t* ul_in = cur < 0 ? a.ul_static : a.ul + (size_t)cur * n;
  const int un = st.un;
  const int nxt = cur < 0 ? 0 : cur ^ 1;
  int32_t* ul_out = a.ul + (size_t)nxt * n;
  int32_t* ul_count = &ctl->ul_size[nxt];
  const B full = B::full_of(ctl);
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  LevelAcc acc;
  WarpQueueBig qa(sm.q[wib], aq_out, aq_count);
  WarpQueueBig qu(sm.q[wib] + kWarpQueueBig, ul_out, ul_count);
  const bool deep_cc = a.cc_sum && L >= kDeepLevel;
  if (deep_cc) clear_deep_sums<W>(sm.deep);
  // A pull level entered with a frontier of at least n / 16 vertices keeps
  // no active list: its output frontier is counted, the next level is made
  // a pull (which reads frontier words), and the slot is cleared densely
  // when it goes stale.  Smaller levels queue their output for a push.
  const bool lazy = !a.force && (long long)st.nf * 16 >= n;
  int my_nf = 0;
  // Heavy-row segments: the first pull level deals every segment of the
  // graph (finding its row by binary search); the finisher of a row that
  // stays unfinished re-lists the row's segments as (row, segment) tasks,
  // and later pull levels deal only those.
  const int hcur = st.hs_cur, hn = st.hn;
  const int2* hs_in = a.hv_tasks + (size_t)(hcur < 0 ? 0 : hcur) * hv_segs;
  int2* hs_out = a.hv_tasks + (size_t)(hcur < 0 ? 0 : hcur ^ 1) * hv_segs;
  int32_t* hs_count = &ctl->hs_size[hcur < 0 ? 0 : hcur ^ 1];

  // A warp's first task is its own; the shared counters deal the rest.
  const int gw = tm.warp(), nw = tm.warps();
  for (int t = gw; t < hn; t = nw + __shfl_sync(kFull, lane == 0 ? atomicAdd(&ctl->hwork, 1) : 0, 0)) {
    int lo = 0, sidx = t;
    if (hcur < 0) {
      int hi = a.hv_count - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(hv_segoff + mid) <= sidx) lo = mid; else hi = mid - 1;
      }
    } else {
      const int2 e = hs_in[t];
      lo = e.x;
      sidx = e.y;
    }
    const int32_t u = __ldg(hv_static + lo);
    const B vis = B::ld(visit + (size_t)u * W);
    if (vis == full) continue;
    const int s0 = __ldg(hv_segoff + lo);
    const int nseg = __ldg(hv_segoff + lo + 1) - s0;
    const int rbeg = t_row_ptr[u], rend = t_row_ptr[u + 1];
    const int ks = rbeg + (sidx - s0) * pull_seg, ke = min(ks + pull_seg, rend);
    u64* hacc = hv_acc + (size_t)lo * acc_stride(W);
    B w = B::zero();
    for (int k0 = ks; k0 < ke; k0 += 128) {
      const int k = k0 + lane;
      const int32_t v0 = k < ke ? ld_col(t_col + k, pol) : -1;
      const int32_t v1 = k + 32 < ke ? ld_col(t_col + k + 32, pol) : -1;
      const int32_t v2 = k + 64 < ke ? ld_col(t_col + k + 64, pol) : -1;
      const int32_t v3 = k + 96 < ke ? ld_col(t_col + k + 96, pol) : -1;
      if (v0 >= 0) w = w | B::gather(fin + (size_t)v0 * W);
      if (v1 >= 0) w = w | B::gather(fin + (size_t)v1 * W);
      if (v2 >= 0) w = w | B::gather(fin + (size_t)v2 * W);
      if (v3 >= 0) w = w | B::gather(fin + (size_t)v3 * W);
      if ((w.warp_or() | vis | B::ldcg(hacc)) == full) break;
    }
    w = w.warp_or();
    int last = 0;
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < W; i++)
        if (w.w[i]) atomicOr(hacc + i, w.w[i]);
      __threadfence();
      last = atomicAdd(hacc + W, 1ull) == (u64)(nseg - 1);
    }
    last = __shfl_sync(kFull, last, 0);
    if (!last) continue;
    B nw = B::zero();
    int odeg = 0, ors = 0;
    if (lane == 0) {
      __threadfence();
      B got;
#pragma unroll
      for (int i = 0; i < W; i++) {
        got.w[i] = atomicOr(hacc + i, 0ull);
        hacc[i] = 0ull;
      }
      hacc[W] = 0ull;
      nw = got.andnot(vis);
      if (nw.any()) {
        (vis | nw).st(visit + (size_t)u * W);
        nw.st(fout + (size_t)u * W);
        record_level<W>(a, u, nw, L);
        ors = row_ptr[u];
        odeg = row_ptr[u + 1] - ors;
        acc.add((u64)odeg, (u64)(rend - rbeg), nw.popc(), (vis | nw) == full);
      }
    }
    // a row still missing bits keeps its segments for the next pull level
    const B nw0 = nw.shfl(0);
    if (!((vis | nw0) == full)) {
      int base = 0;
      if (lane == 0) base = atomicAdd(hs_count, nseg);
      base = __shfl_sync(kFull, base, 0);
      for (int j = lane; j < nseg; j += 32) hs_out[base + j] = make_int2(lo, s0 + j);
    }
    if (deep_cc) add_deep_sums<W>(sm.deep, nw, L);
    if (lazy)
      my_nf += __popc(__ballot_sync(kFull, nw.any()));
    else
      emit_routed(nw.any(), u, odeg, ors, qa, seg_out, al_pack);
  }

  // Rows per warp task: 32, or fewer where the list is short.  Rows of 64 and
  // more in-edges go one after another in their task, so graphs that have them
  // (a mean in-degree of 24 and more) want several tasks per warp; elsewhere
  // fewer than 32 rows only where half the warps would stay idle (a 29 us pull
  // of 200,003 mesh vertices took 8 rows a task in four rounds).
  int rows = 32;
  const long long spread = a.m >= 24ll * n ? 8ll * nw : (long long)nw;
  while (rows > 8 && 2ll * un < spread * rows) rows >>= 1;
  for (int base = gw * rows; base < un;
       base = nw * rows + __shfl_sync(kFull, lane == 0 ? atomicAdd(&ctl->work, rows) : 0, 0)) {
    const int idx = base + lane;
    int32_t u = -1;
    B vis = full;
    if (lane < rows && idx < un) {
      u = ul_in[idx];
      vis = B::ld(visit + (size_t)u * W);
    }
    const bool active = !(vis == full);
    int rs = 0, re = 0;
    if (active) {
      rs = t_row_ptr[u];
      re = t_row_ptr[u + 1];
    }
    const int deg = re - rs;
    B got = B::zero();
    uint32_t big = __ballot_sync(kFull, deg >= kPullLaneMax);
    while (big) {
      const int leader = __ffs(big) - 1;
      big &= big - 1;
      const int s = __shfl_sync(kFull, rs, leader), e = __shfl_sync(kFull, re, leader);
      const B lvis = vis.shfl(leader);
      B w = B::zero();
      for (int k0 = s; k0 < e; k0 += 128) {
        const int k = k0 + lane;
        const int32_t v0 = k < e ? ld_col(t_col + k, pol) : -1;
        const int32_t v1 = k + 32 < e ? ld_col(t_col + k + 32, pol) : -1;
        const int32_t v2 = k + 64 < e ? ld_col(t_col + k + 64, pol) : -1;
        const int32_t v3 = k + 96 < e ? ld_col(t_col + k + 96, pol) : -1;
        if (v0 >= 0) w = w | B::gather(fin + (size_t)v0 * W);
        if (v1 >= 0) w = w | B::gather(fin + (size_t)v1 * W);
        if (v2 >= 0) w = w | B::gather(fin + (size_t)v2 * W);
        if (v3 >= 0) w = w | B::gather(fin + (size_t)v3 * W);
        if ((w.warp_or() | lvis) == full) break;
      }
      w = w.warp_or();
      if (lane == leader) got = w;
    }
    // Short rows: each lane walks its own row, four in-neighbours in
    // flight, and stops once its missing bits are all found.  No shared
    // memory and no search per edge: the L1/TEX path carries only the
    // column loads and the gathers.
    if (active && deg < kPullLaneMax) {
      // The row is read in 32-byte aligned chunks of eight entries, one
      // 32-byte load each (from before the row start when it is not
      // aligned; in-edge arrays carry 32 spare bytes, so no load passes
      // their end), so a lane issues one column load per eight gathers.
      B w = B::zero();
      for (int a = rs & ~7; a < re; a += 8) {
        int32_t c[8];
        ld_col8(t_col + a, pol, c);
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (a + j >= rs && a + j < re) w = w | B::gather(fin + (size_t)c[j] * W);
        if ((w | vis) == full) break;
      }
      got = w;
    }
    const B nw = active ? got.andnot(vis) : B::zero();
    const bool has = nw.any();
    const bool still = active && !((vis | nw) == full);
    int odeg = 0, ors = 0;
    if (has) {
      (vis | nw).st(visit + (size_t)u * W);
      nw.st(fout + (size_t)u * W);
      record_level<W>(a, u, nw, L);
      ors = row_ptr[u];
      odeg = row_ptr[u + 1] - ors;
      acc.add((u64)odeg, (u64)deg, nw.popc(), !still);
    }
    if (deep_cc) add_deep_sums<W>(sm.deep, nw, L);
    qu.push(still, u);
    if (lazy)
      my_nf += __popc(__ballot_sync(kFull, has));
    else
      emit_routed(has, u, odeg, ors, qa, seg_out, al_pack);
  }
  end_level(sm, ctl, L % 3, acc, qa, &qu, my_nf, aq_count);
  if (deep_cc) flush_deep_sums<W>(a, sm.deep);
  if (lazy && tm.thread() == 0) ctl->unlisted[L % 3] = 1;
}

// Push, phase 1: the active vertices' rows (short rows warp-cooperatively,
// long rows as segments) are dealt to warps; bits new to a target are
// atomicOr-ed into `next` (not visited yet at that source).  In list mode
// the first toucher (claiming the target in a touched bitmap) queues it for
// phase 2; in dense mode (large frontiers) no queue is kept and phase 2
// sweeps all vertices instead.
template <int W, int kWarps>
__device__ __forceinline__ void scatter_level(const BsArgs& a, const Team& tm, const BsStep& st,
                                              BsSmem<kWarps>& sm) {
  using B = Bits<W>;
  BsCtl* const ctl = a.ctl;
  const int32_t* __restrict__ row_ptr = a.row_ptr;
  const int32_t* __restrict__ col = a.col;
  const u64* const visit = a.visit;
  u64* const nxt = a.nxt;
  uint32_t* const tbm = a.tbm;
  const int32_t n = a.n;
  const int L = st.L;
  const u64* fin = a.fr + (size_t)((L - 1) % 3) * n * W;
  const int32_t* aq_in = a.aq + (size_t)((L - 1) % 3) * n;
  const Seg* seg_in = a.segs + (size_t)((L - 1) % 3) * a.segcap;
  const int qn = st.qn, ln = st.ln;
  const bool dense = st.dense != 0;
  clear_stale<W>(tm, a.fr + (size_t)((L + 1) % 3) * n * W, n, a.aq + (size_t)((L + 1) % 3) * n,
                 st.stale, a.segs + (size_t)((L + 1) % 3) * a.segcap, st.stale_segs, st.stale_unlisted != 0);
  clear_next_slice<W>(tm, a.slices, n, L, a.nbits);
  const int wib = threadIdx.x >> 5;
  int32_t* const deal = sm.q[wib] + kWarpQueueBig;
  // The first two levels expand the sources and their neighbours, whose
  // targets are almost never visited yet: there the visited words are not
  // read (one random load per edge fewer), and the update drops the few
  // visited bits.  Later levels filter first, which saves the atomics of
  // edges back into the visited region (half of a wavefront's edges on a
  // mesh).
  const bool filter = L > 2;
  WarpQueueBig wq(sm.q[wib], a.tq, &ctl->tq_size);
  auto op = [&](int32_t v, int k, bool valid) {
    bool first = false;
    int32_t u = -1;
    if (valid) {
      u = __ldg(col + k);
      // No look at `next` first: its bits are OR-ed in whether or not they
      // are there, which saves a random load per edge (the scatter is bound
      // by the L1/TEX traffic of its random accesses).
      B bits = B::gather(fin + (size_t)v * W);
      if (filter) bits = bits.andnot(B::ldcg(visit + (size_t)u * W));
      if (bits.any()) {
        if (W == 1 && !dense) {
          // one word: the OR that finds it empty is the first touch (no
          // touched bitmap to claim in and clear again)
          first = atomicOr(nxt + u, bits.w[0]) == 0ull;
        } else {
#pragma unroll
          for (int i = 0; i < W; i++)
            if (bits.w[i]) or_word(nxt + (size_t)u * W + i, bits.w[i]);
          if (!dense) first = claim_bit(tbm, u);
        }
      }
    }
    if (!dense) wq.push(first, u);
  };
  seg_expand(tm.warp(), tm.warps(), row_ptr, seg_in, ln, op);
  warp_expand(tm.warp(), tm.warps(), row_ptr, aq_in, qn, deal, deal + 32, deal + 64, op);
  LevelAcc none;
  if (!dense) end_level(sm, ctl, L % 3, none, wq, nullptr, 0, nullptr);
}

// Push, phase 2: fold `next` into visited / frontier / level slices, over
// the touched list (list mode, clearing the touched bitmap) or over every
// vertex (dense mode).
template <int W, int kWarps>
__device__ __forceinline__ void update_level(const BsArgs& a, const Team& tm, const BsStep& st,
                                             BsSmem<kWarps>& sm) {
  using B = Bits<W>;
  BsCtl* const ctl = a.ctl;
  const int32_t* __restrict__ row_ptr = a.row_ptr;
  const int32_t* __restrict__ t_row_ptr = a.t_row_ptr;
  u64 *const visit = a.visit, *const nxt = a.nxt;
  const int32_t* const tq = a.tq;
  uint32_t* const tbm = a.tbm;
  const int32_t n = a.n;
  const int L = st.L;
  u64* fout = a.fr + (size_t)(L % 3) * n * W;
  int32_t* aq_out = a.aq + (size_t)(L % 3) * n;
  Seg* seg_out = a.segs + (size_t)(L % 3) * a.segcap;
  const B full = B::full_of(ctl);
  const bool dense = st.dense != 0;
  const int tn = dense ? n : st.tn;
  // A dense level's output frontier is large enough that the next level is
  // a pull (the decide kernel makes it one), which reads frontier words,
  // not an active list: the sweep then only counts the frontier instead of
  // queueing it and cutting its long rows into segments.  Forced-variant
  // runs keep the list (a forced push reads it).
  const bool lazy = dense && !a.force;
  int my_nf = 0;
  WarpQueueBig wq(sm.q[threadIdx.x >> 5], aq_out, &ctl->aq_size[L % 3]);
  LevelAcc acc;
  const bool deep_cc = a.cc_sum && L >= kDeepLevel;
  if (deep_cc) clear_deep_sums<W>(sm.deep);
  // Vertices per warp: fewer than 32 for a short list, so that its scattered
  // words (some ten sectors a vertex) are spread over all SMs: a level of 45,000
  // vertices on 70 CTAs took 11 us.
  int per = 32;
  while (per > 4 && (long long)(per >> 1) * tm.warps() >= tn) per >>= 1;
  for (int base = tm.warp() * per; base < tn; base += tm.warps() * per) {
    const int i = lane_id() < per ? base + lane_id() : tn;
    B nw = B::zero();
    int32_t u = -1;
    int odeg = 0, ors = 0;
    if (i < tn) {
      u = dense ? i : tq[i];
      if (!dense && W > 1) atomicAnd(tbm + (u >> 5), ~(1u << (u & 31)));
      const B x = B::ld(nxt + (size_t)u * W);
      // A listed vertex was touched, so all of its words and row bounds are
      // fetched in one round trip (three of them took a level of a 700 x 700
      // grid 10 us); a sweep first looks whether it was.
      if (!dense || x.any()) {
        const B vis = B::ld(visit + (size_t)u * W);
        ors = row_ptr[u];
        odeg = row_ptr[u + 1] - ors;
        const int ideg = t_row_ptr[u + 1] - t_row_ptr[u];
        B::zero().st(nxt + (size_t)u * W);
        nw = x.andnot(vis);
        if (nw.any()) {
          (vis | nw).st(visit + (size_t)u * W);
          nw.st(fout + (size_t)u * W);
          record_level<W>(a, u, nw, L);
          acc.add((u64)odeg, (u64)ideg, nw.popc(), (vis | nw) == full);
        }
      }
    }
    if (deep_cc) add_deep_sums<W>(sm.deep, nw, L);
    if (lazy)
      my_nf += __popc(__ballot_sync(kFull, nw.any()));
    else
      emit_routed(nw.any(), u, odeg, ors, wq, seg_out, &ctl->alpack[L % 3]);
  }
  end_level(sm, ctl, L % 3, acc, wq, nullptr, my_nf, &ctl->aq_size[L % 3]);
  if (deep_cc) flush_deep_sums<W>(a, sm.deep);
  if (lazy && tm.thread() == 0) ctl->unlisted[L % 3] = 1;
}

// Both phases of a list-mode push at once, for one-word batches in the persistent
// launch: an edge's bits are claimed in the visited words, and whoever claims a
// bit records its level and puts it in the frontier (the first one queues the
// vertex).  Each bit has one claimer, so nothing is written twice.  One step
// instead of two for the thin levels of meshes and of any graph's first and last
// levels, which are bound by the chain of round trips of a step, not by the
// returning atomics that this takes.  Two phases -> this, us a call: grid 700 x 700
// 23080 -> 15380 (64 sources), 20720 -> 13080 (3); kNN of 75,331 points 3760 ->
// 3540, 3780 -> 2450; Erdos-Renyi 65,536 x 16 126 -> 118 (64).
template <int kWarps>
__device__ __forceinline__ void push_level(const BsArgs& a, const Team& tm, const BsStep& st, BsSmem<kWarps>& sm) {
  BsCtl* const ctl = a.ctl;
  const int32_t* __restrict__ row_ptr = a.row_ptr;
  const int32_t* __restrict__ col = a.col;
  const int32_t n = a.n;
  const int L = st.L;
  const u64* fin = a.fr + (size_t)((L - 1) % 3) * n;
  u64* fout = a.fr + (size_t)(L % 3) * n;
  Seg* seg_out = a.segs + (size_t)(L % 3) * a.segcap;
  clear_stale<1>(tm, a.fr + (size_t)((L + 1) % 3) * n, n, a.aq + (size_t)((L + 1) % 3) * n, st.stale,
                 a.segs + (size_t)((L + 1) % 3) * a.segcap, st.stale_segs, st.stale_unlisted != 0);
  clear_next_slice<1>(tm, a.slices, n, L, a.nbits);
  const int wib = threadIdx.x >> 5;
  int32_t* const deal = sm.q[wib] + kWarpQueueBig;
  const u64 full = ctl->full[0];
  WarpQueueBig wq(sm.q[wib], a.aq + (size_t)(L % 3) * n, &ctl->aq_size[L % 3]);
  LevelAcc acc;
  const bool deep_cc = a.cc_sum && L >= kDeepLevel;
  if (deep_cc) clear_deep_sums<1>(sm.deep);
  auto op = [&](int32_t v, int k, bool valid) {
    bool first = false;
    int32_t u = -1;
    int ors = 0, odeg = 0;
    Bits<1> nw = Bits<1>::zero();
    if (valid) {
      u = __ldg(col + k);
      const u64 bits = Bits<1>::gather(fin + v).w[0] & ~__ldcg(a.visit + u);
      if (bits) {
        const u64 old = atomicOr(a.visit + u, bits);
        ors = __ldg(row_ptr + u);
        odeg = __ldg(row_ptr + u + 1) - ors;
        nw.w[0] = bits & ~old;
        if (nw.w[0]) {
          first = atomicOr(fout + u, nw.w[0]) == 0ull;
          if (L < kDeepLevel) {
            for (unsigned l = (unsigned)L; l; l &= l - 1) atomicOr(a.slices + (size_t)(__ffs(l) - 1) * n + u, nw.w[0]);
          } else {
            record_level<1>(a, u, nw, L);
          }
          acc.reached += (u64)odeg * (u64)nw.popc();
          if (first) acc.mf += (u64)odeg;
          if ((old | bits) == full) acc.dec += (u64)(__ldg(a.t_row_ptr + u + 1) - __ldg(a.t_row_ptr + u));
        }
      }
    }
    if (deep_cc) add_deep_sums<1>(sm.deep, nw, L);
    emit_routed(first, u, odeg, ors, wq, seg_out, &ctl->alpack[L % 3]);
  };
  seg_expand<true>(tm.warp(), tm.warps(), row_ptr, a.segs + (size_t)((L - 1) % 3) * a.segcap, st.ln, op);
  warp_expand<true>(tm.warp(), tm.warps(), row_ptr, a.aq + (size_t)((L - 1) % 3) * n, st.qn, deal, deal + 32, deal + 64,
                    op);
  end_level(sm, ctl, L % 3, acc, wq, nullptr, 0, &ctl->aq_size[L % 3]);
  if (deep_cc) flush_deep_sums<1>(a, sm.deep);
}

// Expands the level slices of one batch into its distance rows: thread per
// vertex, one store per source, consecutive vertices per warp (full lines).
// NB is the number of level bits in use (<= kShallowBits).  src is the
// batch's source list when the traversal went past kDeepLevel, else NULL:
// then a reached pair whose slice bits are all zero is either the source
// itself (level 0) or was written out during the traversal, and is kept.
template <int W, int NB>
__device__ __forceinline__ void emit_vertex(int32_t* __restrict__ dist, int32_t n, int nb_src, size_t u,
                                            const u64* visit, const u64* slices,
                                            const int32_t* __restrict__ src) {
#pragma unroll
  for (int i = 0; i < W; i++) {
    if (64 * i >= nb_src) break;
    const u64 vis = visit[u * W + i];
    u64 w[NB];
    u64 any = 0ull;
#pragma unroll
    for (int k = 0; k < NB; k++) {
      w[k] = slices[((size_t)k * n + u) * W + i];
      any |= w[k];
    }
    const int cnt = min(64, nb_src - 64 * i);
    for (int s = 0; s < cnt; s++) {
      int32_t v = -1;
      if ((vis >> s) & 1ull) {
        if (src && !((any >> s) & 1ull) && src[64 * i + s] != (int32_t)u) continue;  // written at its level
        v = 0;
#pragma unroll
        for (int k = 0; k < NB; k++) v |= (int32_t)((w[k] >> s) & 1ull) << k;
      }
      dist[(size_t)(64 * i + s) * n + u] = v;
    }
  }
}

// emit_vertex4 without deep levels (no pair was written during the
// traversal): the level of source s at vertex j is assembled from the level
// slices eight sources at a time.  Byte c of slices 0-3 goes into one word
// (slice k in byte k); for source 8c + i, ((word >> i) & 0x01010101) holds
// the four level bits at bits 0, 8, 16, 24, and multiplying by 0x01020408
// moves them to bits 24-27 without carries (every partial product lands on
// a distinct bit, and only the four wanted ones land in bits 24-31).  A
// fifth slice adds its bit separately; an unreached pair becomes -1 by
// OR-ing (bit - 1).  About 8 instructions per (source, vertex) instead of
// 19 with a shift and mask per slice.
// One word i and its bytes c0 .. c1 - 1 per call: the items of a batch of 256
// sources are then words, not vertices (RMAT-18 has 65,536 groups of four vertices
// for 311,000 threads: 500 sources 784 -> 757 us a call).
template <int W, int NB>
__device__ __forceinline__ void emit_vertex4_packed(int32_t* __restrict__ dist, int32_t n, int nb_src, size_t u0,
                                                    const u64* visit, const u64* slices, int i, int c0, int c1) {
  if (64 * i + 8 * c0 >= nb_src) return;
  u64 vis[4], w[NB][4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    vis[j] = visit[(u0 + j) * W + i];
#pragma unroll
    for (int k = 0; k < NB; k++) w[k][j] = slices[((size_t)k * n + u0 + j) * W + i];
  }
  const int cnt = min(64, nb_src - 64 * i);
  int32_t* row0 = dist + (size_t)(64 * i) * n + u0;
  for (int c = c0; c < c1 && 8 * c < cnt; c++) {
    uint32_t packed[4], five[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t x = 0;
#pragma unroll
      for (int k = 0; k < (NB < 4 ? NB : 4); k++) x |= (uint32_t)((w[k][j] >> (8 * c)) & 0xffull) << (8 * k);
      packed[j] = x;
      five[j] = NB > 4 ? (uint32_t)(w[NB > 4 ? 4 : 0][j] >> (8 * c)) & 0xffu : 0u;
      vb[j] = (uint32_t)(vis[j] >> (8 * c)) & 0xffu;
    }
    const int lim = min(8, cnt - 8 * c);
    for (int b = 0; b < lim; b++) {
      int32_t v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t x = (((packed[j] >> b) & 0x01010101u) * 0x01020408u) >> 24;
        if (NB > 4) x |= ((five[j] >> b) & 1u) << 4;
        v[j] = (int32_t)(x | (((vb[j] >> b) & 1u) - 1u));
      }
      *reinterpret_cast<int4*>(row0 + (size_t)(8 * c + b) * n) = make_int4(v[0], v[1], v[2], v[3]);
    }
  }
}

// Four consecutive vertices u0..u0+3 per thread: every source row gets one
// 16-byte store, so a warp writes 512 contiguous bytes per row (needs n and
// the output base 16-byte aligned, which the caller checks).  Rows holding a
// pair written during the traversal (see emit_vertex) get scalar stores for
// the other three.
template <int W, int NB>
__device__ __forceinline__ void emit_vertex4(int32_t* __restrict__ dist, int32_t n, int nb_src, size_t u0,
                                             const u64* visit, const u64* slices,
                                             const int32_t* __restrict__ src) {
#pragma unroll
  for (int i = 0; i < W; i++) {
    if (64 * i >= nb_src) break;
    u64 vis[4], any[4];
    u64 w[NB][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      vis[j] = visit[(u0 + j) * W + i];
      any[j] = 0ull;
#pragma unroll
      for (int k = 0; k < NB; k++) {
        w[k][j] = slices[((size_t)k * n + u0 + j) * W + i];
        any[j] |= w[k][j];
      }
    }
    const int cnt = min(64, nb_src - 64 * i);
    for (int s = 0; s < cnt; s++) {
      int32_t v[4];
      bool keep[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        v[j] = -1;
        keep[j] = false;
        if ((vis[j] >> s) & 1ull) {
          int32_t x = 0;
#pragma unroll
          for (int k = 0; k < NB; k++) x |= (int32_t)((w[k][j] >> s) & 1ull) << k;
          v[j] = x;
          keep[j] = src && !((any[j] >> s) & 1ull) && src[64 * i + s] != (int32_t)(u0 + j);
        }
      }
      int32_t* row = dist + (size_t)(64 * i + s) * n + u0;
      if (!(keep[0] | keep[1] | keep[2] | keep[3])) {
        *reinterpret_cast<int4*>(row) = make_int4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (!keep[j]) row[j] = v[j];
      }
    }
  }
}

// Closeness mode of the final pass: per source of the batch, the sum of its
// hop distances (sum over level bits k of 2^k x the vertices whose slice k
// holds the source's bit) and the vertices it reached besides itself,
// without writing distances.  Each warp transposes the words of 32
// consecutive vertices so lane j holds bit j (and j + 32) of all of them and
// counts them with popc; CTA totals go to the batch's rows with one atomic
// per source.
// CTAs per SM of the closeness pass: each adds two words per source to the same
// 512 (closeness of 1,000 sources on RMAT-18, 1 / 2 / 4 / 8: 1603 / 1571 / 1584 /
// 1610 us, 1717 with eight and 64-bit sums in shared memory).
constexpr int kClosenessCtas = 2;
// And in all: a CTA's sums are 32-bit, and exact while its share of the vertices (at
// most 2^31 in all, dealt 256 at a time) times 31 levels stays below 2^32, on
// however few SMs.
constexpr int kClosenessMin = 16;
static_assert(((1ull << 31) / kClosenessMin + 256) * (kDeepLevel - 1) < 1ull << 32, "a CTA's sums fit 32 bits");
template <int W>
__device__ __forceinline__ void emit_closeness(const Team& tm, const BsCtl* ctl, int batch, const u64* visit,
                                               const u64* slices, int32_t n, int nb, int nbits) {
  __shared__ uint32_t s_sum[64 * W], s_cnt[64 * W];
  for (int t = threadIdx.x; t < 64 * W; t += blockDim.x) {
    s_sum[t] = 0;
    s_cnt[t] = 0;
  }
  __syncthreads();
  const int lane = lane_id();
#pragma unroll
  for (int i = 0; i < W; i++) {
    if (64 * i >= nb) break;
    unsigned long long sum_lo = 0, sum_hi = 0;
    unsigned cnt_lo = 0, cnt_hi = 0;
    for (int base = tm.warp() * 32; base < n; base += tm.warps() * 32) {
      const int u = base + lane;
      const bool in = u < n;
      // the words of every slice are loaded before the first is transposed
      u64 x[kShallowBits];
#pragma unroll
      for (int k = 0; k < kShallowBits; k++) x[k] = in && k < nbits ? slices[((size_t)k * n + u) * W + i] : 0ull;
      const u64 vis = in ? visit[(size_t)u * W + i] : 0ull;
      cnt_lo += __popc(warp_transpose32((uint32_t)vis));
      cnt_hi += __popc(warp_transpose32((uint32_t)(vis >> 32)));
#pragma unroll
      for (int k = 0; k < kShallowBits; k++) {
        if (k >= nbits) break;
        sum_lo += (unsigned long long)__popc(warp_transpose32((uint32_t)x[k])) << k;
        sum_hi += (unsigned long long)__popc(warp_transpose32((uint32_t)(x[k] >> 32))) << k;
      }
    }
    if (cnt_lo) {
      atomicAdd(&s_cnt[64 * i + lane], cnt_lo);
      atomicAdd(&s_sum[64 * i + lane], (uint32_t)sum_lo);
    }
    if (cnt_hi) {
      atomicAdd(&s_cnt[64 * i + 32 + lane], cnt_hi);
      atomicAdd(&s_sum[64 * i + 32 + lane], (uint32_t)sum_hi);
    }
  }
  __syncthreads();
  const size_t row0 = (size_t)batch * 64 * W;
  for (int t = threadIdx.x; t < nb; t += blockDim.x) {
    if (s_sum[t]) atomicAdd(ctl->cc_sum + row0 + t, (unsigned long long)s_sum[t]);
    if (s_cnt[t]) atomicAdd(ctl->cc_cnt + row0 + t, (unsigned long long)s_cnt[t]);
  }
}

// Level mode of the final pass, shallow form (the batch ended below
// kDeepLevel): per 64 sources, for every level one word per vertex, the sources
// that reach it there, level after level (n words each) in their level block.
// top receives the deepest level of each 64.
template <int W>
__device__ __forceinline__ void emit_masks(const Team& tm, u64* out, const u64* visit, const u64* slices, int32_t n,
                                           int nbits, int levels, int (&top)[W]) {
  const size_t stride = tm.threads();
  for (size_t u = tm.thread(); u < (size_t)n; u += stride) {
#pragma unroll
    for (int i = 0; i < W; i++) {
      const u64 vis = visit[u * W + i];
      u64 s[kShallowBits];
#pragma unroll
      for (int k = 0; k < kShallowBits; k++) s[k] = k < nbits ? slices[((size_t)k * n + u) * W + i] : 0ull;
      for (int l = 0; l < levels; l++) {
        u64 x = vis;
#pragma unroll
        for (int k = 0; k < kShallowBits; k++) x &= (l >> k) & 1 ? s[k] : ~s[k];
        out[((size_t)i * 32 + l) * n + u] = x;
        if (x) top[i] = max(top[i], l);
      }
    }
  }
}
static_assert(kDeepLevel * sizeof(u64) <= 64 * sizeof(int32_t), "a level block holds every shallow level's words");

// Deep form: each vertex's levels for 64 sources as one 64-word row (-1 where
// unreached), and the lowest and highest level among them (INT_MAX / -1 when
// none).  Entries written during the traversal (src set, as in emit_vertex) are
// kept.
template <int W>
__device__ __forceinline__ void emit_levels(const Team& tm, const BsCtl* ctl, const u64* visit, const u64* slices,
                                            int32_t n, int nsrc, int nbits, const int32_t* __restrict__ src,
                                            int (&top)[W]) {
  const size_t stride = tm.threads();
#pragma unroll
  for (int i = 0; i < W; i++) {
    const int nb = min(64, nsrc - 64 * i);
    for (size_t u = tm.thread(); nb > 0 && u < (size_t)n; u += stride) {
      const u64 vis = visit[u * W + i];
      u64 any = 0ull;
      for (int k = 0; k < nbits; k++) any |= slices[((size_t)k * n + u) * W + i];
      int lo = 0x7fffffff, hi = -1;
      int4* row = reinterpret_cast<int4*>(ctl->lv_block + ((size_t)i * n + u) * 64);
      for (int s0 = 0; s0 < 64; s0 += 4) {
        int32_t v[4];
        int4 old = make_int4(0, 0, 0, 0);
        if (vis & ~any & (0xfull << s0)) old = row[s0 / 4];
        const int32_t kept[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int s = s0 + j;
          v[j] = -1;
          if (s < nb && ((vis >> s) & 1ull)) {
            int32_t x = 0;
            if (!((any >> s) & 1ull) && src[64 * i + s] != (int32_t)u) {
              x = kept[j];
            } else {
              for (int k = 0; k < nbits; k++) x |= (int32_t)((slices[((size_t)k * n + u) * W + i] >> s) & 1ull) << k;
            }
            v[j] = x;
            lo = min(lo, x);
            hi = max(hi, x);
          }
        }
        row[s0 / 4] = make_int4(v[0], v[1], v[2], v[3]);
      }
      int32_t* const range = ctl->lv_range + 2 * ((size_t)i * n + u);
      range[0] = lo;
      range[1] = hi;
      top[i] = max(top[i], hi);
    }
  }
}

// The deepest level of each 64 sources, one atomic per CTA.
template <int W>
__device__ __forceinline__ void record_depth(BsCtl* ctl, const int (&top)[W]) {
  __shared__ int deepest[W];
  if (threadIdx.x < W) deepest[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < W; i++) {
    const int t = __reduce_max_sync(kFull, top[i]);
    if (lane_id() == 0 && t > 0) atomicMax(&deepest[i], t);
  }
  __syncthreads();
  if (threadIdx.x < W && deepest[threadIdx.x] > 0) atomicMax(&ctl->depth[threadIdx.x], deepest[threadIdx.x]);
}

template <int W>
__device__ __forceinline__ void emit_batch(const BsArgs& a, const Team& tm) {
  const BsCtl* const ctl = a.ctl;
  const u64 *const visit = a.visit, *const slices = a.slices;
  const int32_t n = a.n;
  const int batch = batch_of(a);
  const int per = 64 * W;
  const int nb = min(per, ctl->nsrc - batch * per);
  // levels below kDeepLevel are in the slices; deeper ones were written out
  const int nbits = min(32 - __clz(max(ctl->level, 1)), kShallowBits);
  const int32_t* src = ctl->level >= kDeepLevel ? ctl->sources + (size_t)batch * per : nullptr;
  if (ctl->lv_block) {
    int top[W] = {};
    if (!src)
      emit_masks<W>(tm, reinterpret_cast<u64*>(ctl->lv_block), visit, slices, n, nbits, ctl->level, top);
    else
      emit_levels<W>(tm, ctl, visit, slices, n, nb, nbits, src, top);
    record_depth<W>(a.ctl, top);
    return;
  }
  if (ctl->cc_sum) {
    emit_closeness<W>(tm, ctl, batch, visit, slices, n, nb, nbits);
    return;
  }
  int32_t* dist = ctl->dist_base + (size_t)batch * per * n;
  const size_t t0 = tm.thread(), stride = tm.threads();
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(dist) & 15) == 0 && !src) {
    const size_t quads = (size_t)n / 4;
    int split = 1;  // of a word's bytes, while threads are idle
    while (split < 8 && quads * W * split < stride) split *= 2;
    const int bytes = 8 / split;
    for (size_t t = t0; t < quads * W * split; t += stride) {
      const size_t part = t / quads, u0 = 4 * (t - part * quads);
      const int i = (int)part / split, c0 = ((int)part % split) * bytes, c1 = c0 + bytes;
      switch (nbits) {
        case 1: emit_vertex4_packed<W, 1>(dist, n, nb, u0, visit, slices, i, c0, c1); break;
        case 2: emit_vertex4_packed<W, 2>(dist, n, nb, u0, visit, slices, i, c0, c1); break;
        case 3: emit_vertex4_packed<W, 3>(dist, n, nb, u0, visit, slices, i, c0, c1); break;
        case 4: emit_vertex4_packed<W, 4>(dist, n, nb, u0, visit, slices, i, c0, c1); break;
        default: emit_vertex4_packed<W, 5>(dist, n, nb, u0, visit, slices, i, c0, c1); break;
      }
    }
    return;
  }
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(dist) & 15) == 0) {
    for (size_t q = t0; q < (size_t)n / 4; q += stride) {
      switch (nbits) {
        case 1: emit_vertex4<W, 1>(dist, n, nb, 4 * q, visit, slices, src); break;
        case 2: emit_vertex4<W, 2>(dist, n, nb, 4 * q, visit, slices, src); break;
        case 3: emit_vertex4<W, 3>(dist, n, nb, 4 * q, visit, slices, src); break;
        case 4: emit_vertex4<W, 4>(dist, n, nb, 4 * q, visit, slices, src); break;
        default: emit_vertex4<W, 5>(dist, n, nb, 4 * q, visit, slices, src); break;
      }
    }
    return;
  }
  for (size_t u = t0; u < (size_t)n; u += stride) {
    switch (nbits) {
      case 1: emit_vertex<W, 1>(dist, n, nb, u, visit, slices, src); break;
      case 2: emit_vertex<W, 2>(dist, n, nb, u, visit, slices, src); break;
      case 3: emit_vertex<W, 3>(dist, n, nb, u, visit, slices, src); break;
      case 4: emit_vertex<W, 4>(dist, n, nb, u, visit, slices, src); break;
      default: emit_vertex<W, 5>(dist, n, nb, u, visit, slices, src); break;
    }
  }
}

// (kBsPush: both phases of a push)
enum : int32_t { kBsClear = 0, kBsInit, kBsScatter, kBsUpdate, kBsPull, kBsPush };

// One warp.  Ends the batch when the frontier is empty, otherwise picks
// the next level's variant: the forced one if set, else the learned
// selector if weights are loaded, else push while
// push_ratio x frontier edges < unfinished in-edges, dense once the
// frontier's edges reach n.
// Read through volatile loads: inside the persistent launch the counters
// that other CTAs raised may sit stale in this SM's L1.  All of them are read
// before lane 0 writes any (one round trip).  Returns whether the batch is
// done, else what the next level needs in `st`.
__device__ __forceinline__ bool decide_level(const BsArgs& a, BsStep& st) {
  BsCtl* const ctl = a.ctl;
  const float* sel_w = a.sel_w;
  const int32_t n = a.n;
  const int lane = lane_id();
  const volatile BsCtl* vc = ctl;
  const bool sel = vc->use_sel && sel_w;
  const int done = vc->done;
  const int L = vc->level;
  const int cur_mode = vc->mode, ul_cur = vc->ul_cur, hs_cur = vc->hs_cur;
  const int ul0 = vc->ul_size[0], ul1 = vc->ul_size[1], hs0 = vc->hs_size[0], hs1 = vc->hs_size[1];
  const long long mu = vc->mu - vc->mu_dec;
  const int policy = vc->policy, ratio = vc->push_ratio, force = vc->force, prev_nf = vc->prev_nf;
  const float sel_margin = vc->sel_margin;
  const long long m = vc->m;
  const int per = 64 * vc->width;
  const int nb = min(per, vc->nsrc - vc->batch * per);
  const int n_push = vc->n_push, n_pull = vc->n_pull;
  const int out = L % 3, old = (L + 2) % 3;  // the frontier this level wrote; the slot the next one clears
  const int qn = vc->aq_size[out], stale = vc->aq_size[old];
  const unsigned long long al = vc->alpack[out], al_old = vc->alpack[old];
  const bool unlisted = vc->unlisted[out] != 0, stale_unlisted = vc->unlisted[old] != 0;
  const long long mf = (long long)vc->mf[out];
  const int nf = qn + long_vertices(al);
  __syncwarp();
  if (done) return true;
  const bool pulled = cur_mode != kModePush;
  const int ul_next = pulled ? (ul_cur < 0 ? 0 : ul_cur ^ 1) : ul_cur;
  const int hs_next = pulled ? (hs_cur < 0 ? 0 : hs_cur ^ 1) : hs_cur;
  if (lane == 0) {
    if (!pulled) {
      ctl->n_push = n_push + 1;
    } else {
      ctl->n_pull = n_pull + 1;
      ctl->ul_cur = ul_next;
      ctl->ul_size[ul_next ^ 1] = 0;
      ctl->hs_cur = hs_next;
      ctl->hs_size[hs_next ^ 1] = 0;
    }
    ctl->mu = mu;
    ctl->mu_dec = 0;
    ctl->tq_size = 0;
    ctl->work = 0;
    ctl->hwork = 0;
  }
  if (nf == 0 || L >= n) {
    if (lane == 0) ctl->done = 1;
    return true;
  }
  int variant;
  if (policy == DAWN_VARIANT_PUSH || mf * ratio < mu) {
    // A push whose frontier edges reach n touches enough vertices that a
    // dense update sweep beats queueing every first touch (at n/16 the
    // sweeps of a 2048x2048 grid cost 35% more than the lists, and 6% more
    // on a kNN graph at n/1.5).
    variant = mf >= (long long)n ? kVarDense : kVarPush;
  } else {
    variant = kVarPull;
  }
  if (force) {
    variant = force - 1;
  } else if (sel) {
    float x[kSelIn];
    sel_features(x, (float)n, (float)m, (float)nf, (float)mf, (float)mu, (float)(L + 1), (float)prev_nf,
                 (float)nb);
    const unsigned allowed = policy == DAWN_VARIANT_PUSH ? (1u << kVarPush) | (1u << kVarDense) : 7u;
    variant = sel_pick(sel_w, x, allowed, variant, sel_margin);
  }
  if (unlisted) variant = kVarPull;  // no active list to push from (never with a forced variant)
  if (lane == 0) {
    // Level L+1 writes list (L+1)%3, whose stale frontier words level L cleared.
    ctl->aq_size[(L + 1) % 3] = 0;
    ctl->alpack[(L + 1) % 3] = 0;
    ctl->mf[(L + 1) % 3] = 0;
    ctl->unlisted[(L + 1) % 3] = 0;
    ctl->dense = variant == kVarDense;
    ctl->mode = variant == kVarPull ? kModePull : kModePush;
    ctl->prev_nf = nf;
    ctl->level = L + 1;
  }
  st.phase = variant == kVarPull ? kBsPull : kBsScatter;
  st.L = L + 1;
  st.dense = variant == kVarDense;
  st.qn = qn;
  st.ln = seg_count(al);
  st.stale = stale;
  st.stale_segs = seg_count(al_old);
  st.stale_unlisted = stale_unlisted;
  st.tn = 0;
  st.ul_cur = ul_next;
  st.un = ul_next < 0 ? a.ul_static_size : (ul_next ? ul1 : ul0);
  st.hs_cur = hs_next;
  st.hn = hs_next < 0 ? a.hv_segs : (hs_next ? hs1 : hs0);
  st.nf = nf;
  // Warp tasks of the level, for its CTAs: a vertex or 32 edges of a push,
  // eight rows or a segment of a pull, 128 words to clear (0: all CTAs).
  st.ctas = 0;
  long long work = max((long long)qn + seg_count(al), mf / 32);
  if (variant == kVarPull) work = (long long)st.un / 8 + st.hn;
  work = max(work, (long long)(clears_slot(stale, stale_unlisted, n) ? n : stale) / 128);
  if ((((unsigned)L + 2) & ((unsigned)L + 1)) == 0) work = max(work, (long long)n / 128);  // level L + 2 opens a slice
  if (variant != kVarDense) st.ctas = (int)min((long long)n, work + 1);
  return false;
}

// The running level's BsStep from the control block.
__device__ __forceinline__ BsStep read_step(const BsArgs& a) {
  const BsCtl* c = a.ctl;
  BsStep st = {};
  const int L = c->level, in = (L - 1) % 3, old = (L + 1) % 3;
  st.L = L;
  st.dense = c->dense;
  st.qn = c->aq_size[in];
  st.ln = seg_count(c->alpack[in]);
  st.stale = c->aq_size[old];
  st.stale_segs = seg_count(c->alpack[old]);
  st.stale_unlisted = c->unlisted[old];
  st.tn = c->tq_size;
  st.ul_cur = c->ul_cur;
  st.un = st.ul_cur < 0 ? a.ul_static_size : c->ul_size[st.ul_cur];
  st.hs_cur = c->hs_cur;
  st.hn = st.hs_cur < 0 ? a.hv_segs : c->hs_size[st.hs_cur];
  st.nf = st.qn + long_vertices(c->alpack[in]);
  return st;
}

// One thread: the batch's counters into the call's.
__device__ __forceinline__ void count_batch(BsCtl* ctl) {
  const volatile BsCtl* vc = ctl;
  ctl->total_reached = vc->total_reached + vc->reached;
  ctl->total_levels = vc->total_levels + vc->level;
  ctl->total_push = vc->total_push + vc->n_push;
  ctl->total_pull = vc->total_pull + vc->n_pull;
}

// --- one launch per step of a level (traced calls) ------------------------------

constexpr int kStepWarps = kBlock / 32;

__global__ void __launch_bounds__(kBlock) bs_clear(const __grid_constant__ BsArgs a) {
  clear_words(Team{(int)blockIdx.x, (int)gridDim.x}, a.words, a.nwords);
}
template <int W>
__global__ void bs_init(const __grid_constant__ BsArgs a) {
  init_batch<W>(a);
}
template <int W>
__global__ void __launch_bounds__(kBlock, W == 1 ? 5 : 4) bs_pull(const __grid_constant__ BsArgs a) {
  __shared__ BsSmem<kStepWarps> sm;
  if (a.ctl->done || a.ctl->mode != kModePull) return;
  pull_level<W>(a, Team{(int)blockIdx.x, (int)gridDim.x}, read_step(a), sm);
}
template <int W>
__global__ void __launch_bounds__(kBlock) bs_push_scatter(const __grid_constant__ BsArgs a) {
  __shared__ BsSmem<kStepWarps> sm;
  if (a.ctl->done || a.ctl->mode != kModePush) return;
  scatter_level<W>(a, Team{(int)blockIdx.x, (int)gridDim.x}, read_step(a), sm);
}
template <int W>
__global__ void __launch_bounds__(kBlock) bs_push_update(const __grid_constant__ BsArgs a) {
  __shared__ BsSmem<kStepWarps> sm;
  if (a.ctl->done || a.ctl->mode != kModePush) return;
  update_level<W>(a, Team{(int)blockIdx.x, (int)gridDim.x}, read_step(a), sm);
}
template <int W>
__global__ void __launch_bounds__(kBlock) bs_emit_dist(const __grid_constant__ BsArgs a) {
  emit_batch<W>(a, Team{(int)blockIdx.x, (int)gridDim.x});
}
__global__ void bs_decide(const __grid_constant__ BsArgs a) {
  BsStep st;
  decide_level(a, st);
}
__global__ void bs_next(const __grid_constant__ BsArgs a) {
  if (threadIdx.x != 0) return;
  count_batch(a.ctl);
  a.ctl->batch += 1;
}

// --- the persistent launch ----------------------------------------------------------

// Vertices and entries per CTA of a small graph: 1024 / 4096, 64 sources: grid 40 x
// 60 880 / 1006 us, kNN of 2,127 points 545 / 593, RMAT-12 107 / 114.
constexpr int kBsEntries = 1024;

// CTAs for `work` warp tasks.
__device__ __forceinline__ int bs_ctas(int work, int warps) {
  const int c = (work + warps - 1) / warps;
  return c < 1 ? 1 : min(c, (int)gridDim.x);
}

// One warp of the last CTA to finish phase st; every other participant has
// arrived and the rest only poll.  Turns st into the next phase; returns false
// when the batch is done.
// Not inlined: its registers would be the levels' spills.
template <bool kThin, int kWarps>
__device__ __noinline__ bool next_phase(const BsArgs& a, BsStep& step) {
  BsStep st = step;
  BsCtl* const ctl = a.ctl;
  const volatile BsCtl* vc = ctl;
  if (st.phase == kBsClear) {
    if (lane_id() == 0) ctl->batch = a.batch;
    st.phase = kBsInit;
    st.ctas = 1;
    step = st;
    return true;
  }
  if (st.phase == kBsScatter) {
    st.tn = vc->tq_size;
    st.phase = kBsUpdate;
    st.ctas = st.dense ? (int)gridDim.x : bs_ctas((st.tn + 3) / 4, kWarps);
    step = st;
    return true;
  }
  if (st.phase == kBsInit) {
    const uint32_t arrived = st.arrived;
    __threadfence();
    st = read_step(a);
    st.arrived = arrived;
    st.phase = vc->mode != kModePush ? kBsPull : kThin && !st.dense ? kBsPush : kBsScatter;
    st.ctas = (int)gridDim.x;
    step = st;
    return true;
  }
  if (decide_level(a, st)) {
    if (lane_id() == 0) count_batch(ctl);
    return false;
  }
  if (kThin && st.phase == kBsScatter && !st.dense) st.phase = kBsPush;
  st.ctas = st.ctas ? bs_ctas(st.ctas, kWarps) : (int)gridDim.x;
  step = st;
  return true;
}

constexpr int kStepWords = 9;
__device__ __forceinline__ u64 pack_step(const BsStep& st, int i) {
  const uint32_t lo[kStepWords] = {(uint32_t)st.L, (uint32_t)st.qn, (uint32_t)st.ln, (uint32_t)st.stale,
                                   (uint32_t)st.stale_segs, (uint32_t)(st.phase == kBsPull ? st.un : st.tn),
                                   (uint32_t)st.hn, (uint32_t)st.nf, st.arrived};
  const uint32_t hi = i == 0 ? (uint32_t)st.ctas
                             : (uint32_t)(st.phase | st.dense << 3 | st.stale_unlisted << 4 | (st.ul_cur + 1) << 5 |
                                          (st.hs_cur + 1) << 7);
  uint32_t x = lo[0];
#pragma unroll
  for (int k = 1; k < kStepWords; k++) x = i == k ? lo[k] : x;
  return (u64)(hi & 0xffffu) << 32 | x;
}
__device__ __forceinline__ BsStep unpack_step(const u64* w) {
  BsStep st;
  const uint32_t f = (uint32_t)(w[1] >> 32) & 0xffffu;
  st.ctas = (int)((w[0] >> 32) & 0xffffu);
  st.phase = f & 7;
  st.dense = (f >> 3) & 1;
  st.stale_unlisted = (f >> 4) & 1;
  st.ul_cur = (int)((f >> 5) & 3) - 1;
  st.hs_cur = (int)((f >> 7) & 3) - 1;
  st.L = (int)(uint32_t)w[0];
  st.qn = (int)(uint32_t)w[1];
  st.ln = (int)(uint32_t)w[2];
  st.stale = (int)(uint32_t)w[3];
  st.stale_segs = (int)(uint32_t)w[4];
  st.tn = st.un = (int)(uint32_t)w[5];
  st.hn = (int)(uint32_t)w[6];
  st.nf = (int)(uint32_t)w[7];
  st.arrived = (uint32_t)w[8];
  return st;
}

// One batch in one cooperative launch: clear, seed, levels (the distances
// follow in a launch of their own, whose 89 registers would cost this one its
// occupancy).  As launches in a conditional graph a level was four kernels, of
// which one or two returned at once: 12 to 20 us before any work, the bound of
// every batch with small or many levels.  Here a step of a level ends with one
// block barrier and one arrival per CTA, and about 2 us in the last CTA for the
// decision; steps with little work name fewer CTAs, the others poll.  The CTAs
// keep the occupancy of the per-level pull: 1,280 threads per SM at 48
// registers (W = 1), 1,024 at 64.  Per call, graph form -> this:
//   Erdos-Renyi, 65,536 vertices, 64 sources   201 -> 132 us
//   RMAT-16, 64 sources                         254 -> 164
//   RMAT-18, 500 sources                       1068 -> 860
//   RMAT-22, 64 sources                        1176 -> 1128
//   grid 700 x 700, 64 sources                26060 -> 22050
//   kNN, 200,000 vertices, 64 sources         16050 -> 7450
// kThin: list-mode pushes as one phase (push_level), for graphs whose rows are all
// short.  A kernel of its own: beside it the pull loses registers, and 3 to 7% on
// RMAT graphs, whose thin levels are few.
template <int W, bool kThin = false>
__global__ void __launch_bounds__(W == 1 ? 640 : 512, 2) bs_traverse(const __grid_constant__ BsArgs a) {
  constexpr int kWarps = (W == 1 ? 640 : 512) / 32;
  __shared__ BsSmem<kWarps> sm;
  BsCtl* const ctl = a.ctl;
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  // no phase can open before every CTA has arrived, so all read the same
  uint32_t gen = (uint32_t)(*static_cast<const volatile unsigned long long*>(&ctl->sync.word[0]) >> 48);
  const BsStep& st = sm.st;  // in shared memory: its fields would cost the levels their registers
  if (threadIdx.x == 0) {
    sm.st = BsStep{};
    sm.st.phase = kBsClear;
    sm.st.ctas = *static_cast<const volatile uint32_t*>(&ctl->sync.broken) ? 0 : (int)gridDim.x;
    sm.st.arrived = (uint32_t)*static_cast<const volatile unsigned long long*>(&ctl->sync.word[8]);
  }
  __syncthreads();
  if (st.ctas == 0) return;
  for (;;) {
    const Team tm{(int)blockIdx.x, st.ctas};
    switch (st.phase) {
      case kBsClear: clear_words(tm, a.words, a.nwords); break;
      case kBsInit: init_batch<W>(a); break;
      case kBsScatter: scatter_level<W>(a, tm, st, sm); break;
      case kBsUpdate: update_level<W>(a, tm, st, sm); break;
      case kBsPush:
        if constexpr (kThin) push_level(a, tm, st, sm);
        break;
      default: pull_level<W>(a, tm, st, sm);
    }
    __syncthreads();
    if (wib == 0) {
      int last = 0;
      if (lane == 0) {
        __threadfence();
        last = atomicAdd(&ctl->arrive.n, 1u) + 1 == st.arrived + (uint32_t)st.ctas;
      }
      if (__shfl_sync(kFull, last, 0)) {
        __threadfence();
        if (lane == 0) {
          sm.next = st;
          sm.next.arrived = st.arrived + (uint32_t)st.ctas;
        }
        __syncwarp();
        const bool more = next_phase<kThin, kWarps>(a, sm.next);
        __syncwarp();
        if (!more && lane == 0) sm.next.ctas = 0;
        const u64 tag = (u64)((gen + 1) & 0xffffu) << 48;
        __syncwarp();
        __threadfence();
        if (lane < kStepWords) *static_cast<volatile unsigned long long*>(&ctl->sync.word[lane]) = tag | pack_step(sm.next, lane);
      }
      __syncwarp();
      bool idle = false;
      for (uint32_t polls = 0;; polls++) {
        u64 w;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(&ctl->sync.word[lane < kStepWords ? lane : 0]) : "memory");
        const uint32_t tag = (uint32_t)(w >> 48), tag0 = __shfl_sync(kFull, tag, 0);
        if (__all_sync(kFull, tag == tag0) && tag != gen) {
          gen = tag;
          polls = 0;
          const uint32_t ctas = (uint32_t)(__shfl_sync(kFull, w, 0) >> 32) & 0xffffu;
          if (ctas == 0 || blockIdx.x < ctas) {
            if (lane < kStepWords) sm.word[lane] = w;
            __syncwarp();
            if (lane == 0) sm.st = unpack_step(sm.word);
            break;
          }
          idle = true;
        }
        if (polls == a.polls) {
          if (lane == 0) {
            *a.err = DAWN_ERR_TIMEOUT;
            *static_cast<volatile uint32_t*>(&ctl->sync.broken) = 1;
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

void probe_bs(const void* p, LevelProbe* out) {
  const BsCtl* c = static_cast<const BsCtl*>(p);
  const int pin = (c->level - 1) % 3;
  out->level = c->level;
  out->mode = c->mode;
  out->done = c->done;
  out->frontier = c->aq_size[pin] + (int64_t)(c->alpack[pin] >> 32);
  out->frontier_edges = (int64_t)c->mf[pin];
  out->unvisited_edges = c->mu;
}

// Static pull lists.  Light rows (0 < in-degree < 2 x seg) are swept in
// id order, 32 per warp task; heavy rows are cut into seg-entry
// segments, one warp task each, so a hub row that cannot stop early is
// spread over many warps instead of holding one warp for the whole level.
__global__ void flag_rows(const int32_t* __restrict__ t_row_ptr, int32_t n, int heavy, int seg,
                          int64_t* __restrict__ flags, int64_t* __restrict__ segs) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += stride) {
    const int d = t_row_ptr[i + 1] - t_row_ptr[i];
    const bool h = d >= 2 * seg;
    flags[i] = heavy ? h : (d > 0 && !h);
    if (segs) segs[i] = h ? (d + seg - 1) / seg : 0;
  }
}

__global__ void scatter_flagged(const int64_t* __restrict__ flags, const int64_t* __restrict__ pos, int32_t n,
                                int32_t* __restrict__ out, const int64_t* __restrict__ segpos,
                                int32_t* __restrict__ segoff) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += stride)
    if (flags[i]) {
      out[pos[i]] = (int32_t)i;
      if (segoff) segoff[pos[i]] = (int32_t)segpos[i];
    }
}

}  // namespace

// Static pull lists of the in-edge CSR (shared with the weighted pull).
dawn_status build_static_list(dawn_graph* g) {
  if (g->ul_static.p && g->static_seg == g->pull_seg) return DAWN_OK;
  // Captured traversal graphs (weighted, level by level) hold these
  // lists' addresses and sizes; a rebuild for a new segment size may move
  // or resize them.
  if (g->ul_static.p) drop_graphs(g);
  const int seg = g->pull_seg;
  const int32_t n = g->n;
  const size_t n1 = (size_t)n + 1;
  int64_t* tmp = nullptr;
  DAWN_CHECK(pool_alloc((void**)&tmp, sizeof(int64_t) * 4 * n1, g->stream));
  int64_t *flags = tmp, *pos = tmp + n1, *segs = tmp + 2 * n1, *segpos = tmp + 3 * n1;
  int64_t cnt[2] = {0, 0}, nseg = 0;
  DAWN_CHECK(ensure(g->ul_static, sizeof(int32_t) * (size_t)n, g->stream));
  DAWN_CHECK(ensure(g->hv_static, sizeof(int32_t) * (size_t)n, g->stream));
  DAWN_CHECK(ensure(g->hv_segoff, sizeof(int32_t) * n1, g->stream));
  for (int heavy = 0; heavy < 2; heavy++) {
    flag_rows<<<g->geo.sms * 4, kBlock, 0, g->stream>>>(g->t_row_ptr, n, heavy, seg, flags, heavy ? segs : nullptr);
    DAWN_CUDA(cudaGetLastError());
    DAWN_CUDA(cudaMemsetAsync(flags + n, 0, sizeof(int64_t), g->stream));
    DAWN_CHECK(exclusive_scan_i64(flags, pos, (int64_t)n1, g->stream));
    if (heavy) {
      DAWN_CUDA(cudaMemsetAsync(segs + n, 0, sizeof(int64_t), g->stream));
      DAWN_CHECK(exclusive_scan_i64(segs, segpos, (int64_t)n1, g->stream));
    }
    scatter_flagged<<<g->geo.sms * 4, kBlock, 0, g->stream>>>(
        flags, pos, n, heavy ? g->hv_static.as<int32_t>() : g->ul_static.as<int32_t>(), heavy ? segpos : nullptr,
        heavy ? g->hv_segoff.as<int32_t>() : nullptr);
    DAWN_CUDA(cudaGetLastError());
    DAWN_CUDA(cudaMemcpyAsync(&cnt[heavy], pos + n, sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream));
    if (heavy) DAWN_CUDA(cudaMemcpyAsync(&nseg, segpos + n, sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream));
    DAWN_CUDA(cudaStreamSynchronize(g->stream));
  }
  // closing offset of the heavy segment prefix
  const int32_t total = (int32_t)nseg;
  DAWN_CUDA(cudaMemcpyAsync(g->hv_segoff.as<int32_t>() + cnt[1], &total, sizeof(int32_t), cudaMemcpyHostToDevice,
                            g->stream));
  const size_t acc_bytes = sizeof(u64) * acc_stride(kMaxW) * (size_t)(cnt[1] > 0 ? cnt[1] : 1);
  DAWN_CHECK(ensure(g->hv_acc, acc_bytes, g->stream));
  DAWN_CHECK(ensure(g->hv_tasks, sizeof(int2) * 2 * (size_t)(nseg > 0 ? nseg : 1), g->stream));
  DAWN_CUDA(cudaMemsetAsync(g->hv_acc.p, 0, acc_bytes, g->stream));
  pool_free(tmp, g->stream);
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  g->ul_static_size = (int32_t)cnt[0];
  g->hv_count = (int32_t)cnt[1];
  g->hv_segs = (int32_t)nseg;
  g->static_seg = seg;
  return DAWN_OK;
}

namespace {
int slice_count(int32_t n) { return std::min(32 - __builtin_clz((unsigned)n), kShallowBits); }
}  // namespace

// words (per vertex w each): visit | fr[3] | nxt | level slices
dawn_status bitset_reserve(dawn_graph* g, int w) {
  return ensure(g->bs_words, sizeof(u64) * w * (5 + (size_t)slice_count(g->n)) * (size_t)g->n, g->stream);
}

namespace {

template <int W>
dawn_status run_width(dawn_graph* g, const int32_t* sources, int32_t nsrc, int32_t* d_dist,
                      unsigned long long* cc_sum, unsigned long long* cc_cnt, int32_t* lv_block = nullptr,
                      int32_t* lv_range = nullptr) {
  const int32_t n = g->n;
  const size_t nn = (size_t)n;
  DAWN_CHECK(build_static_list(g));
  if (reinterpret_cast<uintptr_t>(g->t_col) % 32 != 0) {  // the pull's 256-bit column loads
    set_error("in-edge column array is not 32-byte aligned");
    return DAWN_ERR_CUDA;
  }
  // words (per vertex W each): visit | fr[3] | nxt | level slices[nbits]
  // lists: aq[3] | tq | ul[2] | touched bitmap ; segments[3]
  // Levels never exceed n, and levels from kDeepLevel on bypass the slices.
  const int nbits = slice_count(n);
  DAWN_CHECK(bitset_reserve(g, W));
  const bool fresh = g->bs_queues.p == nullptr;
  DAWN_CHECK(ensure(g->bs_queues, sizeof(int32_t) * 6 * nn + sizeof(uint32_t) * (nn / 32 + 1), g->stream));
  // The touched bitmap starts clear; list-mode updates clear what they set.
  if (fresh)
    DAWN_CUDA(cudaMemsetAsync(g->bs_queues.as<int32_t>() + 6 * nn, 0, sizeof(uint32_t) * (nn / 32 + 1), g->stream));
  const size_t segcap = seg_capacity(n, g->m);
  DAWN_CHECK(ensure(g->bs_segs, sizeof(Seg) * 3 * segcap, g->stream));
  // one upload: the control block, then the sources
  const size_t up_bytes = sizeof(BsCtl) + sizeof(int32_t) * (size_t)nsrc;
  DAWN_CHECK(ensure(g->bs_ctl, up_bytes, g->stream));
  BsCtl c = {};
  c.nsrc = nsrc;
  c.policy = DAWN_VARIANT_BITSET;
  c.push_ratio = g->bs_ratio_set ? g->bs_push_ratio : default_push_ratio(g);
  c.nbits = nbits;
  c.width = W;
  c.dist_base = d_dist;
  c.sources = reinterpret_cast<const int32_t*>(g->bs_ctl.as<BsCtl>() + 1);
  c.cc_sum = cc_sum;
  c.cc_cnt = cc_cnt;
  c.lv_block = lv_block;
  c.lv_range = lv_range;
  c.use_sel = g->sel_call;
  c.sel_margin = g->sel_margin;
  c.force = g->force_variant;
  c.m = g->m;
  std::vector<unsigned char> up(up_bytes);
  std::memcpy(up.data(), &c, sizeof(c));
  std::memcpy(up.data() + sizeof(c), sources, sizeof(int32_t) * (size_t)nsrc);
  // pageable: staged before the call returns
  DAWN_CUDA(cudaMemcpyAsync(g->bs_ctl.p, up.data(), up_bytes, cudaMemcpyHostToDevice, g->stream));

  BsArgs a = {};
  a.sel_w = g->sel_slot.as<float>();
  a.ctl = g->bs_ctl.as<BsCtl>();
  a.row_ptr = g->row_ptr;
  a.col = g->col;
  a.t_row_ptr = g->t_row_ptr;
  a.t_col = g->t_col;
  a.ul_static = g->ul_static.as<int32_t>();
  a.ul_static_size = g->ul_static_size;
  a.hv_static = g->hv_static.as<int32_t>();
  a.hv_segoff = g->hv_segoff.as<int32_t>();
  a.hv_acc = g->hv_acc.as<u64>();
  a.hv_tasks = g->hv_tasks.as<int2>();
  a.hv_count = g->hv_count;
  a.hv_segs = g->hv_segs;
  a.pull_seg = g->pull_seg;
  a.words = g->bs_words.as<u64>();
  a.visit = a.words;
  a.fr = a.words + W * nn;
  a.nxt = a.words + 4 * W * nn;
  a.slices = a.words + 5 * W * nn;
  a.aq = g->bs_queues.as<int32_t>();
  a.tq = a.aq + 3 * nn;
  a.ul = a.aq + 4 * nn;
  a.tbm = reinterpret_cast<uint32_t*>(a.aq + 6 * nn);
  a.segs = g->bs_segs.as<Seg>();
  a.segcap = segcap;
  a.nwords = W * (5 + (size_t)(nbits < kSlicesCleared ? nbits : kSlicesCleared)) * nn;
  a.n = n;
  a.m = g->m;
  a.nbits = nbits;
  a.force = g->force_variant;
  a.batch = -1;
  a.polls = g->wait_polls;
  a.err = g->h_err;
  a.dist_base = d_dist;
  a.lv_block = lv_block;
  a.cc_sum = cc_sum;
  const int nbatches = (nsrc + 64 * W - 1) / (64 * W);
  void* args[] = {&a};
  const int sms = g->geo.sms;
  const int emit_ctas = cc_sum ? std::max(sms * kClosenessCtas, kClosenessMin) : sms * 8;
  SsFamily fam;
  if (g->l2_persist) {
    // the three rotating frontier slots: every pull level gathers from one
    fam.l2_base = a.fr;
    fam.l2_bytes = sizeof(u64) * 3 * W * nn;
  }
  if (!g->trace) {
    const void* fn = (const void*)bs_traverse<W>;
    if constexpr (W == 1) {
      DAWN_CHECK(longest_row(g));
      if (g->max_row < kLongRow) fn = (const void*)bs_traverse<1, true>;
    }
    const int threads = W == 1 ? 640 : 512;
    // a small graph takes few CTAs: each adds to the arrivals of its phases
    const int64_t want = ((int64_t)n + g->m) / kBsEntries + 1;
    const int full = persistent_blocks(fn, threads, 0, g->blocks_per_sm);
    const int ctas = want < full ? (int)want : full;
    for (a.batch = 0; a.batch < nbatches; a.batch++) {
      DAWN_CHECK(launch_cooperative(fam, fn, ctas, threads, args, g->stream));
      DAWN_CUDA(cudaLaunchKernel((const void*)bs_emit_dist<W>, dim3(emit_ctas), dim3(kBlock), args, 0, g->stream));
    }
    return DAWN_OK;
  }
  const Launch step[] = {
      {(const void*)bs_clear, args, dim3(sms * 8), dim3(kBlock), "bs_clear"},
      {(const void*)bs_init<W>, args, dim3(1), dim3(64 * W), "bs_init"},
      {(const void*)bs_pull<W>, args, dim3(persistent_blocks((const void*)bs_pull<W>, kBlock, 0, g->blocks_per_sm)),
       dim3(kBlock), "bs_pull", kModePull},
      {(const void*)bs_push_scatter<W>, args,
       dim3(persistent_blocks((const void*)bs_push_scatter<W>, kBlock, 0, g->blocks_per_sm)), dim3(kBlock),
       "bs_push_scatter", kModePush},
      {(const void*)bs_push_update<W>, args,
       dim3(persistent_blocks((const void*)bs_push_update<W>, kBlock, 0, g->blocks_per_sm)), dim3(kBlock),
       "bs_push_update", kModePush},
      {(const void*)bs_decide, args, dim3(1), dim3(32), "bs_decide"},
      {(const void*)bs_emit_dist<W>, args, dim3(emit_ctas), dim3(kBlock), "bs_emit_dist"},
      {(const void*)bs_next, args, dim3(1), dim3(32), "bs_next"}};
  fam.npre = 2;
  fam.nbody = 4;
  fam.npost = 2;
  for (int i = 0; i < 2; i++) fam.pre[i] = step[i];
  for (int i = 0; i < 4; i++) fam.body[i] = step[2 + i];
  for (int i = 0; i < 2; i++) fam.post[i] = step[6 + i];
  fam.ctl = a.ctl;
  fam.ctl_bytes = sizeof(BsCtl);
  fam.probe = probe_bs;
  return ss_run_traced(g, fam, nbatches);
}

}  // namespace

// 2 from 16 entries a vertex on: there a push, which reads a frontier's rows once,
// beats a pull of half as many entries (4 / 2: RMAT-18, 500 sources 859 / 794 us,
// closeness of 1,000 1798 / 1670, RMAT-16 x 64 168 / 149; RMAT-22 and Erdos-Renyi
// the same; grid 60 x 40 x 20 1165 / 1184).
int default_push_ratio(const dawn_graph* g) { return g->m < 16 * (int64_t)g->n ? kPushRatio : 2; }

int bitset_width(const dawn_graph* g, int32_t nsrc) {
  if (g->bs_width > 0) return g->bs_width;
  if (nsrc > 128) return 4;
  if (nsrc > 64) return 2;
  return 1;
}

dawn_status bfs_bitset(dawn_graph* g, const int32_t* sources, int32_t nsrc, int32_t* d_dist,
                       unsigned long long* cc_sum, unsigned long long* cc_cnt) {
  const int w = bitset_width(g, nsrc);
  if (w == 4) return run_width<4>(g, sources, nsrc, d_dist, cc_sum, cc_cnt);
  if (w == 2) return run_width<2>(g, sources, nsrc, d_dist, cc_sum, cc_cnt);
  return run_width<1>(g, sources, nsrc, d_dist, cc_sum, cc_cnt);
}

dawn_status bfs_bitset_levels(dawn_graph* g, int w, const int32_t* sources, int32_t nsrc, int32_t* d_levels,
                              int32_t* d_range, int32_t* h_end) {
  if (nsrc < 1 || nsrc > 64 * w) {
    set_error("level mode takes one batch of sources per call");
    return DAWN_ERR_INVALID_ARG;
  }
  if (w == 4)
    DAWN_CHECK(run_width<4>(g, sources, nsrc, nullptr, nullptr, nullptr, d_levels, d_range));
  else if (w == 2)
    DAWN_CHECK(run_width<2>(g, sources, nsrc, nullptr, nullptr, nullptr, d_levels, d_range));
  else
    DAWN_CHECK(run_width<1>(g, sources, nsrc, nullptr, nullptr, nullptr, d_levels, d_range));
  static_assert(offsetof(BsCtl, depth) == offsetof(BsCtl, level) + sizeof(int32_t) && kMaxW == 4, "five words");
  DAWN_CUDA(cudaMemcpyAsync(h_end, &g->bs_ctl.as<BsCtl>()->level, kLevelsEnd * sizeof(int32_t),
                            cudaMemcpyDeviceToHost, g->stream));
  return DAWN_OK;
}

dawn_status bfs_bitset_stats(dawn_graph* g, dawn_stats* st, int32_t nsrc) {
  BsCtl h;
  DAWN_CUDA(cudaMemcpyAsync(&h, g->bs_ctl.p, sizeof(BsCtl), cudaMemcpyDeviceToHost, g->stream));
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  DAWN_CHECK(device_status(g));
  st->edges_traversed = (int64_t)h.total_reached;
  st->levels = h.total_levels;
  st->push_levels = h.total_push;
  st->pull_levels = h.total_pull;
  st->batches = (nsrc + 64 * h.width - 1) / (64 * h.width);
  return DAWN_OK;
}

}  // namespace dawn
