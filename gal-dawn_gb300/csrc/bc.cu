// BCDAWN betweenness on sm_103a.
//
// The reference computes it on the CPU only (src/algorithm/cpu/bc.cpp:9-191;
// include/dawn/algorithm/gpu/bc.cuh is empty), one source at a time.  Its
// dependency for a source s, with levels counted from s:
//   * a vertex c at level >= 2 has amount(c) predecessor entries: CSR
//     entries j -> c with level(j) = level(c) - 1 (duplicates count);
//   * delta(v) = sum over v's entries v -> c with level(c) = level(v) + 1 of
//     1 / amount(c) + delta(c);
//   * the betweenness of v is the sum of delta(v) over the sources.
// Sources go 64 together, and up to four such blocks through each pass (grid
// y): one traversal serves all of them, and a level's few heavy rows or its last
// wave leave fewer SMs idle.  For 64 sources:
//   1. the batched bitset traversal leaves, per level, one 64-bit word per
//      vertex: the sources that reach it at that level (M[l]);
//   2. bc_amount: for each in-edge j -> c the sources whose shortest paths use
//      it, OR over c's levels l of M[l][c] & M[l - 1][j], counted per source;
//      it stores 1 / amount per source;
//   3. bc_sweep, from the deepest level up: for level l and every out-edge
//      v -> c with M[l][v] & M[l + 1][c] not empty, the term 1 / amount(c) +
//      delta(c) of those sources is summed into v; the sum is added to v's own
//      term (which then holds 1 / amount + delta) and to its betweenness.
//      Terms of level l + 1 are final when level l runs, and every (vertex,
//      source) slot is written by one warp in one sweep, so no atomics are
//      needed.
// What bounds it is the 256-byte term row of an edge, read from L2; the words
// tell which edges need it.  On RMAT-16 with 64 sources 2.4 M rows are read of
// the 4.7 M edges that the sweeps pass, in part only (9.7 M sectors).  With
// level rows (256 bytes an edge too) beside every term row the passes of a
// block took 580 us, now 200 (of three blocks together); the sweep of the widest
// level moves 0.7 sectors per SM clock, near what L1/TEX gathers reach.  Batches
// of kDeepLevel levels and more have no such words: they have level rows, and on
// graphs of short rows go by pairs (bc_pairs).
// Rows of at least kHeavy entries (the hubs of power-law graphs) would keep
// one warp busy for thousands of dependent row loads while the rest of the
// grid idles, so they are cut into kBcSeg-entry segments, each a warp task
// of its own: in-row segments add their counts to a per-row counter
// (integers, so the order does not matter), out-row segments write their
// partial sums to a slot of their own.  The warp that finishes a row's last
// segment ends the row (with level rows: a second kernel per pass), adding the
// partials in segment order.
// Terms are float (the reference's bc_temp is float); the sums over
// sources are double.  The additions group as (1 / amount + delta) per
// entry, and a heavy row's sum by segments, rather than the reference's
// sequence, so values agree with it to float rounding, not bit for bit.
#include <algorithm>
#include <cstring>
#include <vector>

#include "dawn_device.cuh"

namespace dawn {
namespace {

constexpr int kLanes = 64;
constexpr int kUnroll = 4;
constexpr int kRows = 8;     // term rows a warp has in flight
constexpr int kHeavy = 128;  // rows of at least this many entries are cut into segments
constexpr int kBcSeg = 64;   // entries per segment

// Rows cut into segments: per row its first segment, and per segment its row,
// vertex, first entry and length (the search for them was 12 dependent loads a
// task).
struct HeavyRows {
  const int4* seg;     // segs entries: row index, vertex, first entry, entries
  const int32_t* v;    // count entries
  const int32_t* off;  // count + 1 entries, off[count] = segs
  int32_t count, segs;
};

// Warp task t: vertices 0..n-1 whose rows are short, then the segments of
// the heavy rows.  Sets the vertex, the CSR range and the heavy row index
// (-1 for a short row); false for a heavy vertex's own task (its segments
// cover it).
__device__ __forceinline__ bool task_range(int t, int32_t n, const int32_t* __restrict__ rp, const HeavyRows& h,
                                           int32_t& v, int& ks, int& ke, int& hidx, int& seg) {
  if (t < n) {
    v = t;
    ks = rp[t];
    ke = rp[t + 1];
    hidx = -1;
    seg = -1;
    return ke - ks < kHeavy;
  }
  seg = t - n;
  const int4 hv = __ldg(h.seg + seg);
  hidx = hv.x;
  v = hv.y;
  ks = hv.z;
  ke = hv.z + hv.w;
  return true;
}

// --- batches below kDeepLevel: level words -----------------------------------------

using u64 = unsigned long long;

// 32 x 32 bit transpose across a warp: bit e of lane s's result = bit s of
// lane e's input.
__device__ __forceinline__ uint32_t transpose32(uint32_t x) {
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

// Light rows go to warps in chunks of `per` vertices whose entries are laid
// end to end, one entry per lane: a row of three entries then costs three
// lanes, not a warp's round trips.
// Vertices per chunk: enough chunks for every warp of the grid.
__host__ __device__ inline int chunk_rows(int32_t n, int warps) {
  int per = 32;
  while (per > 1 && (n + per - 1) / per < warps) per >>= 1;
  return per;
}

// The warp that finishes the last of a heavy row's segments.
__device__ __forceinline__ bool last_segment(int32_t* done, int segs) {
  __syncwarp();
  __threadfence();
  int last = 0;
  if (lane_id() == 0) {
    last = atomicAdd(done, 1) == segs - 1;
    if (last) *done = 0;
  }
  last = __shfl_sync(kFull, last, 0);
  if (last) __threadfence();
  return last;
}

// 1 / amount of every (vertex, source) slot at level 2 or deeper.  `levels`
// counts level 0 in.
__global__ void __launch_bounds__(kBlock) bc_amount(const int32_t* __restrict__ t_row_ptr,
                                                    const int32_t* __restrict__ t_col, const u64* __restrict__ M,
                                                    float* __restrict__ T, int32_t n, int32_t levels, int32_t per,
                                                    HeavyRows h, int32_t* __restrict__ cnt, int32_t* __restrict__ done) {
  const int lane = lane_id();
  const size_t nn = (size_t)n;
  M += blockIdx.y * nn * 32;
  T += blockIdx.y * nn * kLanes;
  cnt += (size_t)blockIdx.y * h.count * kLanes;
  done += (size_t)blockIdx.y * h.count;
  const int chunks = (n + per - 1) / per;
  for (int t = global_warp(); t < h.segs + chunks; t += num_warps()) {
    if (t < h.segs) {
      const int4 hv = __ldg(h.seg + t);
      const int hidx = hv.x;
      const int32_t c = hv.y;
      const u64 w = lane >= 2 && lane < levels ? __ldg(M + lane * nn + c) : 0ull;  // lane l: level l
      const unsigned set = __ballot_sync(kFull, w != 0ull);
      if (!set) continue;
      const uint32_t ra = __reduce_or_sync(kFull, (uint32_t)w), rb = __reduce_or_sync(kFull, (uint32_t)(w >> 32));
      const int s0 = __ldg(h.off + hidx), s1 = __ldg(h.off + hidx + 1);
      const int ks = hv.z, ke = ks + hv.w;
      int ca = 0, cb = 0;
      for (int kb = ks; kb < ke; kb += 32) {
        const int k = kb + lane;
        const int32_t j = k < ke ? __ldg(t_col + k) : -1;
        u64 p = 0ull;
        for (unsigned b = set; b; b &= b - 1) {
          const int l = __ffs(b) - 1;
          const u64 wl = __shfl_sync(kFull, w, l);
          if (j >= 0) p |= wl & __ldg(M + (l - 1) * nn + j);
        }
        ca += __popc(transpose32((uint32_t)p));
        cb += __popc(transpose32((uint32_t)(p >> 32)));
      }
      int32_t* const cr = cnt + (size_t)hidx * kLanes;
      if (ca) atomicAdd(cr + lane, ca);
      if (cb) atomicAdd(cr + lane + 32, cb);
      if (!last_segment(done + hidx, s1 - s0)) continue;
      ca = __ldcg(cr + lane);
      cb = __ldcg(cr + lane + 32);
      cr[lane] = 0;
      cr[lane + 32] = 0;
      float* const Tc = T + (size_t)c * kLanes;
      if ((ra >> lane) & 1u) Tc[lane] = ca ? 1.0f / (float)ca : 0.0f;
      if ((rb >> lane) & 1u) Tc[lane + 32] = cb ? 1.0f / (float)cb : 0.0f;
      continue;
    }
    const int32_t c0 = (t - h.segs) * per, c = c0 + lane;
    const bool in = lane < per && c < n;
    const int32_t ks = in ? t_row_ptr[c] : 0;
    int32_t deg = in ? t_row_ptr[c + 1] - ks : 0;
    if (deg >= kHeavy) deg = 0;
    unsigned set = 0;
    u64 reach = 0ull;
    for (int l = 2; l < levels; l++) {
      const u64 w = deg ? __ldg(M + l * nn + c) : 0ull;
      reach |= w;
      if (__any_sync(kFull, w != 0ull)) set |= 1u << l;
    }
    if (!set) continue;
    if (!reach) deg = 0;
    const RowChunk ch(ks, deg);
    int ca = 0, cb = 0;
    for (int f0 = 0; f0 < ch.total; f0 += 32) {
      const int f = f0 + lane;
      const int q = ch.row(f);
      const int32_t k = __shfl_sync(kFull, ch.ks, q) + f - __shfl_sync(kFull, ch.off, q);
      u64 p = 0ull;
      if (f < ch.total) {
        const int32_t j = __ldg(t_col + k);
        for (unsigned b = set; b; b &= b - 1) {
          const int l = __ffs(b) - 1;
          p |= __ldg(M + l * nn + c0 + q) & __ldg(M + (l - 1) * nn + j);
        }
      }
      const uint32_t ta = transpose32((uint32_t)p), tb = transpose32((uint32_t)(p >> 32));
      const int qe = __shfl_sync(kFull, q, min(31, ch.total - 1 - f0));
      for (int r = __shfl_sync(kFull, q, 0); r <= qe; r++) {
        const int d = __shfl_sync(kFull, deg, r);
        if (!d) continue;
        const int o = __shfl_sync(kFull, ch.off, r) - f0;
        const int b = max(o, 0), e = min(o + d, 32);
        const unsigned m = (e == 32 ? kFull : (1u << e) - 1u) & ~((1u << b) - 1u);
        ca += __popc(ta & m);
        cb += __popc(tb & m);
        if (o + d > 32) break;  // the row goes on in the next 32 entries
        const u64 w = __shfl_sync(kFull, reach, r);
        float* const Tc = T + (size_t)(c0 + r) * kLanes;
        if ((w >> lane) & 1ull) Tc[lane] = ca ? 1.0f / (float)ca : 0.0f;
        if ((w >> (lane + 32)) & 1ull) Tc[lane + 32] = cb ? 1.0f / (float)cb : 0.0f;
        ca = cb = 0;
      }
    }
  }
}

// A lane's two sources of a 64-bit word (lane l: sources 2 l and 2 l + 1).
__device__ __forceinline__ unsigned bit_pair(u64 w) { return (unsigned)(w >> (2 * lane_id())) & 3u; }

// The sum of a vertex's terms at a level: into its own term o (read by the
// next sweep, so not at level 1) and into its betweenness.  This warp alone
// touches both in this sweep.
__device__ __forceinline__ void add_delta(float* __restrict__ T, double* __restrict__ bc, int32_t v, u64 w,
                                          int32_t level, float2 s, float2 o) {
  const int lane = lane_id();
  if (level > 1) {
    const unsigned m = bit_pair(w);
    float* const Tv = T + (size_t)v * kLanes + 2 * lane;
    if (m & 1u) Tv[0] = o.x + s.x;
    if (m & 2u) Tv[1] = o.y + s.y;
  }
  double pd = (double)s.x + (double)s.y;  // zero for sources without the vertex's bit
#pragma unroll
  for (int d = 16; d; d >>= 1) pd += __shfl_xor_sync(kFull, pd, d);
  if (lane == 0 && pd != 0.0) atomicAdd(bc + v, pd);  // fire and forget
}

// Level l of the backward sweep.
// The words of a group's edges are compacted into shared memory, so that an
// edge costs its term row's load, two masked adds a lane and little else: with
// its words passed by shuffles the sweeps were bound by issue, 60 instructions
// an edge.
__global__ void __launch_bounds__(kBlock, 5) bc_sweep(const int32_t* __restrict__ row_ptr,
                                                   const int32_t* __restrict__ col, const u64* __restrict__ M,
                                                   float* __restrict__ T, double* __restrict__ bc, int32_t n,
                                                   int32_t level, int32_t per, HeavyRows h, float* __restrict__ part,
                                                   int32_t* __restrict__ done) {
  __shared__ uint2 edges[kBlock / 32][32][2];  // target, and its low or high 32 sources
  const int lane = lane_id();
  uint2(*const edge)[2] = edges[threadIdx.x >> 5];
  M += (size_t)blockIdx.y * n * 32;
  T += (size_t)blockIdx.y * n * kLanes;
  bc += (size_t)blockIdx.y * n;
  part += (size_t)blockIdx.y * h.segs * kLanes;
  done += (size_t)blockIdx.y * h.count;
  const u64 *const here = M + (size_t)level * n, *const below = here + n;
  const int chunks = (n + per - 1) / per;
  for (int t = global_warp(); t < h.segs + chunks; t += num_warps()) {
    const bool heavy = t < h.segs;
    int hidx = 0, s0 = 0, s1 = 0;
    int32_t v0, ks = 0, deg = 0;
    u64 w = 0ull;
    if (heavy) {  // one row: the segment's entries
      const int4 hv = __ldg(h.seg + t);
      hidx = hv.x;
      v0 = hv.y;
      w = __ldg(here + v0);
      s0 = __ldg(h.off + hidx);
      s1 = __ldg(h.off + hidx + 1);
      if (lane == 0) {
        ks = hv.z;
        deg = hv.w;
      }
      if (!w) continue;
    } else {
      v0 = (t - h.segs) * per;
      const int32_t v = v0 + lane;
      if (lane < per && v < n) {
        w = __ldg(here + v);
        ks = row_ptr[v];
        deg = row_ptr[v + 1] - ks;
        if (deg >= kHeavy || !w) deg = 0;
      }
    }
    const RowChunk ch(ks, deg);
    int32_t cur = -1;  // the row being summed
    float2 s = make_float2(0.0f, 0.0f), own = s;
    for (int f0 = 0; f0 < ch.total; f0 += 32) {
      const int f = f0 + lane;
      const int q = ch.row(f);
      const int32_t k = __shfl_sync(kFull, ch.ks, q) + f - __shfl_sync(kFull, ch.off, q);
      const u64 wq = __shfl_sync(kFull, w, q);
      int32_t c = 0;
      u64 x = 0ull;
      if (f < ch.total) {
        c = __ldg(col + k);
        x = wq & __ldg(below + c);
      }
      unsigned todo = __ballot_sync(kFull, x != 0ull);
      if (x) {
        const int slot = __popc(todo & ((1u << lane) - 1u));
        edge[slot][0] = make_uint2((unsigned)c, (unsigned)x);
        edge[slot][1] = make_uint2((unsigned)c, (unsigned)(x >> 32));
      }
      __syncwarp();
      for (int at = 0; todo;) {
        const int r = __shfl_sync(kFull, q, __ffs(todo) - 1);
        const unsigned mine = todo & __ballot_sync(kFull, q == r);
        todo &= ~mine;
        if (r != cur) {
          if (cur >= 0) add_delta(T, bc, v0 + cur, __shfl_sync(kFull, w, cur), level, s, own);
          cur = r;
          s = make_float2(0.0f, 0.0f);
          if (!heavy && level > 1) own = __ldcg(reinterpret_cast<const float2*>(T + (size_t)(v0 + r) * kLanes) + lane);
        }
        const int end = at + __popc(mine);
        for (; at < end; at += kRows) {
          float2 x2[kRows];
          unsigned m[kRows];
#pragma unroll
          for (int i = 0; i < kRows; i++) {
            const uint2 e = at + i < end ? edge[at + i][lane >> 4] : make_uint2(0u, 0u);
            m[i] = (e.y >> (2 * (lane & 15))) & 3u;
            x2[i] = m[i] ? __ldcg(reinterpret_cast<const float2*>(T + (size_t)e.x * kLanes) + lane)
                         : make_float2(0.0f, 0.0f);
          }
#pragma unroll
          for (int i = 0; i < kRows; i++) {
            if (m[i] & 1u) s.x += x2[i].x;
            if (m[i] & 2u) s.y += x2[i].y;
          }
        }
        at = end;
      }
      __syncwarp();
    }
    if (!heavy) {
      if (cur >= 0) add_delta(T, bc, v0 + cur, __shfl_sync(kFull, w, cur), level, s, own);
      continue;
    }
    float2* const rows = reinterpret_cast<float2*>(part);
    rows[(size_t)t * 32 + lane] = s;
    if (!last_segment(done + hidx, s1 - s0)) continue;
    s = make_float2(0.0f, 0.0f);
    for (int sg = s0; sg < s1; sg += kRows) {
      float2 x2[kRows];
#pragma unroll
      for (int i = 0; i < kRows; i++)
        x2[i] = sg + i < s1 ? __ldcg(rows + (size_t)(sg + i) * 32 + lane) : make_float2(0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < kRows; i++) {
        s.x += x2[i].x;
        s.y += x2[i].y;
      }
    }
    if (level > 1) own = __ldcg(reinterpret_cast<const float2*>(T + (size_t)v0 * kLanes) + lane);
    add_delta(T, bc, v0, w, level, s, own);
  }
}

// The betweenness of the blocks, added in their order.
__global__ void __launch_bounds__(kBlock) bc_fold(const double* __restrict__ acc, double* __restrict__ bc, int32_t n,
                                                  int blocks) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < (size_t)n; v += stride) {
    double s = 0.0;
    for (int b = 0; b < blocks; b++) s += acc[b * (size_t)n + v];
    bc[v] = s;
  }
}

// --- deeper batches on short rows: (vertex, source) pairs by level ------------------
//
// On a mesh a vertex is at 40 levels for 64 sources, and a sweep over vertices
// reads 512 bytes an edge for the one source or two that are at its level: 44 us a
// level on a kNN graph of 50,000 points.  Here the pairs are sorted by level
// once, and a lane takes one pair and walks its row, eight bytes an edge.  The
// additions are those of the level rows: along a row, one after another.  Rows
// of kHeavy entries and more would hold a lane too long, so graphs with one keep
// the level rows.  Per call, sweeps over vertices -> pairs: kNN of 50,000 points, 60
// sources 8.2 -> 4.5 ms, of 3,000 points, 200 sources 4.6 -> 2.2, grid 150 x 150,
// 60 sources 6.5 -> 4.4.

constexpr int kPairLevels = 4096;  // levels counted in shared memory

// Counts the pairs of every level (kPlace false), or puts pair ids (vertex x 64 +
// source) in their level's part of the list, where cursor[l] stands (kPlace).
// Level 0 is left out.
template <bool kPlace>
__global__ void __launch_bounds__(kBlock) bc_pairs(const int32_t* __restrict__ L, size_t quads, int levels,
                                                   uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
  __shared__ uint32_t cnt[kPairLevels];
  const bool local = levels <= kPairLevels;
  const size_t per = (quads + gridDim.x - 1) / gridDim.x, q0 = blockIdx.x * per, q1 = min(q0 + per, quads);
  if (local) {
    for (int l = threadIdx.x; l < levels; l += kBlock) cnt[l] = 0;
    __syncthreads();
    for (size_t q = q0 + threadIdx.x; q < q1; q += kBlock) {
      const int4 x = __ldg(reinterpret_cast<const int4*>(L) + q);
      if (x.x > 0) atomicAdd(cnt + x.x, 1u);
      if (x.y > 0) atomicAdd(cnt + x.y, 1u);
      if (x.z > 0) atomicAdd(cnt + x.z, 1u);
      if (x.w > 0) atomicAdd(cnt + x.w, 1u);
    }
    __syncthreads();
    for (int l = threadIdx.x; l < levels; l += kBlock)
      if (cnt[l]) cnt[l] = atomicAdd(cursor + l, cnt[l]);
    if (!kPlace) return;
    __syncthreads();
  }
  uint32_t* const at = local ? cnt : cursor;
  for (size_t q = q0 + threadIdx.x; q < q1; q += kBlock) {
    const int4 x = __ldg(reinterpret_cast<const int4*>(L) + q);
    const int32_t l[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (l[i] > 0) {
        const uint32_t pos = atomicAdd(at + l[i], 1u);
        if (kPlace) list[pos] = (uint32_t)(4 * q + i);
      }
  }
}

// Counts to first positions: off[l], and the same in cursor for the placing.  One
// CTA.
__global__ void __launch_bounds__(1024) bc_pair_offsets(uint32_t* __restrict__ cursor, uint32_t* __restrict__ off,
                                                        int levels) {
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t base;
  if (threadIdx.x == 0) base = 0;
  const int lane = lane_id(), w = threadIdx.x >> 5;
  for (int l0 = 0; l0 <= levels; l0 += 1024) {
    const int l = l0 + threadIdx.x;
    const uint32_t x = l < levels ? cursor[l] : 0u;
    const uint32_t incl = (uint32_t)warp_incl_scan((int)x);
    __syncthreads();
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) warp_tot[lane] = (uint32_t)warp_incl_scan((int)warp_tot[lane]);
    __syncthreads();
    const uint32_t first = base + (w ? warp_tot[w - 1] : 0u) + incl - x;
    if (l <= levels) off[l] = first;
    if (l < levels) cursor[l] = first;
    __syncthreads();
    if (threadIdx.x == 0) base += warp_tot[31];
  }
}

// 1 / amount of the pairs at level 2 and deeper.
__global__ void __launch_bounds__(kBlock) bc_pair_amounts(const int32_t* __restrict__ t_row_ptr,
                                                          const int32_t* __restrict__ t_col,
                                                          const int32_t* __restrict__ L, float* __restrict__ T,
                                                          const uint32_t* __restrict__ list,
                                                          const uint32_t* __restrict__ off, int levels) {
  const size_t stride = (size_t)gridDim.x * kBlock;
  for (size_t i = off[2] + blockIdx.x * (size_t)kBlock + threadIdx.x; i < off[levels]; i += stride) {
    const uint32_t p = list[i], src = p & 63u;
    const int l = L[p], ke = __ldg(t_row_ptr + (p >> 6) + 1);
    int amount = 0;
    for (int k = __ldg(t_row_ptr + (p >> 6)); k < ke; k += kUnroll) {
      int32_t x[kUnroll];
#pragma unroll
      for (int j = 0; j < kUnroll; j++) x[j] = k + j < ke ? __ldg(L + (size_t)__ldg(t_col + k + j) * kLanes + src) : -2;
#pragma unroll
      for (int j = 0; j < kUnroll; j++) amount += x[j] == l - 1;
    }
    T[p] = amount ? 1.0f / (float)amount : 0.0f;
  }
}

// Level l of the backward sweep.
__global__ void __launch_bounds__(kBlock) bc_pair_sweep(const int32_t* __restrict__ row_ptr,
                                                        const int32_t* __restrict__ col,
                                                        const int32_t* __restrict__ L, float* __restrict__ T,
                                                        float* __restrict__ delta, const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ off, int level) {
  const size_t stride = (size_t)gridDim.x * kBlock, end = off[level + 1];
  for (size_t i = off[level] + blockIdx.x * (size_t)kBlock + threadIdx.x; i < end; i += stride) {
    const uint32_t p = list[i], src = p & 63u;
    const int ke = __ldg(row_ptr + (p >> 6) + 1);
    const float own = level > 1 ? __ldcg(T + p) : 0.0f;
    float sum = 0.0f;
    for (int k = __ldg(row_ptr + (p >> 6)); k < ke; k += kUnroll) {
      int32_t x[kUnroll];
      float t[kUnroll];
#pragma unroll
      for (int j = 0; j < kUnroll; j++) {
        const size_t c = k + j < ke ? (size_t)__ldg(col + k + j) * kLanes + src : 0;
        x[j] = k + j < ke ? __ldg(L + c) : -2;
        t[j] = k + j < ke ? __ldcg(T + c) : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < kUnroll; j++)
        if (x[j] == level + 1) sum += t[j];
    }
    delta[p] = sum;
    if (level > 1) T[p] = own + sum;
  }
}

// The vertices' betweenness from the block: half a warp per vertex.
__global__ void __launch_bounds__(kBlock) bc_pair_sums(const int32_t* __restrict__ L, const float* __restrict__ delta,
                                                       double* __restrict__ bc, int32_t n, int levels) {
  const int lane = lane_id(), sub = lane & 15;
  for (int v0 = global_warp() * 2; v0 < n; v0 += num_warps() * 2) {
    const int v = v0 + (lane >> 4);
    double sum = 0.0;
    if (v < n) {
      const int4 l = __ldg(reinterpret_cast<const int4*>(L + (size_t)v * kLanes) + sub);
      const float4 d = __ldg(reinterpret_cast<const float4*>(delta + (size_t)v * kLanes) + sub);
      // pairs at level 1 to the last but one have a delta
      if (l.x > 0 && l.x < levels - 1) sum += (double)d.x;
      if (l.y > 0 && l.y < levels - 1) sum += (double)d.y;
      if (l.z > 0 && l.z < levels - 1) sum += (double)d.z;
      if (l.w > 0 && l.w < levels - 1) sum += (double)d.w;
    }
#pragma unroll
    for (int k = 8; k; k >>= 1) sum += __shfl_xor_sync(kFull, sum, k);
    if (sub == 0 && v < n && sum != 0.0) bc[v] += sum;
  }
}

// The passes of one deep block of 64 sources whose deepest level is deepest.
void pair_passes(dawn_graph* g, const int32_t* L, float* T, double* out, int deepest) {
  const size_t nn = (size_t)g->n;
  const int levels = deepest + 1, sms = g->geo.sms;
  uint32_t* const list = g->bc_pairs.as<uint32_t>();
  float* const delta = reinterpret_cast<float*>(list + kLanes * nn);
  uint32_t *const off = list + 2 * kLanes * nn, *const cursor = off + nn + 2;
  cudaMemsetAsync(cursor, 0, sizeof(uint32_t) * (size_t)levels, g->stream);
  bc_pairs<false><<<sms * 4, kBlock, 0, g->stream>>>(L, 16 * nn, levels, cursor, nullptr);
  bc_pair_offsets<<<1, 1024, 0, g->stream>>>(cursor, off, levels);
  bc_pairs<true><<<sms * 4, kBlock, 0, g->stream>>>(L, 16 * nn, levels, cursor, list);
  if (levels > 2) bc_pair_amounts<<<sms * 8, kBlock, 0, g->stream>>>(g->t_row_ptr, g->t_col, L, T, list, off, levels);
  for (int l = deepest - 1; l >= 1; l--)
    bc_pair_sweep<<<sms, kBlock, 0, g->stream>>>(g->row_ptr, g->col, L, T, delta, list, off, l);
  bc_pair_sums<<<sms * 8, kBlock, 0, g->stream>>>(L, delta, out, g->n, levels);
}

// --- deeper batches: level rows -----------------------------------------------------

// Per lane, the entries j -> c in [ks, ke) whose level row holds la - 1
// (lanes 0-31) and lb - 1 (lanes 32-63 of the row).
__device__ __forceinline__ void count_preds(const int32_t* __restrict__ t_col, const int32_t* __restrict__ L,
                                            int ks, int ke, bool wa, bool wb, int32_t la, int32_t lb, int& ca,
                                            int& cb) {
  const int lane = lane_id();
  for (int kb = ks; kb < ke; kb += 32) {
    const int k = kb + lane;
    const int32_t jv = k < ke ? __ldg(t_col + k) : -1;
    const int cnt = min(32, ke - kb);
    for (int j0 = 0; j0 < cnt; j0 += kUnroll) {
      int32_t ra[kUnroll], rb[kUnroll];
#pragma unroll
      for (int i = 0; i < kUnroll; i++) {
        const int32_t j = __shfl_sync(kFull, jv, (j0 + i) & 31);
        const bool ok = j0 + i < cnt;
        const int32_t* Lj = L + (size_t)(ok ? j : 0) * kLanes;
        ra[i] = ok && wa ? __ldcg(Lj + lane) : -2;
        rb[i] = ok && wb ? __ldcg(Lj + lane + 32) : -2;
      }
#pragma unroll
      for (int i = 0; i < kUnroll; i++) {
        ca += ra[i] == la - 1;
        cb += rb[i] == lb - 1;
      }
    }
  }
}

// Per lane, the sum of term(c) over entries v -> c in [ks, ke) with c at
// level + 1 for the lane's sources.
__device__ __forceinline__ void sum_terms(const int32_t* __restrict__ col, const int32_t* __restrict__ L,
                                          const float* __restrict__ T, int ks, int ke, bool wa, bool wb,
                                          int32_t level, float& sa, float& sb) {
  const int lane = lane_id();
  for (int kb = ks; kb < ke; kb += 32) {
    const int k = kb + lane;
    const int32_t cv = k < ke ? __ldg(col + k) : -1;
    const int cnt = min(32, ke - kb);
    for (int j0 = 0; j0 < cnt; j0 += kUnroll) {
      int32_t la[kUnroll], lb[kUnroll];
      float ta[kUnroll], tb[kUnroll];
#pragma unroll
      for (int i = 0; i < kUnroll; i++) {
        const int32_t c = __shfl_sync(kFull, cv, (j0 + i) & 31);
        const bool ok = j0 + i < cnt;
        const size_t row = (size_t)(ok ? c : 0) * kLanes;
        la[i] = ok && wa ? __ldcg(L + row + lane) : -2;
        lb[i] = ok && wb ? __ldcg(L + row + lane + 32) : -2;
        ta[i] = ok && wa ? __ldcg(T + row + lane) : 0.0f;
        tb[i] = ok && wb ? __ldcg(T + row + lane + 32) : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < kUnroll; i++) {
        if (la[i] == level + 1) sa += ta[i];
        if (lb[i] == level + 1) sb += tb[i];
      }
    }
  }
}

// 1 / amount for every (vertex, source) slot of the short in-rows; heavy
// in-rows' segments add their counts to cnt (one 64-entry row per heavy row).
__global__ void __launch_bounds__(kBlock) bc_rows_amount(const int32_t* __restrict__ t_row_ptr,
                                                    const int32_t* __restrict__ t_col,
                                                    const int32_t* __restrict__ L, float* __restrict__ T,
                                                    int32_t n, HeavyRows h, int32_t* __restrict__ cnt) {
  const int lane = lane_id();
  for (int t = global_warp(); t < n + h.segs; t += num_warps()) {
    int32_t c;
    int ks, ke, hidx, seg;
    if (!task_range(t, n, t_row_ptr, h, c, ks, ke, hidx, seg)) continue;  // warp-uniform
    const int32_t* Lc = L + (size_t)c * kLanes;
    const int32_t la = Lc[lane], lb = Lc[lane + 32];
    const bool wa = la >= 2, wb = lb >= 2;
    int ca = 0, cb = 0;
    if (__any_sync(kFull, wa || wb)) count_preds(t_col, L, ks, ke, wa, wb, la, lb, ca, cb);
    if (hidx < 0) {
      float* Tc = T + (size_t)c * kLanes;
      Tc[lane] = wa && ca ? 1.0f / (float)ca : 0.0f;
      Tc[lane + 32] = wb && cb ? 1.0f / (float)cb : 0.0f;
    } else {
      if (ca) atomicAdd(cnt + (size_t)hidx * kLanes + lane, ca);
      if (cb) atomicAdd(cnt + (size_t)hidx * kLanes + lane + 32, cb);
    }
  }
}

// Heavy in-rows: 1 / amount from the summed counts, which are cleared for
// the next batch.
__global__ void __launch_bounds__(kBlock) bc_rows_amount_heavy(const int32_t* __restrict__ L, float* __restrict__ T,
                                                          HeavyRows h, int32_t* __restrict__ cnt) {
  const int lane = lane_id();
  for (int hidx = global_warp(); hidx < h.count; hidx += num_warps()) {
    const int32_t c = __ldg(h.v + hidx);
    const int32_t la = L[(size_t)c * kLanes + lane], lb = L[(size_t)c * kLanes + lane + 32];
    int32_t* cr = cnt + (size_t)hidx * kLanes;
    const int ca = cr[lane], cb = cr[lane + 32];
    cr[lane] = 0;
    cr[lane + 32] = 0;
    float* Tc = T + (size_t)c * kLanes;
    Tc[lane] = la >= 2 && ca ? 1.0f / (float)ca : 0.0f;
    Tc[lane + 32] = lb >= 2 && cb ? 1.0f / (float)cb : 0.0f;
  }
}

// Level l of the backward sweep (see the file comment) over the short
// out-rows; heavy out-rows' segments leave their partial sums in part.
__global__ void __launch_bounds__(kBlock) bc_rows_sweep(const int32_t* __restrict__ row_ptr,
                                                   const int32_t* __restrict__ col,
                                                   const int32_t* __restrict__ L, const int32_t* __restrict__ range,
                                                   float* __restrict__ T, double* __restrict__ bc, int32_t n,
                                                   int32_t level, HeavyRows h, float* __restrict__ part) {
  const int lane = lane_id();
  for (int t = global_warp(); t < n + h.segs; t += num_warps()) {
    int32_t v;
    int ks, ke, hidx, seg;
    if (!task_range(t, n, row_ptr, h, v, ks, ke, hidx, seg)) continue;  // warp-uniform
    if (level < range[2 * v] || level > range[2 * v + 1]) continue;      // warp-uniform
    const int32_t* Lv = L + (size_t)v * kLanes;
    const bool wa = Lv[lane] == level, wb = Lv[lane + 32] == level;
    if (!__any_sync(kFull, wa || wb)) continue;
    float sa = 0.0f, sb = 0.0f;
    sum_terms(col, L, T, ks, ke, wa, wb, level, sa, sb);
    if (hidx >= 0) {
      part[(size_t)seg * kLanes + lane] = sa;
      part[(size_t)seg * kLanes + lane + 32] = sb;
      continue;
    }
    float* Tv = T + (size_t)v * kLanes;
    if (wa) Tv[lane] += sa;
    if (wb) Tv[lane + 32] += sb;
    double pd = (wa ? (double)sa : 0.0) + (wb ? (double)sb : 0.0);
#pragma unroll
    for (int d = 16; d; d >>= 1) pd += __shfl_xor_sync(kFull, pd, d);
    if (lane == 0 && pd != 0.0) bc[v] += pd;  // this warp alone touches bc[v] in this sweep
  }
}

// Level l for the heavy out-rows: their segments' partial sums, added in
// segment order.
__global__ void __launch_bounds__(kBlock) bc_rows_sweep_heavy(const int32_t* __restrict__ L,
                                                         const int32_t* __restrict__ range, float* __restrict__ T,
                                                         double* __restrict__ bc, int32_t level, HeavyRows h,
                                                         const float* __restrict__ part) {
  const int lane = lane_id();
  for (int hidx = global_warp(); hidx < h.count; hidx += num_warps()) {
    const int32_t v = __ldg(h.v + hidx);
    if (level < range[2 * v] || level > range[2 * v + 1]) continue;
    const int32_t* Lv = L + (size_t)v * kLanes;
    const bool wa = Lv[lane] == level, wb = Lv[lane + 32] == level;
    if (!__any_sync(kFull, wa || wb)) continue;
    float sa = 0.0f, sb = 0.0f;
    const int s1 = __ldg(h.off + hidx + 1);
    for (int sg = __ldg(h.off + hidx); sg < s1; sg++) {
      sa += part[(size_t)sg * kLanes + lane];
      sb += part[(size_t)sg * kLanes + lane + 32];
    }
    float* Tv = T + (size_t)v * kLanes;
    if (wa) Tv[lane] += sa;
    if (wb) Tv[lane + 32] += sb;
    double pd = (wa ? (double)sa : 0.0) + (wb ? (double)sb : 0.0);
#pragma unroll
    for (int d = 16; d; d >>= 1) pd += __shfl_xor_sync(kFull, pd, d);
    if (lane == 0 && pd != 0.0) bc[v] += pd;
  }
}

// Heavy-row lists of one CSR (host side): rows of at least kHeavy entries
// and the prefix of their segment counts.
void heavy_rows(const std::vector<int32_t>& rp, std::vector<int32_t>& ids, std::vector<int32_t>& off) {
  ids.clear();
  off.assign(1, 0);
  for (size_t v = 0; v + 1 < rp.size(); v++) {
    const int deg = rp[v + 1] - rp[v];
    if (deg < kHeavy) continue;
    ids.push_back((int32_t)v);
    off.push_back(off.back() + (deg + kBcSeg - 1) / kBcSeg);
  }
}

// Builds the heavy-row lists once per handle (out-rows for the sweeps,
// in-rows for the amounts).
dawn_status prepare_heavy(dawn_graph* g) {
  if (g->bc_hout >= 0) return DAWN_OK;
  const size_t nn = (size_t)g->n;
  std::vector<int32_t> rps[2], out_ids, out_off, in_ids, in_off;
  for (int side = 0; side < 2; side++) {
    std::vector<int32_t>& rp = rps[side];
    if (side && g->t_row_ptr == g->row_ptr) {
      rp = rps[0];
    } else {
      rp.resize(nn + 1);
      DAWN_CUDA(cudaMemcpyAsync(rp.data(), side ? g->t_row_ptr : g->row_ptr, sizeof(int32_t) * (nn + 1),
                                cudaMemcpyDeviceToHost, g->stream));
      DAWN_CUDA(cudaStreamSynchronize(g->stream));
    }
    heavy_rows(rp, side ? in_ids : out_ids, side ? in_off : out_off);
  }
  std::vector<int32_t> all;
  for (int side = 0; side < 2; side++) {
    const std::vector<int32_t>&ids = side ? in_ids : out_ids, &off = side ? in_off : out_off;
    for (size_t i = 0; i < ids.size(); i++)
      for (int32_t sg = off[i]; sg < off[i + 1]; sg++) {
        const int32_t first = rps[side][ids[i]] + (sg - off[i]) * kBcSeg;
        all.insert(all.end(), {(int32_t)i, ids[i], first, std::min(kBcSeg, rps[side][ids[i] + 1] - first)});
      }
  }
  all.insert(all.end(), out_ids.begin(), out_ids.end());
  all.insert(all.end(), out_off.begin(), out_off.end());
  all.insert(all.end(), in_ids.begin(), in_ids.end());
  all.insert(all.end(), in_off.begin(), in_off.end());
  DAWN_CHECK(ensure(g->bc_heavy, sizeof(int32_t) * all.size(), g->stream));
  DAWN_CUDA(cudaMemcpyAsync(g->bc_heavy.p, all.data(), sizeof(int32_t) * all.size(), cudaMemcpyHostToDevice,
                            g->stream));
  DAWN_CUDA(cudaStreamSynchronize(g->stream));
  g->bc_segs_out = out_off.back();
  g->bc_hin = (int32_t)in_ids.size();
  g->bc_segs_in = in_off.back();
  g->bc_hout = (int32_t)out_ids.size();
  return DAWN_OK;
}

// Scratch of one block's partial sums of the out-row segments, in-row counts and
// finished segments of the heavy rows.
size_t part_words(const dawn_graph* g) {
  return ((size_t)g->bc_segs_out + g->bc_hin) * kLanes + g->bc_hout + g->bc_hin;
}

// The buffers for batches of `blocks` x 64 sources.
dawn_status reserve(dawn_graph* g, int blocks) {
  const size_t nn = (size_t)g->n, b = (size_t)blocks;
  DAWN_CHECK(bitset_reserve(g, blocks));
  DAWN_CHECK(ensure(g->bc_levels, sizeof(int32_t) * kLanes * nn * 2 * b, g->stream));
  DAWN_CHECK(ensure(g->bc_terms, sizeof(float) * kLanes * nn * b, g->stream));
  DAWN_CHECK(ensure(g->bc_range, sizeof(int32_t) * 2 * nn * 2 * b, g->stream));
  if (blocks > 1) DAWN_CHECK(ensure(g->bc_acc, sizeof(double) * nn * b, g->stream));
  if (g->bc_blocks < blocks) {
    // the counts start at zero (the warp that ends a row clears them)
    const size_t bytes = sizeof(float) * (part_words(g) * b + 1);
    g->bc_blocks = 0;
    DAWN_CHECK(ensure(g->bc_part, bytes, g->stream));
    DAWN_CUDA(cudaMemsetAsync(g->bc_part.p, 0, bytes, g->stream));
    g->bc_blocks = blocks;
  }
  return DAWN_OK;
}

}  // namespace

dawn_status betweenness(dawn_graph* g, const int32_t* sources, int32_t nsrc, double* d_bc, dawn_stats* st) {
  const size_t nn = (size_t)g->n;
  DAWN_CHECK(prepare_heavy(g));
  DAWN_CHECK(longest_row(g));
  // Batches of up to 256 sources: RMAT-16, 150 sources, takes 810 us in one and
  // took 1150 in three of 64.  A block of 64 takes about 0.9 KB a vertex and 5 bytes an
  // edge, so large graphs take fewer at a time, and so do devices with little
  // memory left.
  constexpr size_t kScratch = (size_t)24 << 30;
  int width = bitset_width(g, nsrc);
  while (width > 1 && width * (nn * 900 + part_words(g) * sizeof(float)) > kScratch) width /= 2;
  for (;; width /= 2) {
    const dawn_status s = reserve(g, width);
    if (s == DAWN_OK) break;
    if (width == 1) return s;
    cudaGetLastError();
    clear_error();
  }
  if (!g->bc_h_level) DAWN_CHECK(pinned_slot((void**)&g->bc_h_level));
  const int32_t nb = (nsrc + kLanes - 1) / kLanes, nbatches = (nb + width - 1) / width;
  const int32_t nacc = std::max(1, std::min<int32_t>(nb, width));  // no sources: zeros all the same
  double* const acc = nacc > 1 ? g->bc_acc.as<double>() : d_bc;
  DAWN_CUDA(cudaMemsetAsync(acc, 0, sizeof(double) * nn * nacc, g->stream));
  // Level blocks and ranges are double-buffered: the traversal of batch b runs
  // while the host waits for batch b - 1's depth, so the stream always has
  // work queued (traversal b, then the sweeps of b - 1).  The terms need one
  // buffer: the amount and sweep passes of the batches follow one another.
  const size_t lv = kLanes * nn * width, rg = 2 * nn * width;
  int32_t* const Ls[2] = {g->bc_levels.as<int32_t>(), g->bc_levels.as<int32_t>() + lv};
  int32_t* const Rs[2] = {g->bc_range.as<int32_t>(), g->bc_range.as<int32_t>() + rg};
  float* T = g->bc_terms.as<float>();
  const int4* const seg_out = g->bc_heavy.as<int4>();
  const int4* const seg_in = seg_out + g->bc_segs_out;
  const int32_t* hv = reinterpret_cast<const int32_t*>(seg_in + g->bc_segs_in);
  HeavyRows hout{seg_out, hv, hv + g->bc_hout, g->bc_hout, g->bc_segs_out};
  const int32_t* hin_base = hv + 2 * g->bc_hout + 1;
  HeavyRows hin{seg_in, hin_base, hin_base + g->bc_hin, g->bc_hin, g->bc_segs_in};
  const size_t blocks = (size_t)g->bc_blocks;
  float* part = g->bc_part.as<float>();
  int32_t* const cnt = g->bc_part.as<int32_t>() + blocks * g->bc_segs_out * kLanes;
  int32_t* const done_out = cnt + blocks * g->bc_hin * kLanes;
  int32_t* const done_in = done_out + blocks * g->bc_hout;
  const int ctas = persistent_blocks((const void*)bc_sweep, kBlock, 0, g->blocks_per_sm);
  const int ctas_amount = persistent_blocks((const void*)bc_amount, kBlock, 0, g->blocks_per_sm);
  // the level pass runs the plain batched traversal (direction heuristic)
  DAWN_CHECK(call_selector(g, DAWN_VARIANT_BITSET, &g->sel_call));
  cudaEvent_t done[2] = {nullptr, nullptr};
  dawn_status status = DAWN_OK;
  int64_t levels = 0;
  const auto in_batch = [&](int32_t b) { return std::min(nsrc - b * kLanes * width, kLanes * width); };
  for (int i = 0; i < 2; i++)
    if (cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming) != cudaSuccess) {
      set_error("betweenness: cudaEventCreate failed");
      status = DAWN_ERR_CUDA;
    }
  for (int32_t b = 0; b <= nbatches && status == DAWN_OK; b++) {
    if (b < nbatches) {
      status = bfs_bitset_levels(g, width, sources + b * kLanes * width, in_batch(b), Ls[b & 1], Rs[b & 1],
                                 g->bc_h_level + kLevelsEnd * (b & 1));
      if (status == DAWN_OK && cudaEventRecord(done[b & 1], g->stream) != cudaSuccess) {
        set_error("betweenness: cudaEventRecord failed");
        status = DAWN_ERR_CUDA;
      }
      if (status != DAWN_OK) break;
    }
    if (b == 0) continue;
    // the dependency passes of batch b - 1, once its depth is known
    const int p = (b - 1) & 1;
    if (cudaEventSynchronize(done[p]) != cudaSuccess) {
      set_error("betweenness: %s", cudaGetErrorString(cudaGetLastError()));
      status = DAWN_ERR_CUDA;
      break;
    }
    if ((status = device_status(g)) != DAWN_OK) break;
    const int32_t* const end = g->bc_h_level + kLevelsEnd * p;  // level, depth of each 64
    const int32_t k = (in_batch(b - 1) + kLanes - 1) / kLanes;  // blocks
    for (int32_t i = 0; i < k; i++) levels += end[1 + i];
    if (end[0] < kDeepLevel) {
      const u64* M = reinterpret_cast<const u64*>(Ls[p]);
      const dim3 grid(std::max(1, ctas / k), k), grid_amount(std::max(1, ctas_amount / k), k);
      const int per = chunk_rows(g->n, grid.x * (kBlock / 32));
      bc_amount<<<grid_amount, kBlock, 0, g->stream>>>(g->t_row_ptr, g->t_col, M, T, g->n, end[0],
                                                       chunk_rows(g->n, grid_amount.x * (kBlock / 32)), hin, cnt,
                                                       done_in);
      for (int32_t l = end[0] - 2; l >= 1; l--)
        bc_sweep<<<grid, kBlock, 0, g->stream>>>(g->row_ptr, g->col, M, T, acc, g->n, l, per, hout, part, done_out);
    } else {
      // pair ids are 32-bit, and the lists are scratch that large graphs may not get
      bool pairs = g->max_row < kHeavy && nn < (size_t)1 << 25;
      if (pairs && ensure(g->bc_pairs, sizeof(uint32_t) * (2 * kLanes + 2) * (nn + 2), g->stream) != DAWN_OK) {
        cudaGetLastError();
        clear_error();
        pairs = false;
      }
      for (int32_t i = 0; i < k; i++) {
        const int32_t *const L = Ls[p] + i * kLanes * nn, *const R = Rs[p] + i * 2 * nn;
        double* const out = acc + i * nn;
        if (pairs) {
          pair_passes(g, L, T, out, end[1 + i]);
          continue;
        }
        bc_rows_amount<<<ctas, kBlock, 0, g->stream>>>(g->t_row_ptr, g->t_col, L, T, g->n, hin, cnt);
        if (hin.count) bc_rows_amount_heavy<<<ctas, kBlock, 0, g->stream>>>(L, T, hin, cnt);
        for (int32_t l = end[1 + i] - 1; l >= 1; l--) {
          bc_rows_sweep<<<ctas, kBlock, 0, g->stream>>>(g->row_ptr, g->col, L, R, T, out, g->n, l, hout, part);
          if (hout.count) bc_rows_sweep_heavy<<<ctas, kBlock, 0, g->stream>>>(L, R, T, out, l, hout, part);
        }
      }
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error("betweenness: %s", cudaGetErrorString(e));
      status = DAWN_ERR_CUDA;
    }
  }
  for (cudaEvent_t e : done)
    if (e) cudaEventDestroy(e);
  DAWN_CHECK(status);
  if (nacc > 1) {
    bc_fold<<<g->geo.sms * 4, kBlock, 0, g->stream>>>(acc, d_bc, g->n, nacc);
    DAWN_CUDA(cudaGetLastError());
  }
  if (st) {
    std::memset(st, 0, sizeof(*st));
    st->levels = (int32_t)levels;
    st->batches = nb;
  }
  return DAWN_OK;
}

}  // namespace dawn
