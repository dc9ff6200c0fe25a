// kernels_compact.cu -- output compaction: fixed-shape sampler outputs to a
// dense (src, dst) edge list.
//
// The reference cuts invalid walkers out of each step's frontier: it radix
// sorts the (transit, sample) pairs, finds the first INVALID_VERTEX with a
// binary search kernel (invalidVertexStartPos, GT/src/grass.cu:1085-1117,
// launched :1641) and truncates there.  The samplers here never sort; they
// write fixed-shape outputs with GRASS_INVALID_VERTEX in the slots that a dead
// end leaves empty.  Compaction is a separate, order-preserving pass for
// callers that want only the sampled edges:
//   1. count: each block counts the valid slots of its share, a run of tiles
//      of 4096 slots;
//   2. fill: the same block takes the same share again, starts at the sum of
//      the counts before its own (one load or two a thread), and writes: each
//      warp owns 512 consecutive slots of a tile; a valid one is ranked inside
//      its warp with __ballot_sync and __popc, among the warps by a prefix over
//      the eight warp counts, so the output keeps the input order.
// Parent indices advance incrementally (32 / div and 32 % div per step), in 32
// bits from the tile's first slot.
//
// Shares make the tile counts, their scan (three launches) and the copy of the
// total unnecessary: a call on 16 K slots took 33 us with those, on 2.7 M 33, on
// 18 M 95, walk paths of 84 M 470; now 17, 17, 62 and 284.  One pass that looks back over the tiles' published counts measured
// 13.5, 25 and 107 us: with 592 tiles under way at a time a block waits longer
// for its place than a second pass over the children takes.
#include "graph.h"

namespace grass {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kPer = 16;                     // slots per lane per tile
constexpr uint32_t kWarpSlots = 32 * kPer;   // a warp's contiguous chunk
constexpr uint32_t kTileEntries = kThreads * kPer;

// A segment as the kernels see it; q and r name a slot's parent and its place
// under it: slot e = q div + r.
struct KSeg {
  const uint32_t *parent;
  const uint32_t *child;
  uint64_t n, tile0;
  uint32_t div, adv_q, adv_r;    // 32 / div and 32 % div, the step of (q, r) between a
                                 // lane's consecutive slots
  uint32_t tile_q, tile_r;       // the same for a tile's slots
};

struct Plan {
  KSeg seg[kCompactMaxSegs];
  uint32_t nseg;
  uint64_t tiles;
};

// (q, r) some slots on, for a step of (dq, dr), dr < div, without overflow.
template <class Q>
__device__ __forceinline__ void advance(Q &q, uint32_t &r, uint32_t div, uint32_t dq, uint32_t dr) {
  const bool wrap = r >= div - dr;
  r = wrap ? r - (div - dr) : r + dr;
  q += dq + (wrap ? 1u : 0u);
}

// The tiles of a block's share one after the other.
struct Walk {
  const KSeg *sg;
  uint64_t e, q;  // the tile's first slot and its parent
  uint32_t r;

  __device__ __forceinline__ void enter(const Plan &pl, uint64_t tile) {
    uint32_t k = 0;
    while (k + 1 < pl.nseg && tile >= pl.seg[k + 1].tile0) k++;
    sg = &pl.seg[k];
    e = (tile - sg->tile0) * kTileEntries;
    q = e / sg->div;
    r = (uint32_t)(e - q * sg->div);
  }
  __device__ __forceinline__ void next(const Plan &pl, uint64_t tile) {  // on to `tile`
    e += kTileEntries;
    if (e >= sg->n) enter(pl, tile);
    else advance(q, r, sg->div, sg->tile_q, sg->tile_r);
  }
  __device__ __forceinline__ uint32_t slots() const {
    return (uint32_t)min((uint64_t)kTileEntries, sg->n - e);
  }
  // The lane's first slot: parent and place from the tile's first.
  __device__ __forceinline__ void lane_start(uint32_t off, uint32_t &dq, uint32_t &dr) const {
    const uint64_t x = (uint64_t)r + off;
    const uint32_t div = sg->div;
    dq = div > kTileEntries ? (x >= div ? 1u : 0u) : (uint32_t)x / div;
    dr = (uint32_t)(x - (uint64_t)dq * div);
  }
};

// Child values of the lane's slots (and their parents), from the tile's first
// slot at offset `off`; walk-major path: slot e's child is entry e + q + 1.
template <int KIND, bool PARENTS>
__device__ __forceinline__ void tile_load(const Walk &t, uint32_t off, uint32_t (&cv)[kPer],
                                          uint32_t (&pv)[kPer]) {
  const uint32_t n = t.slots(), div = t.sg->div;
  const uint32_t *child = t.sg->child + t.e, *parent = t.sg->parent + t.q;
  uint32_t q = 0, r = 0;
  if (KIND == kCompactPath || PARENTS) t.lane_start(off, q, r);
  if (KIND == kCompactPath) {
    parent = child + t.q;
    child = parent + 1;
  }
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const uint32_t e = off + k * 32;
    const bool in = e < n;
    cv[k] = in ? __ldg(child + (KIND == kCompactPath ? e + q : e)) : GRASS_INVALID_VERTEX;
    if (PARENTS) pv[k] = in ? __ldg(parent + (KIND == kCompactPath ? e + q : q)) : 0u;
    if (KIND == kCompactPath || PARENTS) advance(q, r, div, t.sg->adv_q, t.sg->adv_r);
  }
}

// Sum of a value over the block's warps (lane 0's of each).
__device__ __forceinline__ uint64_t block_sum(uint64_t v, uint64_t *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) v += red[w];
  return v;
}

template <int KIND>
__global__ void __launch_bounds__(kThreads) compact_count_kernel(Plan pl, uint64_t share,
                                                                 uint64_t *counts) {
  __shared__ uint64_t red[kWarps];
  const uint32_t off = (threadIdx.x >> 5) * kWarpSlots + (threadIdx.x & 31);
  uint64_t tile = blockIdx.x * share;
  const uint64_t end = min(pl.tiles, tile + share);
  uint64_t cnt = 0;
  Walk t;
  t.enter(pl, tile);
  for (;;) {
    uint32_t cv[kPer];
    tile_load<KIND, false>(t, off, cv, cv);
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) c += cv[k] != GRASS_INVALID_VERTEX;
    cnt += c;
    if (++tile >= end) break;
    t.next(pl, tile);
  }
  cnt = block_sum(cnt, red);
  if (threadIdx.x == 0) counts[blockIdx.x] = cnt;
}

// Resident 256-thread blocks per SM: 4 (64 registers).
#ifndef GRASS_COMPACT_MIN_BLOCKS
#define GRASS_COMPACT_MIN_BLOCKS 4
#endif
// Shares per resident block: 1 and 4 took 70 and 62 us on 18 M slots, 313 and
// 284 on 84 M (with 3 and 5 resident blocks per SM and one share 71 and 64, 335
// and 356); a block adds up all counts before its own, 10 a thread at most.
#ifndef GRASS_COMPACT_SHARES
#define GRASS_COMPACT_SHARES 4
#endif

template <int KIND>
__global__ void __launch_bounds__(kThreads, GRASS_COMPACT_MIN_BLOCKS)
    compact_fill_kernel(Plan pl, uint64_t share, const uint64_t *counts, uint32_t *src,
                        uint32_t *dst, uint64_t cap, unsigned long long *count) {
  __shared__ uint64_t red[kWarps];
  __shared__ uint32_t wsum[2][kWarps];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t below = (1u << lane) - 1, off = warp * kWarpSlots + lane;
  uint64_t tile = blockIdx.x * share;
  const uint64_t end = min(pl.tiles, tile + share);
  uint64_t pos = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kThreads) pos += counts[b];
  Walk t;
  t.enter(pl, tile);
  uint32_t cv[kPer], pv[kPer];
  tile_load<KIND, true>(t, off, cv, pv);
  pos = block_sum(pos, red);
  for (uint32_t odd = 0;; odd ^= 1) {
    uint32_t total = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++)
      total += __popc(__ballot_sync(0xffffffffu, cv[k] != GRASS_INVALID_VERTEX));
    if (lane == 0) wsum[odd][warp] = total;
    __syncthreads();  // (the other half of wsum is read no more after this)
    uint32_t at = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const uint32_t c = wsum[odd][w];
      at += w < (int)warp ? c : 0u;
      all += c;
    }
    uint32_t *s = src + pos, *d = dst + pos;
    const uint32_t room = pos < cap ? (uint32_t)min((uint64_t)kTileEntries, cap - pos) : 0u;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const bool valid = cv[k] != GRASS_INVALID_VERTEX;
      const uint32_t m = __ballot_sync(0xffffffffu, valid);
      const uint32_t i = at + __popc(m & below);
      if (valid && i < room) {
        store_out_u32(s + i, pv[k]);
        store_out_u32(d + i, cv[k]);
      }
      at += __popc(m);
    }
    pos += all;
    if (++tile >= end) break;
    t.next(pl, tile);
    tile_load<KIND, true>(t, off, cv, pv);
  }
  if (tile == pl.tiles && threadIdx.x == 0) *count = pos;
}

template <int KIND>
void launch_kind(const Plan &pl, uint64_t share, unsigned grid, uint64_t *counts, uint32_t *src,
                 uint32_t *dst, uint64_t cap, unsigned long long *count, cudaStream_t s) {
  compact_count_kernel<KIND><<<grid, kThreads, 0, s>>>(pl, share, counts);
  compact_fill_kernel<KIND><<<grid, kThreads, 0, s>>>(pl, share, counts, src, dst, cap, count);
  count_launch(2);
}

}  // namespace

int launch_compact(const CompactSeg *segs, uint32_t nseg, uint32_t *src, uint32_t *dst,
                   uint64_t cap, unsigned long long *count, cudaStream_t s) {
  if (nseg == 0 || nseg > kCompactMaxSegs) return set_error(GRASS_E_ARG, "compaction: bad segment count");
  Plan pl{};
  pl.nseg = nseg;
  uint64_t tiles = 0;
  for (uint32_t k = 0; k < nseg; k++) {
    if (segs[k].kind != segs[0].kind) return set_error(GRASS_E_ARG, "compaction: mixed segment kinds");
    KSeg &q = pl.seg[k];
    q.parent = segs[k].parent;
    q.child = segs[k].child;
    q.n = segs[k].n;
    q.div = segs[k].div ? segs[k].div : 1u;
    q.adv_q = 32u / q.div;
    q.adv_r = 32u % q.div;
    q.tile_q = kTileEntries / q.div;
    q.tile_r = kTileEntries % q.div;
    q.tile0 = tiles;
    tiles += (segs[k].n + kTileEntries - 1) / kTileEntries;
  }
  pl.tiles = tiles;
  if (tiles == 0) {
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(unsigned long long), s);
    return e == cudaSuccess ? GRASS_OK : cuda_fail(e, "compaction count");
  }
  int dev = 0;
  cudaGetDevice(&dev);
  // each block has a run of `share` tiles
  const uint64_t blocks = (uint64_t)sm_count(dev) * GRASS_COMPACT_MIN_BLOCKS * GRASS_COMPACT_SHARES;
  const uint64_t share = (tiles + blocks - 1) / blocks;
  const unsigned grid = (unsigned)((tiles + share - 1) / share);
  uint64_t *counts = nullptr;
  cudaError_t e = scratch_alloc(reinterpret_cast<void **>(&counts), grid * sizeof(uint64_t), s);
  if (e != cudaSuccess) return cuda_fail(e, "compaction scratch");
  if (segs[0].kind == kCompactFan)
    launch_kind<kCompactFan>(pl, share, grid, counts, src, dst, cap, count, s);
  else
    launch_kind<kCompactPath>(pl, share, grid, counts, src, dst, cap, count, s);
  scratch_free(counts, s);
  return GRASS_OK;
}

}  // namespace grass
