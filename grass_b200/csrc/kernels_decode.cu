// kernels_decode.cu -- decode-only sweep: every neighbor list into CSR.
//
// Replaces the reference's two decoders for whole lists: the block-cooperative
// GlobalDecoder (GT/src/bcg.cuh:171-345, used by the grid/thread-block
// kernels at GT/src/grass.cu:529-553, 762-786) and repeated
// BCGVertex::get_vertex calls (LE/src/bcg.cuh:195-261).
//
// Work is split over the neighbor index space, not over vertices: task t
// covers neighbors [t*C, (t+1)*C) of the CSR being written, whatever
// vertices they belong to, so a hub vertex with 10^5 neighbors is spread over
// many warps instead of serialising one.  Per task a warp
//  1. finds the vertex holding the first neighbor with a 32-ary search of
//     rowptr (one coalesced probe per level);
//  2. for each round of 32 consecutive neighbors, loads the row ends and
//     records of a window of 32 vertices (coalesced), maps every lane to its
//     vertex by a shuffle binary search and takes the header by shuffle;
//  3. decodes each neighbor as one independent draw (its slot's head and one
//     offset);
//  4. writes its 32 ids with one coalesced store.
#include <vector>

#include "graph.h"

namespace grass {

namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr uint32_t kTaskNeighbors = 2048;  // multiple of 32

__device__ __forceinline__ uint4 shfl_rec(const uint4 &r, int src) {
  return make_uint4(__shfl_sync(FULL, r.x, src), __shfl_sync(FULL, r.y, src),
                    __shfl_sync(FULL, r.z, src), __shfl_sync(FULL, r.w, src));
}

// Largest v in [0, n) with rowptr[v] <= x, for x < rowptr[n].
__device__ __forceinline__ uint32_t warp_row_of(const uint64_t *rowptr, uint32_t n, uint64_t x) {
  const int lane = threadIdx.x & 31;
  uint64_t lo = 0, hi = n;  // rowptr[lo] <= x < rowptr[hi]
  while (hi - lo > 1) {
    const uint64_t step = (hi - lo + 31) / 32;
    const uint64_t p = lo + (uint64_t)(lane + 1) * step;
    const bool le = p < hi && rowptr[p] <= x;
    const uint32_t c = __popc(__ballot_sync(FULL, le));
    const uint64_t nlo = lo + (uint64_t)c * step;
    hi = min(hi, lo + (uint64_t)(c + 1) * step);
    lo = nlo;
  }
  return (uint32_t)lo;
}

// Largest v in [lo, n) with rowptr[v] <= x, one thread (rare fallback).
__device__ __forceinline__ uint32_t row_of_serial(const uint64_t *rowptr, uint32_t lo, uint32_t n,
                                                  uint64_t x) {
  uint32_t hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (rowptr[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(256) decode_all_kernel(DevGraph g, const uint64_t *rowptr,
                                                           uint32_t *cols, uint64_t E,
                                                           unsigned int *err) {
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t tasks = (E + kTaskNeighbors - 1) / kTaskNeighbors;
  bool bad = false;
  for (uint64_t t = warp; t < tasks; t += nwarps) {
    const uint64_t g0 = t * kTaskNeighbors;
    const uint64_t g1 = min(E, g0 + kTaskNeighbors);
    uint32_t vr = warp_row_of(rowptr, g.n, g0);
    // Header of the vertex that holds the whole current round (fast path),
    // kept across rounds of the same vertex.
    uint32_t cv = 0xFFFFFFFFu;
    uint64_t cstart = 0, cend = 0;
    VHdr ch{};
    bool ch_ok = false;
    for (uint64_t r = g0; r < g1; r += 32) {  // warp-uniform
      const uint64_t gl = r + lane;
      const bool act = gl < g1;
      const uint64_t rlast = min(g1, r + 32) - 1;
      if (vr != cv) {
        cv = vr;
        cstart = rowptr[vr];
        cend = rowptr[vr + 1];
        ch_ok = false;
      }
      VHdr hk;
      uint64_t startv;
      bool far = false;
      int k = 0;
      const bool single = cstart <= r && rlast < cend;  // warp-uniform
      if (single) {
        // Fast path: the round lies inside vertex vr (most rounds of a
        // skewed graph): no window, no owner search.
        if (!ch_ok) {
          ch = header<kSlots>(g, vr);
          ch_ok = true;
        }
        hk = ch;
        startv = cstart;
      } else {
        // window of vertices [vr, vr + 32): row ends and headers, one per lane
        const uint32_t wv = vr + lane;
        const uint64_t base = rowptr[vr];
        const uint64_t e = wv < g.n ? rowptr[wv + 1] : ~0ull;
        const uint4 rw = wv < g.n ? load_record(g.recs + wv) : make_uint4(0u, 0u, 0u, 0u);
        // owner lane k: number of window rows that end at or before gl
        // (binary lifting over 31 probes gives the exact count when it is
        // below 32)
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const uint64_t ek = __shfl_sync(FULL, e, k + step - 1);
          if (ek <= gl) k += step;
        }
        // a count of 32 means gl lies beyond the window (a run of >= 32 empty
        // rows); those lanes resolve their vertex and header on their own.
        const uint64_t e31 = __shfl_sync(FULL, e, 31);
        far = act && e31 <= gl;
        const int src = far ? 0 : k;
        const uint64_t prev_e = __shfl_sync(FULL, e, src > 0 ? src - 1 : 0);
        hk = record_header<kSlots>(shfl_rec(rw, src));
        startv = src == 0 ? base : prev_e;
        if (far) {
          const uint32_t v = row_of_serial(rowptr, vr + 32, g.n, gl);
          hk = header<kSlots>(g, v);
          startv = rowptr[v];
        }
      }
      // each neighbor is one independent draw of one sector slot
      const uint32_t val = act ? neighbor<kSlots>(g, hk, (uint32_t)(gl - startv)) : 0u;
      if (act) {
        if (val >= g.n) bad = true;
        cols[gl] = val;
      }
      // next window starts at the vertex of the round's last neighbor
      if (!single) {
        const uint32_t vlast = __shfl_sync(FULL, far ? 0xFFFFFFFFu : vr + (uint32_t)k, 31);
        if (vlast != 0xFFFFFFFFu) {
          vr = vlast;
        } else {
          const uint64_t gl31 = r + 31;
          vr = gl31 < g1 ? warp_row_of(rowptr, g.n, gl31) : vr;
        }
      }
    }
  }
  if (bad && err) atomicOr(err, 1u);
}

// ---------------------------------------------------------------------------
// Plan of the staged sweep (decode_stage_depth 1, 2 or 4), built by the first
// such sweep of a graph: vertices of degree >= 32 become neighbor ranges of at
// most 2048 (hubs are split), the others are grouped by floor(log2(degree)).
//  * A range is decoded by one warp, a neighbor per lane, from whole sectors
//    staged in shared memory (decode_range_kernel);
//  * a small vertex is decoded by one lane, slot after slot; a warp takes 32
//    vertices of one degree class, so its lanes run for similar lengths.
constexpr uint32_t kBigDegree = 32;
#ifndef GRASS_DECODE_RANGE
#define GRASS_DECODE_RANGE 2048
#endif
constexpr uint32_t kRange = GRASS_DECODE_RANGE;  // neighbors per range item

// Sequential decoder of one vertex (one lane), from neighbor 0.
struct SlotSeq {
  const uint32_t *w;
  VHdr h;
  uint32_t c, id;  // slot, index in it
  DrawAt at;
  Sec A;

  __device__ __forceinline__ void load_slot() {
    at = slot_at(h, c);
    A = load_sector(w, at.sec);
  }
  __device__ __forceinline__ void init(const uint32_t *words, const VHdr &hd) {
    w = words;
    h = hd;
    c = id = 0;
    if (h.cb) load_slot();
  }
  __device__ __forceinline__ uint32_t next() {
    if (h.cb == 0) return h.base;
    if (id == h.T) {
      c++;
      id = 0;
      load_slot();
    }
    at.id = id++;
    return draw_value(A, at, h);
  }
};

// Plan construction, in vertex order so that a warp of the small-vertex
// kernel takes 32 neighbouring vertices of one class (adjacent payloads).
// One warp per chunk of kPlanChunk vertices: the count pass stores, per
// chunk, the number of ranges and of vertices in each class; the host turns
// them into per-chunk cursors; the fill pass writes in order (ballot ranks).
constexpr int kCats = 6;  // ranges, then classes floor(log2(d)) = 0..4
constexpr uint32_t kPlanChunk = 1024;

__device__ __forceinline__ void plan_cat(uint32_t d, int &cat, uint32_t &w) {
  if (d >= kBigDegree) {
    cat = 0;
    w = (d + kRange - 1) / kRange;
  } else if (d) {
    cat = 1 + (31 - __clz(d));
    w = 1;
  } else {
    cat = -1;
    w = 0;
  }
}

__global__ void plan_count_kernel(const uint4 *__restrict__ recs, uint32_t n, uint32_t nchunks,
                                  uint32_t *counts) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= nchunks) return;
  uint32_t tot[kCats] = {0, 0, 0, 0, 0, 0};
  const uint32_t v0 = warp * kPlanChunk, v1 = min(n, v0 + kPlanChunk);
  for (uint32_t b = v0; b < v1; b += 32) {
    const uint32_t v = b + lane;
    int cat;
    uint32_t w;
    plan_cat(v < v1 ? recs[v].z : 0u, cat, w);
#pragma unroll
    for (int c = 0; c < kCats; c++) tot[c] += __reduce_add_sync(FULL, cat == c ? w : 0u);
  }
  if (lane < kCats) {
    uint32_t x = 0;
#pragma unroll
    for (int c = 0; c < kCats; c++)
      if (lane == c) x = tot[c];
    counts[(uint64_t)warp * kCats + lane] = x;
  }
}

__global__ void plan_fill_kernel(const uint4 *__restrict__ recs, uint32_t n, uint32_t nchunks,
                                 const unsigned long long *cursors, uint4 *big,
                                 uint32_t *small) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= nchunks) return;
  unsigned long long cur[kCats];
#pragma unroll
  for (int c = 0; c < kCats; c++) cur[c] = cursors[(uint64_t)warp * kCats + c];
  const uint32_t v0 = warp * kPlanChunk, v1 = min(n, v0 + kPlanChunk);
  const unsigned below = (1u << lane) - 1u;
  for (uint32_t b = v0; b < v1; b += 32) {
    const uint32_t v = b + lane;
    const uint32_t d = v < v1 ? recs[v].z : 0u;
    int cat;
    uint32_t w;
    plan_cat(d, cat, w);
    // ranges: exclusive scan of the range counts over the lanes
    uint32_t incl = cat == 0 ? w : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (cat == 0) {
      const unsigned long long p = cur[0] + incl - w;
      for (uint32_t j = 0; j < w; j++)
        big[p + j] = make_uint4(v, j * kRange, min(d, (j + 1) * kRange), 0u);
    }
    cur[0] += __shfl_sync(FULL, incl, 31);
#pragma unroll
    for (int c = 1; c < kCats; c++) {
      const unsigned m = __ballot_sync(FULL, cat == c);
      if (cat == c) small[cur[c] + __popc(m & below)] = v;
      cur[c] += __popc(m);
    }
  }
}

// ---- whole sectors from shared memory, a neighbor per lane ----
// Where the bits of one neighbor are: the shared-memory addresses of the words
// of its slot's head and of its offset, the bits in those words, and 32 less
// the offset's width (a slot's first neighbor has none).
struct Place {
  uint32_t head, head_bit, off, off_bit, drop;
};
__device__ __forceinline__ Place place_of(const VHdr &h, uint32_t r, uint32_t stage) {
  const uint32_t c = div_small(r, h.T), id = r - c * h.T;  // neighbor r of a sector
  const uint32_t hb = h.off + c * h.cb, ob = id ? hb + h.a + (id - 1) * h.b : hb;
  return Place{stage + (hb >> 5) * 4, hb, stage + (ob >> 5) * 4, ob, id ? 32 - h.b : 32u};
}
__device__ __forceinline__ uint32_t lds_bits(uint32_t addr, uint32_t bit, uint32_t drop) {
  uint32_t hi, lo;
  asm volatile("ld.shared.u32 %0, [%2];\n\tld.shared.u32 %1, [%2+4];" : "=r"(hi), "=r"(lo) : "r"(addr));
  return shr_clamp(__funnelshift_l(lo, hi, bit), drop);
}

// The decoding of a vertex's staged sectors by a warp, R = 64 / N whole sectors
// (N = T K neighbors each) a round, two neighbors a lane: the lane's places in
// the R sectors stay the same from round to round, and a neighbor costs its
// field reads, one add and the store.
struct SectorLanes {
  uint32_t N, R, chunk;  // chunk: sectors staged at a time, rounds of R
  Place pl[2];           // the lane's places in a round, in shared memory from address 0
  uint32_t j[2];         // its neighbors there (from i0): a lane without one
                         // (R N < 64) reads place 0 and is never inside [0, len)
  uint32_t *o;           // the lane's first neighbor of the round in the output

  __device__ __forceinline__ void size(const VHdr &h) {
    N = h.T * h.K;
    R = N < 64 ? div_small(64u, N) : 1u;
    chunk = div_small(32u, R) * R;
  }
  // (q0: the first sector, which holds neighbor i0; after size())
  __device__ __forceinline__ void start(const VHdr &h, uint32_t q0, uint32_t i0, uint32_t *out) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t p = u * 32 + lane, k = N < 64 ? div_small(p, N) : 0u;
      const bool ok = k < R;
      pl[u] = place_of(h, ok ? p - k * N : 0u, ok ? k * 32 : 0u);
      j[u] = ok ? q0 * N + p - i0 : 1u << 31;
    }
    o = out + (q0 * N + lane);
  }
  // Sectors q .. q + end - 1 of the vertex, staged at shared address st; its
  // neighbors i0 .. i0 + len - 1 go to out.
  __device__ __forceinline__ void decode(const VHdr &h, uint32_t st, uint32_t q, uint32_t end,
                                         uint32_t i0, uint32_t len, uint32_t *out,
                                         uint32_t &vmax) {
    uint32_t at = st;  // address of the round's first sector
    for (uint32_t e = 0; e < end; e += R) {
      uint32_t v[2];
#pragma unroll
      for (int u = 0; u < 2; u++) v[u] = h.base + lds_bits(pl[u].head + at, pl[u].head_bit, 32 - h.a);
      if (h.T > 1) {  // (warp-uniform)
#pragma unroll
        for (int u = 0; u < 2; u++) v[u] += lds_bits(pl[u].off + at, pl[u].off_bit, pl[u].drop);
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (j[u] < len) {
          o[u * 32] = v[u];
          vmax = max(vmax, v[u]);
        }
        j[u] += R * N;
      }
      if (N > 64) {  // the rest of a sector of more than 64 neighbors
        for (uint32_t r = 64 + (threadIdx.x & 31); r < N; r += 32) {
          const uint32_t i = (q + e) * N + r;
          const Place p = place_of(h, r, at);
          const uint32_t w = h.base + lds_bits(p.head, p.head_bit, 32 - h.a) + lds_bits(p.off, p.off_bit, p.drop);
          if (i - i0 < len) {
            out[i] = w;
            vmax = max(vmax, w);
          }
        }
      }
      o += R * N;
      at += R * 32;
    }
  }
};

// ---- sector staging for the range sweep ----
// Lane 0 of a warp copies each group of up to 32 sectors into one of the warp's
// D shared-memory buffers with one bulk copy (cp.async.bulk, completion counted
// on that buffer's mbarrier), D - 1 groups ahead of the group being decoded (D =
// 1: copy, then decode).  Every wait is bounded: a copy that has not landed
// after kStagePolls polls is reported (error word bit 2, GRASS_E_TIMEOUT) and
// the warp loads the sectors itself from then on, waiting once more, bounded,
// for its copies in flight before it exits.
constexpr int kDecodeWarps = 8;          // warps per range block
constexpr uint32_t kGroupBytes = 1088;   // 32 sectors, and two that the reads of
                                         // lanes without a neighbor may touch
// Polls of the copy's mbarrier before the warp gives up (far beyond the
// microseconds one copy takes).
#ifndef GRASS_STAGE_POLLS
#define GRASS_STAGE_POLLS (1u << 22)
#endif
constexpr uint32_t kStagePolls = GRASS_STAGE_POLLS;
// Test hook, off in the library: with GRASS_STAGE_NEVER_COPY the barrier is
// armed for the copy's bytes but no copy is issued, so the phase never
// completes and every wait runs out -- the timeout path is exercised with
// nothing in flight.
#ifndef GRASS_STAGE_NEVER_COPY
#define GRASS_STAGE_NEVER_COPY 0
#endif

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void stage_bar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Copies `bytes` (a multiple of 16) from 16-byte aligned global `src` to
// shared `dst`; the barrier's current phase completes when they have landed.
__device__ __forceinline__ void stage_copy(void *dst, const void *src, uint32_t bytes,
                                           uint64_t *bar) {
  // order the lanes' earlier reads of dst before the copy's writes
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
  if (GRASS_STAGE_NEVER_COPY) return;
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Waits for phase `parity` of the barrier, at most kStagePolls polls.
__device__ __forceinline__ bool stage_wait(uint64_t *bar, uint32_t parity) {
  for (uint32_t i = 0; i < kStagePolls; i++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Metadata of the 32 range items a warp takes at a time (lane k loads item k's
// record and row start once; the group loop reads them back by broadcast).
struct RangeMeta {
  uint4 rec[32];
  uint64_t base[32];
  uint32_t i0[32], i1[32];
};

// Shared memory of one range warp, in a block of its own that starts on a
// 128-byte boundary: DEPTH staging buffers (each a multiple of 16 bytes, as
// cp.async.bulk requires of its destination) and one for the loads after a
// timeout, the item metadata, then the buffers' mbarriers (8-byte aligned).
template <int DEPTH>
struct WarpSmem {
  static constexpr uint32_t meta_off() { return (DEPTH + 1) * kGroupBytes; }
  static constexpr uint32_t bar_off() { return meta_off() + (uint32_t)sizeof(RangeMeta); }
  static constexpr uint32_t bytes() { return (bar_off() + DEPTH * 8 + 127) / 128 * 128; }
};
static_assert(kGroupBytes % 16 == 0 && sizeof(RangeMeta) % 16 == 0,
              "staging alignment");

// Range sweep: a warp takes 32 range items at a time: lane k loads item k's
// record and row start, and a scan over the lanes numbers the items' groups of
// up to 32 sectors 0 .. total-1 in item order.  The warp then walks that
// sequence, a neighbor per lane, straight to the CSR.  Each group's sectors are
// staged in shared memory DEPTH - 1 groups ahead (1, 2 or 4; across item
// boundaries, see above).  A lane per slot, its neighbors brought into order
// through shared memory, took 1.54 ms at depth 1 on R-MAT s22 ef32 (250 M
// neighbors; slots hold 3 neighbors there); this takes 0.90 ms, and 0.77 at
// depths 2 and 4 (the flat sweep: 0.52).
template <int DEPTH>
__global__ void __launch_bounds__(256) decode_range_kernel(DevGraph g, const uint64_t *rowptr,
                                                           uint32_t *cols,
                                                           const uint4 *__restrict__ items,
                                                           uint64_t nitems, unsigned int *err) {
  extern __shared__ __align__(128) unsigned char le_smem[];
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  using WS = WarpSmem<DEPTH>;
  static_assert(WS::bytes() % 128 == 0 && WS::bar_off() % 8 == 0 && WS::meta_off() % 16 == 0,
                "warp block alignment");
  unsigned char *mine = le_smem + (threadIdx.x >> 5) * WS::bytes();
  RangeMeta &m = *reinterpret_cast<RangeMeta *>(mine + WS::meta_off());
  uint64_t *bars = reinterpret_cast<uint64_t *>(mine + WS::bar_off());
  const uint32_t st = smem_u32(mine);
  uint32_t phase = 0;    // bit b: parity of buffer b's next completion
  uint32_t pending = 0;  // bit b: buffer b has a copy issued and not yet waited for
  bool stage_ok = true;
  if (lane < DEPTH) stage_bar_init(bars + lane);
  __syncwarp();
  uint32_t vmax = 0;
  for (uint64_t tb = warp * 32; tb < nitems; tb += nwarps * 32) {
    // lane k: item tb + k, its sectors qs .. qs + qn - 1 of the layout, in
    // groups of gs
    const uint64_t t = tb + lane;
    uint32_t qs = 0, qn = 0, gs = 1, ng = 0;
    if (t < nitems) {
      const uint4 it = items[t];
      const uint4 r = load_record(g.recs + it.x);
      const VHdr h = record_header<kSlots>(r);
      const uint32_t q = div_small(div_small(it.y, h.T), h.K);
      m.rec[lane] = r;
      m.base[lane] = rowptr[it.x];
      m.i0[lane] = it.y;
      m.i1[lane] = it.z;
      SectorLanes sl;
      sl.size(h);
      gs = sl.chunk;
      qs = h.sec + q;
      qn = div_small(div_small(it.z - 1, h.T), h.K) - q + 1;
      ng = div_small(qn - 1, gs) + 1;
    }
    uint32_t incl = ng;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t excl = incl - ng;  // this item's first group in the sequence
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    __syncwarp();
    // the item holding group s of the sequence (items with groups come first)
    auto item_of = [&](uint32_t s) -> int {
      return __popc(__ballot_sync(FULL, ng > 0 && excl <= s)) - 1;
    };
    // the layout's sectors [qa, qa + n) of group s
    auto group_sectors = [&](uint32_t s, uint32_t &qa, uint32_t &n) {
      const int k = item_of(s);
      const uint32_t kgs = __shfl_sync(FULL, gs, k);
      const uint32_t at = (s - __shfl_sync(FULL, excl, k)) * kgs;
      qa = __shfl_sync(FULL, qs, k) + at;
      n = min(kgs, __shfl_sync(FULL, qn, k) - at);
    };
    auto issue = [&](uint32_t s) {
      if (!stage_ok) return;
      const uint32_t b = s % DEPTH;
      uint32_t qa, n;
      group_sectors(s, qa, n);
      if (lane == 0)
        stage_copy(mine + b * kGroupBytes, g.words + (uint64_t)qa * 8, n * 32u, bars + b);
      pending |= 1u << b;
    };
    if constexpr (DEPTH > 1)
      for (uint32_t s = 0; s + 1 < (uint32_t)DEPTH && s < total; s++) issue(s);
    int kcur = -1;
    VHdr h;
    SectorLanes sl;
    uint32_t *out = nullptr;
    uint32_t i0 = 0, len = 0, q = 0, left = 0;  // the next sector of the vertex, the sectors left
    for (uint32_t s = 0; s < total; s++) {  // warp-uniform
      if (s + DEPTH - 1 < total) issue(s + DEPTH - 1);
      const int k = item_of(s);
      if (k != kcur) {  // the next item: its header and range from the metadata
        kcur = k;
        h = record_header<kSlots>(m.rec[k]);
        i0 = m.i0[k];
        len = m.i1[k] - i0;
        out = cols + m.base[k];
        q = __shfl_sync(FULL, qs, k) - h.sec;
        left = __shfl_sync(FULL, qn, k);
        sl.size(h);
        sl.start(h, q, i0, out);
      }
      uint32_t b = s % DEPTH;
      if (stage_ok) {
        if (__all_sync(FULL, stage_wait(bars + b, (phase >> b) & 1u))) {
          phase ^= 1u << b;
          pending &= ~(1u << b);
        } else {  // the copy did not land in time: report, go on from global memory
          if (lane == 0 && err) atomicOr(err, 2u);
          stage_ok = false;
        }
      }
      const uint32_t n = min(sl.chunk, left);
      if (!stage_ok) {  // into the buffer that no copy writes
        b = DEPTH;
        uint4 *dst = reinterpret_cast<uint4 *>(mine + DEPTH * kGroupBytes);
        const uint4 *src = reinterpret_cast<const uint4 *>(g.words + (uint64_t)(h.sec + q) * 8);
        for (uint32_t w = lane; w < 2 * n; w += 32) dst[w] = __ldg(src + w);
        __syncwarp();
      }
      sl.decode(h, st + b * kGroupBytes, q, n, i0, len, out, vmax);
      q += n;
      left -= n;
      __syncwarp();  // the group's buffer is free for the next group
    }
    __syncwarp();  // the metadata is free for the next batch
  }
  // copies still in flight after a timeout: one more bounded wait each
  for (int b = 0; b < DEPTH; b++)
    if ((pending >> b) & 1u) stage_wait(bars + b, (phase >> b) & 1u);
  if (vmax >= g.n && err) atomicOr(err, 1u);
}

// ---- the flat sweep (the default) ----
// A warp takes one item of the flat plan: a run of consecutive vertices
// [v0, v1) (w == 0), or one vertex's neighbor range [z, w) (hubs, degree >=
// kFlatHub).  It walks a run 32 vertices at a time (lane k loads vertex k's
// record) and decodes one neighbor per lane, straight to the CSR; a neighbor is
// n_0 + head + offset, two fields of one slot, so lanes need nothing from one
// another:
//  * vertices of degree >= kFlatBig one after another (flat_big), from sectors
//    staged in shared memory;
//  * the other vertices together: their neighbors are numbered by a warp scan,
//    and in a round of 32 each lane finds its vertex from the bit mask of the
//    vertices that start in the round (one OR-reduction and a population
//    count), and reads its fields through L1.
// It is bound by instruction issue (67 % of the slots, 117 M warp instructions
// on R-MAT s21 ef16, 63 M neighbors).  The whole decode there took 0.341 ms
// with one lane per slot of LE's own code, 0.466 ms the same way on this layout
// (its slots hold 3 neighbors, so the set-up of a slot is most of the work),
// 0.259 ms with one neighbor per lane whose place in the slots advances by
// wrapping counters, and takes 0.166 ms this way.
#ifndef GRASS_FLAT_VERTEX
#define GRASS_FLAT_VERTEX 16
#endif
// A vertex's share of an item beside its neighbors (32: 0.180 against 0.178 ms).
constexpr uint32_t kFlatVertex = GRASS_FLAT_VERTEX;
#ifndef GRASS_FLAT_BIG
#define GRASS_FLAT_BIG 128
#endif
constexpr uint32_t kFlatHub = kRange;  // degree from which a vertex is split into ranges
// Degree from which a vertex is decoded by itself: its set-up is some 250 warp
// instructions, and a round of 32 neighbors then takes about 25, against 70 in
// a group (0.166 ms at 96, 128 and 192, 0.174 at 64; at most 2048, see FlatSmem::vb).
constexpr uint32_t kFlatBig = GRASS_FLAT_BIG;

// Warps per block, one item each, and resident blocks per SM (64 registers).
// Items differ in cost, and a block's place is free only when its last warp is
// done: two warps a block ran the sweep in 0.178 ms, eight in 0.191; 12 or 20
// blocks in 0.196 and 0.191.
#ifndef GRASS_FLAT_WARPS
#define GRASS_FLAT_WARPS 2
#endif
#ifndef GRASS_DECODE_FLAT_MIN_BLOCKS
#define GRASS_DECODE_FLAT_MIN_BLOCKS 16
#endif
constexpr int kFlatWarps = GRASS_FLAT_WARPS;

// A warp's share of shared memory.
struct FlatSmem {
  uint32_t stage[32 * 8 + 4];  // 32 sectors, and the word that a field's read may touch
  // the group's small vertices with neighbors, in order:
  uint4 va[32];  // n_0; sector; bit in it | a << 8 | b << 14 | T << 20 | K << 26; first
                 // neighbor's number in the group
  uint4 vb[32];  // 2^16 / T and 2^16 / K rounded up; cb; first entry in the CSR less the
                 // number of the first neighbor, from the group's first entry
};

// Copies one word to shared memory through L1, which brings its sector there
// and holds no register while it is on the way.
__device__ __forceinline__ void prefetch_l1(uint32_t *dump, const uint32_t *p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dump)), "l"(p) : "memory");
}
__device__ __forceinline__ void prefetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The field of `width` (0..32) bits at bit `off` from word w.
__device__ __forceinline__ uint32_t word_field(const uint32_t *w, uint32_t off, uint32_t width) {
  const uint32_t *q = w + (off >> 5);
  return shr_clamp(__funnelshift_l(q[1], q[0], off), 32u - width);
}

// Neighbors [i0, i1) of a vertex of header h (warp-uniform, cb > 0) to
// out[i0 .. i1); vmax: the largest value written so far.  The vertex's sectors
// are consecutive: the warp copies up to 32 of them at a time into shared
// memory with two 16-byte loads a lane, the next ones already on their way in
// registers.
__device__ __forceinline__ void flat_big(const uint32_t *words, const VHdr &h, uint32_t i0,
                                         uint32_t i1, uint32_t *out, uint32_t *stage,
                                         uint32_t &vmax) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t q0 = i0 ? div_small(div_small(i0, h.T), h.K) : 0u;
  const uint32_t nq = div_small(div_small(i1 - 1, h.T), h.K) - q0 + 1;
  const uint32_t len = i1 - i0, st = smem_u32(stage);
  SectorLanes sl;
  sl.size(h);
  sl.start(h, q0, i0, out);
  const uint4 *src = reinterpret_cast<const uint4 *>(words + (uint64_t)(h.sec + q0) * 8) + lane;
  uint4 *dst = reinterpret_cast<uint4 *>(stage) + lane;
  const uint32_t half = lane >> 1;  // the lane's sector of 16
  uint4 x = make_uint4(0, 0, 0, 0), y = x;
  if (half < nq) x = __ldg(src);
  if (half + 16 < nq) y = __ldg(src + 32);
  for (uint32_t q = 0; q < nq; q += sl.chunk) {  // warp-uniform
    dst[0] = x;
    dst[32] = y;
    __syncwarp();
    src += 2 * sl.chunk;
    if (q + sl.chunk + half < nq) x = __ldg(src);
    if (q + sl.chunk + half + 16 < nq) y = __ldg(src + 32);
    sl.decode(h, st, q0 + q, min(sl.chunk, nq - q), i0, len, out, vmax);
    __syncwarp();
  }
}

template <int MODE>
__global__ void __launch_bounds__(32 * kFlatWarps, GRASS_DECODE_FLAT_MIN_BLOCKS) decode_flat_kernel(DevGraph g, const uint64_t *__restrict__ rowptr,
                                                          uint32_t *__restrict__ cols,
                                                          const uint4 *__restrict__ items,
                                                          uint64_t nitems, unsigned int *err) {
  __shared__ __align__(16) FlatSmem smem[kFlatWarps];
  FlatSmem &sm = smem[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t upto = 0xFFFFFFFFu >> (31 - lane);  // this lane and those below
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t vmax = 0;
  for (uint64_t t = warp; t < nitems; t += nwarps) {
    const uint4 it = items[t];
    const bool run = it.w == 0;
    const uint32_t v0 = it.x, v1 = run ? it.y : it.x + 1;
    for (uint32_t vb = v0; vb < v1; vb += 32) {
      const uint32_t v = vb + lane;
      uint4 r = make_uint4(0, 0, 0, 0);
      uint64_t ob = 0;
      if (v < v1) {
        r = graph_record<MODE>(g, v);
        ob = rowptr[v];
      }
      const bool big = r.z >= kFlatBig;
      // the small vertices of the group
      const uint32_t d = big ? 0u : r.z;
      uint32_t incl = d;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      const uint32_t ex = d ? incl - d : 0xFFFFFFFFu, total = __shfl_sync(FULL, incl, 31);
      const unsigned has = __ballot_sync(FULL, d > 0);
      const uint64_t ob0 = __shfl_sync(FULL, ob, 0);
      if (d) {
        const VHdr h = record_header<MODE>(r);
        const uint32_t at = __popc(has & upto) - 1;
        sm.va[at] = make_uint4(h.base, h.sec, h.off | (r.y & ~0xFFu), ex);
        sm.vb[at] = make_uint4(65535u / h.T + 1, 65535u / h.K + 1, h.cb, (uint32_t)(ob - ob0) - ex);
        // bring the vertex's lines into L1 (a word of each into a dump) while
        // the others are set up
        const uint32_t lines = h.cb ? (div_small(div_small(d - 1, h.T), h.K) + (h.sec & 3u)) / 4 + 1 : 0;
        const uint32_t *p = g.words + (uint64_t)(h.sec & ~3u) * 8;
#pragma unroll
        for (uint32_t l = 0; l < kFlatBig * 32 / 1024 + 2; l++)
          if (l < lines) prefetch_l1(&sm.stage[lane], p + l * 32);
      }
      __syncwarp();
      uint32_t *out0 = cols + ob0;
      uint32_t before = 0xFFFFFFFFu;  // the vertices that start before the round, less one
      for (uint32_t j = 0; j < total; j += 32) {
        const unsigned starts = __reduce_or_sync(FULL, __funnelshift_lc(0u, 1u, ex - j));
        const uint32_t own = before + __popc(starts & upto);
        before += __popc(starts);
        if (j + lane < total) {
          const uint4 A = sm.va[own], B = sm.vb[own];
          // neighbor i of its vertex: slot c, index id; exact for i < 2048
          const uint32_t i = j + lane - A.w;
          const uint32_t c = (i * B.x) >> 16, id = i - c * ((A.z >> 20) & 63u);
          const uint32_t q = (c * B.y) >> 16, at = (A.z & 255u) + (c - q * (A.z >> 26)) * B.z;
          const uint32_t *w = g.words + (uint64_t)(A.y + q) * 8;
          const uint32_t a = (A.z >> 8) & 63u, b = (A.z >> 14) & 63u;
          uint32_t x = A.x;
          if (a) x += word_field(w, at, a);
          if (id) x += word_field(w, at + a + (id - 1) * b, b);
          vmax = max(vmax, x);
          out0[B.w + j + lane] = x;
        }
      }
      prefetch_wait();  // (before the dump is used again)
      __syncwarp();
      // the large ones
      for (unsigned m = __ballot_sync(FULL, big); m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const VHdr h = record_header<MODE>(shfl_rec(r, k));
        uint32_t *out = cols + __shfl_sync(FULL, ob, k);
        flat_big(g.words, h, run ? 0u : it.z, run ? h.d : it.w, out, sm.stage, vmax);
      }
      __syncwarp();  // the group's shared memory is free
    }
  }
  if (vmax >= g.n && err) atomicOr(err, 1u);
}

// Flat plan: items in vertex order.  One warp per chunk of kPlanChunk
// vertices.  A vertex of degree >= kFlatHub becomes ceil(d / kRange) range
// items (v, v + 1, i0, i1); the others form runs, a run starting at the
// chunk's first vertex, after a hub, and wherever the chunk's running sum of
// degree + kFlatVertex crosses a multiple of kRange: a group of 32 vertices
// costs the latency of its records however few neighbors it has, and without
// the second term the runs of low-degree vertices, which come last in
// graph_sort's order, held most warps idle at the end of the sweep.  Runs get (v0, 0, 0, 0) here; their end
// is the next item's first vertex (flat_plan_link_kernel).
template <bool FILL>
__global__ void flat_plan_kernel(const uint4 *__restrict__ recs, uint32_t n, uint32_t nchunks,
                                 uint32_t *counts, const unsigned long long *cursors,
                                 uint4 *items) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= nchunks) return;
  const uint32_t v0 = warp * kPlanChunk, v1 = min(n, v0 + kPlanChunk);
  unsigned long long cur = FILL ? cursors[warp] : 0ull;
  uint32_t tot = 0;
  uint64_t carry = 0;       // the chunk's sum before this sub-chunk
  bool prev_hub = true;     // (the chunk's first vertex starts a run)
  uint64_t prev_win = 0;
  for (uint32_t b = v0; b < v1; b += 32) {
    const uint32_t v = b + lane;
    const uint32_t d = v < v1 ? recs[v].z : 0u;
    const bool hub = v < v1 && d >= kFlatHub;
    const uint32_t cost = d + kFlatVertex;
    uint64_t incl = cost;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    const uint64_t pre = carry + incl - cost;  // the chunk's sum before v
    const uint64_t win = pre / kRange;
    const uint32_t hub_up = __shfl_up_sync(FULL, (uint32_t)hub, 1);
    const bool ph = lane ? hub_up != 0u : prev_hub;
    const uint64_t pw_up = __shfl_up_sync(FULL, win, 1);
    const uint64_t pw = lane ? pw_up : prev_win;
    const bool start = v < v1 && !hub && (ph || win != pw);
    const uint32_t w_items = hub ? (d + kRange - 1) / kRange : (start ? 1u : 0u);
    uint32_t wi = w_items;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, wi, o);
      if (lane >= o) wi += y;
    }
    if (FILL && w_items) {
      const unsigned long long at = cur + wi - w_items;
      if (hub) {
        for (uint32_t j = 0; j < w_items; j++)
          items[at + j] = make_uint4(v, v + 1, j * kRange, min(d, (j + 1) * kRange));
      } else {
        items[at] = make_uint4(v, 0u, 0u, 0u);
      }
    }
    const uint32_t wsum = __shfl_sync(FULL, wi, 31);
    cur += wsum;
    tot += wsum;
    carry += __shfl_sync(FULL, incl, 31);
    prev_hub = __shfl_sync(FULL, (uint32_t)hub, 31) != 0u;
    prev_win = __shfl_sync(FULL, win, 31);
  }
  if (!FILL && lane == 0) counts[warp] = tot;
}

// A run ends where the next item starts (or at n).
__global__ void flat_plan_link_kernel(uint4 *items, uint64_t nitems, uint32_t n) {
  const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (k >= nitems) return;
  if (items[k].w == 0) items[k].y = k + 1 < nitems ? items[k + 1].x : n;
}

__global__ void __launch_bounds__(256) decode_small_kernel(DevGraph g, const uint64_t *rowptr,
                                                             uint32_t *cols,
                                                             const uint32_t *__restrict__ verts,
                                                             uint64_t nv, unsigned int *err) {
  bool bad = false;
  const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t q0 = (uint64_t)blockIdx.x * blockDim.x; q0 < nv; q0 += nt) {
    const uint64_t q = q0 + threadIdx.x;
    uint32_t d = 0;
    uint32_t *out = nullptr;
    SlotSeq st;
    if (q < nv) {
      const uint32_t v = verts[q];
      const VHdr h = header<kSlots>(g, v);
      d = h.d;
      out = cols + rowptr[v];
      st.init(g.words, h);
    }
    for (uint32_t k = 0; k < d; k++) {
      const uint32_t val = st.next();
      bad |= val >= g.n;
      out[k] = val;
    }
  }
  if (bad && err) atomicOr(err, 1u);
}

}  // namespace

static void launch_plan_kernels(const grass_graph *g, const uint64_t *rowptr, uint32_t *cols,
                                unsigned int *err, cudaStream_t s);

template <int DEPTH>
static void launch_range(const DevGraph &v, const uint64_t *rowptr, uint32_t *cols,
                         const grass_graph *g, unsigned grid, unsigned int *err, cudaStream_t s) {
  const uint32_t smem = kDecodeWarps * WarpSmem<DEPTH>::bytes();
  // The opt-in to more than 48 KB of dynamic shared memory holds for the current
  // device, so it goes with each launch.  (Its error is the launch's.)
  if (cudaFuncSetAttribute(decode_range_kernel<DEPTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return;
  decode_range_kernel<DEPTH><<<grid, 32 * kDecodeWarps, smem, s>>>(
      v, rowptr, cols, g->d_plan_big, g->plan_nbig, err);
}

static void launch_range_depth(const DevGraph &v, const uint64_t *rowptr, uint32_t *cols,
                               const grass_graph *g, unsigned grid, unsigned int *err,
                               cudaStream_t s) {
  switch (g->tuning.decode_stage_depth) {
    case 1: launch_range<1>(v, rowptr, cols, g, grid, err, s); break;
    case 2: launch_range<2>(v, rowptr, cols, g, grid, err, s); break;
    default: launch_range<4>(v, rowptr, cols, g, grid, err, s);
  }
}

// Builds the flat plan (once) on stream s.
static int build_flat_plan(const grass_graph *g, cudaStream_t s) {
  const uint32_t n = (uint32_t)g->info.n;
  const uint32_t nchunks = (n + kPlanChunk - 1) / kPlanChunk;
  const unsigned pgrid = (nchunks + 7) / 8;  // 8 warps (chunks) per block
  uint32_t *cnt = nullptr;
  unsigned long long *cur = nullptr;
  GRASS_CUDA(cudaMalloc(&cnt, (uint64_t)nchunks * sizeof(uint32_t)));
  cudaError_t e = cudaMalloc(&cur, (uint64_t)nchunks * sizeof(unsigned long long));
  std::vector<uint32_t> hc(nchunks);
  std::vector<unsigned long long> hcur(nchunks);
  uint64_t tot = 0;
  if (e == cudaSuccess) {
    flat_plan_kernel<false><<<pgrid, 256, 0, s>>>(g->d_recs, n, nchunks, cnt, nullptr, nullptr);
    count_launch();
    e = cudaMemcpyAsync(hc.data(), cnt, hc.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) {
    for (uint32_t ch = 0; ch < nchunks; ch++) {
      hcur[ch] = tot;
      tot += hc[ch];
    }
    e = cudaMalloc(&g->d_plan_flat, std::max<uint64_t>(tot, 1) * sizeof(uint4));
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(cur, hcur.data(), hcur.size() * sizeof(unsigned long long),
                        cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    flat_plan_kernel<true><<<pgrid, 256, 0, s>>>(g->d_recs, n, nchunks, nullptr, cur,
                                                 g->d_plan_flat);
    count_launch();
    if (tot) {
      flat_plan_link_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(g->d_plan_flat, tot, n);
      count_launch();
    }
    e = cudaStreamSynchronize(s);
  }
  cudaFree(cnt);
  cudaFree(cur);
  if (e != cudaSuccess) {
    cudaFree(g->d_plan_flat);
    g->d_plan_flat = nullptr;
    return cuda_fail(e, "flat decode plan build");
  }
  g->plan_nflat = tot;
  g->plan_flat_ok = true;
  return GRASS_OK;
}

static void launch_flat(const grass_graph *g, const uint64_t *rowptr, uint32_t *cols,
                        unsigned int *err, cudaStream_t s) {
  if (!g->plan_nflat) return;
  const DevGraph v = g->view();
  const unsigned grid =
      (unsigned)std::min<uint64_t>((g->plan_nflat + kFlatWarps - 1) / kFlatWarps, 1u << 30);
  decode_flat_kernel<kSlots><<<grid, 32 * kFlatWarps, 0, s>>>(v, rowptr, cols, g->d_plan_flat, g->plan_nflat, err);
  count_launch();
}

int launch_decode_planned(const grass_graph *g, const uint64_t *rowptr, uint32_t *cols,
                          unsigned int *err, cudaStream_t s) {
  const uint32_t n = (uint32_t)g->info.n;
  if (!g->info.num_edges) return GRASS_OK;
  if (g->tuning.decode_stage_depth == 0) {  // the flat sweep
    {
      std::lock_guard<std::mutex> lk(g->plan_mu);
      if (!g->plan_flat_ok) {
        const int rc = build_flat_plan(g, s);
        if (rc) return rc;
      }
    }
    launch_flat(g, rowptr, cols, err, s);
    return GRASS_OK;
  }
  {
    std::lock_guard<std::mutex> lk(g->plan_mu);
    if (!g->plan_ok) {
      const uint32_t nchunks = (n + kPlanChunk - 1) / kPlanChunk;
      const unsigned pgrid = (nchunks + 7) / 8;  // 8 warps (chunks) per block
      uint32_t *cnt = nullptr;
      unsigned long long *cur = nullptr;
      GRASS_CUDA(cudaMalloc(&cnt, (uint64_t)nchunks * kCats * sizeof(uint32_t)));
      cudaError_t e = cudaMalloc(&cur, (uint64_t)nchunks * kCats * sizeof(unsigned long long));
      if (e != cudaSuccess) {
        cudaFree(cnt);
        return cuda_fail(e, "decode plan scratch");
      }
      plan_count_kernel<<<pgrid, 256>>>(g->d_recs, n, nchunks, cnt);
      count_launch();
      std::vector<uint32_t> hc((uint64_t)nchunks * kCats);
      std::vector<unsigned long long> hcur(hc.size());
      e = cudaMemcpy(hc.data(), cnt, hc.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost);
      // cursors: ranges in chunk order; the classes back to back, each in chunk order
      uint64_t tot[kCats] = {0, 0, 0, 0, 0, 0};
      for (uint64_t k = 0; k < hc.size(); k++) tot[k % kCats] += hc[k];
      uint64_t base[kCats] = {0, 0, 0, 0, 0, 0};
      for (int c = 2; c < kCats; c++) base[c] = base[c - 1] + tot[c - 1];
      for (uint32_t ch = 0; ch < nchunks; ch++)
        for (int c = 0; c < kCats; c++) {
          hcur[(uint64_t)ch * kCats + c] = base[c];
          base[c] += hc[(uint64_t)ch * kCats + c];
        }
      g->plan_nbig = tot[0];
      g->plan_nsmall = 0;
      for (int c = 1; c < kCats; c++) g->plan_nsmall += tot[c];
      if (e == cudaSuccess)
        e = cudaMalloc(&g->d_plan_big, std::max<uint64_t>(g->plan_nbig, 1) * sizeof(uint4));
      if (e == cudaSuccess)
        e = cudaMalloc(&g->d_plan_small, std::max<uint64_t>(g->plan_nsmall, 1) * sizeof(uint32_t));
      if (e == cudaSuccess)
        e = cudaMemcpy(cur, hcur.data(), hcur.size() * sizeof(unsigned long long),
                       cudaMemcpyHostToDevice);
      if (e == cudaSuccess) {
        plan_fill_kernel<<<pgrid, 256>>>(g->d_recs, n, nchunks, cur, g->d_plan_big,
                                         g->d_plan_small);
        count_launch();
        e = cudaDeviceSynchronize();
      }
      cudaFree(cnt);
      cudaFree(cur);
      if (e != cudaSuccess) {
        cudaFree(g->d_plan_big);
        cudaFree(g->d_plan_small);
        g->d_plan_big = nullptr;
        g->d_plan_small = nullptr;
        return cuda_fail(e, "decode plan build");
      }
      g->plan_ok = true;
    }
  }
  launch_plan_kernels(g, rowptr, cols, err, s);
  return GRASS_OK;
}

bool launch_decode_if_planned(const grass_graph *g, const uint64_t *rowptr, uint32_t *cols,
                              unsigned int *err, cudaStream_t s) {
  const bool flat = g->tuning.decode_stage_depth == 0;
  {
    std::lock_guard<std::mutex> lk(g->plan_mu);
    if (flat ? !g->plan_flat_ok : !g->plan_ok) return false;
  }
  if (!g->info.num_edges) return true;
  if (flat) launch_flat(g, rowptr, cols, err, s);
  else launch_plan_kernels(g, rowptr, cols, err, s);
  return true;
}

// The range and small-vertex sweeps of a built plan (launches only).
static void launch_plan_kernels(const grass_graph *g, const uint64_t *rowptr, uint32_t *cols,
                                unsigned int *err, cudaStream_t s) {
  const int dev = g->device;
  const DevGraph v = g->view();
  const int per_sm = 8;
  if (g->plan_nbig) {
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((g->plan_nbig + 7) / 8, (uint64_t)sm_count(dev) * per_sm));
    launch_range_depth(v, rowptr, cols, g, grid, err, s);
    count_launch();
  }
  if (g->plan_nsmall) {
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((g->plan_nsmall + 255) / 256, (uint64_t)sm_count(dev) * per_sm));
    decode_small_kernel<<<grid, 256, 0, s>>>(v, rowptr, cols, g->d_plan_small,
                                                  g->plan_nsmall, err);
    count_launch();
  }
}

void launch_decode_all(const DevGraph &g, const uint64_t *rowptr, uint32_t *cols, uint64_t E,
                       unsigned int *err, cudaStream_t s) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (!E) return;
  const uint64_t tasks = (E + kTaskNeighbors - 1) / kTaskNeighbors;
  const uint64_t blocks_needed = (tasks + 7) / 8;
  const unsigned grid = (unsigned)std::max<uint64_t>(
      1, std::min<uint64_t>(blocks_needed, (uint64_t)sm_count(dev) * 8));
  decode_all_kernel<<<grid, 256, 0, s>>>(g, rowptr, cols, E, err);
  count_launch();
}

}  // namespace grass
