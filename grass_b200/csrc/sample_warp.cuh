// sample_warp.cuh -- warp-level sampling routines shared by the standalone
// multi-RW kernel and the batched persistent kernel.  Each routine is run by
// all 32 lanes of one warp and needs at most the warp's own shared-memory
// slot (SmemHdr), so a persistent warp can pick up any job type from a work
// queue.
#pragma once
#include "device_common.cuh"

namespace grass {

constexpr unsigned kFull = 0xFFFFFFFFu;

// Path output of a warp's 32 walkers, one column (step) after the other.
// Step-major columns are stored as they come, 32 consecutive entries.  In the
// walk-major layout a column's entries lie L + 1 apart: stored one by one, each
// would be a write of 4 bytes to a sector of its own, and a sector would be
// touched eight times (200,003 walkers x 40, R-MAT s22 ef32: 0.240 ms against
// 0.217 ms step-major).  So COLS columns are collected in shared memory and
// written by rows, COLS lanes a walker (0.225 ms).  The layouts are separate
// instances: with the row code in its loop a step-major walk of 4,096 x 80
// took 57 us instead of 53.
template <int COLS, bool WALK_MAJOR>
struct PathOut {
  static constexpr uint32_t kPitch = COLS + 1;  // (rows in different banks)
  static constexpr uint32_t kWords = 32 * kPitch;
  uint32_t *paths;
  uint32_t *stage;      // kWords of the warp (walk-major)
  uint64_t W, w0, end;  // walkers of the job; the warp's: [w0, min(w0 + 32, end))
  uint32_t L;

  // Column c of the lane's walker w0 + lane (called by the whole warp).
  __device__ __forceinline__ void put(uint32_t c, uint32_t v) const {
    const uint32_t lane = threadIdx.x & 31;
    if constexpr (!WALK_MAJOR) {
      if (w0 + lane < end) store_out_u32(paths + (uint64_t)c * W + w0 + lane, v);
    } else {
      put_row(c, v);
    }
  }
  __device__ __forceinline__ void put_row(uint32_t c, uint32_t v) const {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = c % COLS;
    stage[lane * kPitch + k] = v;
    if (k + 1 < COLS && c < L) return;
    __syncwarp();
    const uint32_t col = lane % COLS, row = lane / COLS;
    if (col <= k) {
      uint32_t *p = paths + (w0 + row) * (uint64_t)(L + 1) + (c - k) + col;
#pragma unroll 4
      for (uint32_t r = row; r < 32; r += 32 / COLS, p += (32 / COLS) * (uint64_t)(L + 1))
        if (w0 + r < end) store_out_u32(p, stage[r * kPitch + col]);
    }
    __syncwarp();
  }
};

// The record of a walker's vertex (INVALID_VERTEX: stopped, no record).
template <int MODE>
__device__ __forceinline__ uint4 walk_record(const DevGraph &g, uint32_t v) {
  return v != INVALID_VERTEX ? graph_record<MODE>(g, v) : make_uint4(0u, 0u, 0u, 0u);
}

// One step of DEPTH independent walkers from their vertices' records; v[k]:
// the walker's next vertex, word(k) its random word of the step.  Every sector
// load is issued before any is decoded, so a lane's loads overlap.
template <int MODE, int DEPTH, class Word>
__device__ __forceinline__ void walk_step(const DevGraph &g, const uint4 (&rec)[DEPTH],
                                          uint32_t (&v)[DEPTH], Word word, uint64_t &cnt,
                                          bool &bad) {
  VHdr h[DEPTH];
  DrawAt at[DEPTH];
  Sec A[DEPTH];
  uint32_t nv[DEPTH];
#pragma unroll
  for (int k = 0; k < DEPTH; k++) {
    const uint32_t rnd = word(k);
    h[k] = record_header<MODE>(rec[k]);
    nv[k] = h[k].base;  // (degree 1)
    const uint32_t i = mulhi_u32(rnd, h[k].d);
    if constexpr (MODE == kCsr) {
      if (h[k].d) nv[k] = load_cold_u32(g.cols + h[k].P + i);
    } else if (h[k].cb) {
      at[k] = draw_at(h[k], i);
      A[k] = load_sector(g.words, at[k].sec);
    }
  }
#pragma unroll
  for (int k = 0; k < DEPTH; k++) {
    if constexpr (MODE != kCsr)
      if (h[k].cb) nv[k] = draw_value(A[k], at[k], h[k]);
    const bool ok = nv[k] < g.n;
    if (h[k].d) {
      bad |= !ok;
      cnt += ok;
    }
    v[k] = h[k].d && ok ? nv[k] : INVALID_VERTEX;
  }
}

// Random walk of walkers [b, e) of a job of W walkers (starts[0..W)), DEPTH
// walkers per lane per pass, `stride` walkers apart (a pass takes the walkers
// [wb + k stride, + 32) below e).  Walker w draws word step & 3 of
// Philox(seed; step >> 2, id0 + w, .., TAG_RW).  stage: kPathStageWords<DEPTH>
// words of the warp for the walk-major layout.
template <int DEPTH>
constexpr uint32_t kPathStageWords = DEPTH * PathOut<16 / DEPTH, true>::kWords;

template <int MODE, int DEPTH, bool WALK_MAJOR>
__device__ __forceinline__ void rw_pass(const DevGraph &g, const uint32_t *starts, uint64_t W,
                                        uint32_t L, uint64_t seed, uint64_t id0,
                                        uint32_t *paths, uint64_t wb, uint64_t stride, uint64_t e,
                                        uint32_t *stage, uint64_t &cnt, bool &bad) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t v[DEPTH];
  u32x4 r[DEPTH];
  using Out = PathOut<16 / DEPTH, WALK_MAJOR>;
  auto out = [&](int k) { return Out{paths, stage + k * Out::kWords, W, wb + k * stride, e, L}; };
#pragma unroll
  for (int k = 0; k < DEPTH; k++) {
    const uint64_t w = wb + k * stride + lane;
    v[k] = INVALID_VERTEX;
    r[k] = u32x4{0, 0, 0, 0};
    const uint32_t s0 = w < e ? starts[w] : INVALID_VERTEX;
    if (s0 < g.n) v[k] = s0;
    out(k).put(0, s0);
  }
  // A step's record loads go out as soon as its vertices are known: the path
  // stores and the Philox rounds run while they are on the way.
  uint4 rec[DEPTH];
#pragma unroll
  for (int k = 0; k < DEPTH; k++) rec[k] = walk_record<MODE>(g, v[k]);
  for (uint32_t s = 0; s < L; s++) {
    walk_step<MODE, DEPTH>(g, rec, v, [&](int k) {
      if ((s & 3) == 0) {
        const uint64_t id = id0 + wb + k * stride + lane;
        r[k] = philox4x32_10(seed, s >> 2, (uint32_t)id, (uint32_t)(id >> 32), TAG_RW);
      }
      return pick(r[k], s & 3);
    }, cnt, bad);
    if (s + 1 < L) {
#pragma unroll
      for (int k = 0; k < DEPTH; k++) rec[k] = walk_record<MODE>(g, v[k]);
    }
#pragma unroll
    for (int k = 0; k < DEPTH; k++) out(k).put(s + 1, v[k]);
  }
}

// ---------------------------------------------------------------------------
// k-hop of one seed (KHopApp, GT/src/apps/khop/khop.cu:1-79, with runtime
// fanouts).  For each hop the frontier is taken in groups of 32 transits, and a
// group's f * 32 draws are spread over the lanes.

struct KhopArgs {
  uint32_t hops;
  uint32_t fan[GRASS_MAX_HOPS];
  uint64_t width[GRASS_MAX_HOPS];  // prod_{j<=h} fan[j]
  uint32_t *out[GRASS_MAX_HOPS];
  uint64_t seed;
};

// A warp's share of shared memory.
constexpr uint32_t kFrontier = 64;
struct SmemHdr {
  uint4 kept[2][kFrontier];  // records of a frontier of up to kFrontier vertices (degree 0:
                             // none), for this hop and the next
  uint4 rec[32];             // a group's records, where the frontier is in global memory
  uint64_t ob[32];           // and its transits' first output slots, with parts > 1
  uint32_t words[128];       // random words of 128 draws
};

// With parts > 1, `parts` warps share the seed: warp `part` takes the subtrees
// of the first hop's children part, part + parts, ... for every later hop.
// Every part draws the first hop itself (the same values: each writes them,
// only part 0 counts them), so no warp waits for another.  Draws keep their
// Philox slot, so the output is the same for any number of parts.
//
// Draw slot k of hop h (its index in the seed's hop-h output row) uses word
// k & 3 of Philox(seed; k >> 2, s, s >> 32, TAG_KHOP | h).  The frontier is
// taken G transits at a time (G = 32, fewer only for fanouts above 2^27, so
// that a group's draw count fits 32 bits).  With one part and G = 32 a group's
// slots are contiguous (pc f + j, pc a multiple of 32), so the lanes compute the
// group's Philox blocks once per 128 draws and hand the words out through
// shared memory; otherwise each draw computes its own block.  INFLIGHT: draws a
// lane has in flight at once (every load is issued before any is decoded).  On a
// CSR a draw is one column load.
//
// A frontier of up to kFrontier vertices stays in shared memory as records,
// loaded by the lanes that drew the vertices: the next hop then starts with its
// slot loads, where it would first read the vertices back and then their
// records.  A lane's place (transit, draw under it) advances by 32 / f and
// 32 % f.  65,536 seeds x (25, 10) on R-MAT s22 ef32: 0.232 ms, of which the 8.9
// M sectors that miss L2 take 0.19 at the rate of random reads; 0.251 with
// 64-bit divisions for the place and the parent, words by shuffle, every
// frontier read back and two draws in flight.
template <int MODE, int INFLIGHT = 1>
__device__ __forceinline__ void khop_seed_warp(const DevGraph &g, const uint32_t *seeds,
                                               const KhopArgs &A, uint64_t s, SmemHdr &my,
                                               uint64_t &cnt, bool &bad, uint32_t part = 0,
                                               uint32_t parts = 1) {
  static_assert(INFLIGHT == 1 || INFLIGHT == 2 || INFLIGHT == 4, "INFLIGHT in {1, 2, 4}");
  const uint32_t lane = threadIdx.x & 31;
  const bool whole = parts == 1;
  auto record = [&](uint32_t v) {
    return v < g.n ? graph_record<MODE>(g, v) : make_uint4(0u, 0u, 0u, 0u);
  };
  __syncwarp();  // (an earlier seed's reads of the shared memory are done)
  if (lane == 0) my.kept[0][0] = record(seeds[s]);
  __syncwarp();
  uint32_t buf = 0;  // which of my.kept holds this hop's frontier
  bool kept = true;  // ... if it does
  for (uint32_t hop = 0; hop < A.hops; hop++) {
    const uint32_t f = A.fan[hop];
    const uint64_t width = A.width[hop];
    uint64_t P = 1, Q = 1;  // this part's parents: Q consecutive ones under each of its
    if (hop) {              // first-hop children
      P = A.width[hop - 1];
      if (!whole) {
        Q = P / A.fan[0];
        P = part < A.fan[0] ? (uint64_t)((A.fan[0] - part + parts - 1) / parts) * Q : 0;
      }
    }
    const bool count = hop || part == 0;
    const bool last_hop = hop + 1 == A.hops;
    const bool keep = whole && !last_hop && width <= kFrontier;
    const uint32_t G = f < (1u << 27) ? 32u : (uint32_t)max(1ull, 0xFFFFFFFFull / f);
    const bool contig = whole && G == 32;
    const uint32_t dp = f < 32 ? 32 / f : f == 32 ? 1u : 0u, dk = f < 32 ? 32 - dp * f : f == 32 ? 0u : 32u;
    const uint32_t p0 = f < 32 ? lane / f : 0u, k0 = lane - p0 * f;
    uint32_t *out = A.out[hop] + s * width;
    const uint32_t *prev = hop ? A.out[hop - 1] + s * A.width[hop - 1] : nullptr;
    uint32_t drawn = 0;
    for (uint64_t pc = 0; pc < P; pc += G) {
      const uint4 *rec = kept ? my.kept[buf] + pc : my.rec;
      if (!kept) {
        __syncwarp();
        if (lane < G && pc + lane < P) {
          uint64_t par = pc + lane;
          if (!whole && hop) par = (part + par / Q * parts) * Q + par % Q;
          my.ob[lane] = par * f;
          my.rec[lane] = record(prev[par]);
        }
        __syncwarp();
      } else if (!whole) {
        if (lane == 0) my.ob[0] = 0;  // (the seed, the only frontier that parts keep)
        __syncwarp();
      }
      const uint32_t total = (uint32_t)min((uint64_t)G, P - pc) * f;  // < 2^32 by the choice of G
      const uint64_t sbase = pc * f;  // with one part: slot = sbase + j
      uint32_t pl = p0, k = k0;       // the lane's draw: transit of the group, draw under it
      for (uint32_t j0 = 0;; j0 += 32 * INFLIGHT) {  // warp-uniform
        if (contig && (j0 & 127u) == 0) {
          __syncwarp();
          const u32x4 r = philox4x32_10(A.seed, (uint32_t)((sbase + j0) >> 2) + lane, (uint32_t)s,
                                        (uint32_t)(s >> 32), TAG_KHOP | hop);
          reinterpret_cast<uint4 *>(my.words)[lane] = make_uint4(r.x, r.y, r.z, r.w);
          __syncwarp();
        }
        // phase 1: each draw's load; phase 2: its value, stored
        Sec S[INFLIGHT];
        DrawAt at[INFLIGHT];
        uint32_t nv[INFLIGHT], y[INFLIGHT], d[INFLIGHT];
        uint64_t slot[INFLIGHT];
#pragma unroll
        for (int u = 0; u < INFLIGHT; u++) {
          const uint32_t j = j0 + u * 32 + lane;
          d[u] = y[u] = 0;
          nv[u] = INVALID_VERTEX;
          slot[u] = ~0ull;
          if (j < total && j >= j0) {  // (j may pass 2^32)
            const uint4 r = rec[pl];
            const VHdr h = record_header<MODE>(r);
            slot[u] = whole ? sbase + j : my.ob[pl] + k;
            uint32_t word;
            if (contig)
              word = my.words[j & 127u];
            else
              word = pick(philox4x32_10(A.seed, (uint32_t)(slot[u] >> 2), (uint32_t)s,
                                        (uint32_t)(s >> 32), TAG_KHOP | hop), (int)(slot[u] & 3));
            const uint32_t i = mulhi_u32(word, h.d);
            d[u] = h.d;
            nv[u] = h.base;
            if constexpr (MODE == kCsr) {
              if (h.d) nv[u] = load_cold_u32(g.cols + h.P + i);
            } else if (h.cb) {
              y[u] = r.y;
              at[u] = draw_at(h, i);
              S[u] = load_sector(g.words, at[u].sec);
            }
          }
          k += dk;
          pl += dp;
          if (k >= f) {
            k -= f;
            pl++;
          }
        }
#pragma unroll
        for (int u = 0; u < INFLIGHT; u++) {
          if (slot[u] == ~0ull) continue;
          if constexpr (MODE != kCsr) {
            if (y[u]) {  // (a slot has bits, so its record's y is not 0)
              VHdr h = record_header<MODE>(make_uint4(0u, y[u], 0u, nv[u]));
              nv[u] = draw_value(S[u], at[u], h);
            }
          }
          const bool ok = nv[u] < g.n;
          if (d[u]) {
            bad |= !ok;
            drawn += ok;
          }
          const uint32_t v = d[u] && ok ? nv[u] : INVALID_VERTEX;
          if (last_hop) store_out_u32(out + slot[u], v);
          else out[slot[u]] = v;  // (read back by the next hop if it is not kept)
          if (keep) my.kept[buf ^ 1][slot[u]] = record(v);
        }
        if (total - j0 <= 32 * INFLIGHT) break;
      }
    }
    if (count) cnt += drawn;
    __syncwarp();
    kept = keep;
    buf ^= 1;
  }
}

// Start vertex i of a multi-RW job whose roots are drawn from its seed: the
// stream of grass_mrw_roots (word i & 3 of Philox(seed; i >> 2, 0, 0,
// TAG_MRW_ROOT), mapped to [0, n)).
__device__ __forceinline__ uint32_t mrw_root(uint32_t n, uint64_t seed, uint64_t i) {
  const u32x4 r = philox4x32_10(seed, (uint32_t)(i >> 2), 0u, 0u, TAG_MRW_ROOT);
  return mulhi_u32(pick(r, (int)(i & 3)), n);
}

// Multi random walk of one sample (MultiRWApp, GT/src/apps/multiRW/multiRW.cu:3-112),
// the walker of each step picked uniformly, by one warp.  vtx[0..R) holds the
// walkers' vertices (shared or global memory), updated in place.  Step t draws
// from Philox(seed; t, sample, .., TAG_MRW): word 0 picks the walker, word 1
// the neighbor.  So the walkers of 32 steps are known before any of them is
// taken, and steps of different walkers do not depend on one another: lane k
// takes step t0 + k, in as many rounds as one walker has steps among the 32
// (2 or 3 with 80 walkers), where one step after the other left 31 lanes idle
// through 32 chains of two memory reads (65,536 samples of 80 walkers x 100
// steps, R-MAT s22 ef32: 0.21 ms against 1.70 ms).
template <int MODE>
__device__ __forceinline__ void mrw_uniform_warp(const DevGraph &g, uint32_t *vtx, uint32_t R,
                                                 uint32_t T, uint64_t seed, uint64_t sample,
                                                 uint32_t *src, uint32_t *dst, uint64_t &cnt,
                                                 bool &bad) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t t0 = 0; t0 < T; t0 += 32) {
    const uint32_t t = t0 + lane;
    const u32x4 r = philox4x32_10(seed, t, (uint32_t)sample, (uint32_t)(sample >> 32), TAG_MRW);
    const uint32_t x = t < T ? mulhi_u32(r.x, R) : INVALID_VERTEX;
    const unsigned same = __match_any_sync(kFull, x);
    const uint32_t turn = __popc(same & ((1u << lane) - 1u));
    const uint32_t turns = __reduce_max_sync(kFull, t < T ? turn : 0u) + 1;
    uint32_t from = INVALID_VERTEX, to = INVALID_VERTEX;
    for (uint32_t k = 0; k < turns; k++) {  // warp-uniform
      if (t < T && turn == k) {
        from = vtx[x];
        const VHdr h = record_header<MODE>(from < g.n ? graph_record<MODE>(g, from)
                                                      : make_uint4(0u, 0u, 0u, 0u));
        if (h.d) {
          const uint32_t nv = neighbor<MODE>(g, h, mulhi_u32(r.y, h.d));
          if (nv < g.n) {
            to = vtx[x] = nv;
            cnt++;
          } else {
            bad = true;
          }
        }
      }
      __syncwarp();
    }
    if (t < T) {
      store_out_u32(src + sample * T + t, from);
      store_out_u32(dst + sample * T + t, to);
    }
  }
}

// Records (all zero: none) of the walkers' vertices vtx[0..R) into rec[0..R),
// lanes gl of the G that share a sample; four independent loads in flight.
template <int MODE, int G>
__device__ __forceinline__ void mrw_load_records(const DevGraph &g, const uint32_t *vtx,
                                                 uint4 *rec, uint32_t R, uint32_t gl) {
  for (uint32_t c0 = 0; c0 < R; c0 += 4 * G) {
    uint4 r[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i = c0 + k * G + gl;
      const uint32_t x = i < R ? vtx[i] : INVALID_VERTEX;
      r[k] = x < g.n ? graph_record<MODE>(g, x) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i = c0 + k * G + gl;
      if (i < R) rec[i] = r[k];
    }
  }
}

// Inclusive sum over the lanes of groups of G.
template <int G, class Sum>
__device__ __forceinline__ Sum group_scan(Sum v) {
  const uint32_t gl = threadIdx.x & (G - 1);
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const Sum y = __shfl_up_sync(kFull, v, o, G);
    if (gl >= (uint32_t)o) v += y;
  }
  return v;
}

// Moves walker x along the neighbor that a random word picks: writes the edge
// and the walker's new vertex and record, and returns the change of its degree.
template <int MODE>
__device__ __forceinline__ int64_t mrw_move(const DevGraph &g, uint32_t *vtx, uint4 *rec,
                                            uint32_t x, uint32_t word, uint32_t *src, uint32_t *dst,
                                            uint64_t &cnt, bool &bad) {
  const VHdr h = record_header<MODE>(rec[x]);
  const uint32_t nv = neighbor<MODE>(g, h, mulhi_u32(word, h.d));
  store_out_u32(src, vtx[x]);
  if (nv >= g.n) {
    bad = true;
    store_out_u32(dst, INVALID_VERTEX);
    return 0;
  }
  const uint4 r = graph_record<MODE>(g, nv);
  store_out_u32(dst, nv);
  vtx[x] = nv;
  rec[x] = r;
  cnt++;
  return (int64_t)r.z - h.d;
}

// Multi random walk with the walker of each step picked in proportion to its
// degree, one sample per warp.  A step depends on the one before it through
// two memory reads (the slot, then the new vertex's record, for its degree).
// The sample's state is vtx[0..R) and rec[0..R), each walker's vertex and
// record, in shared or global memory; lane j keeps the total degree of walkers
// [j B, (j + 1) B), B = ceil(R / 32).  A pick scans the 32 sums with shuffles,
// then the chosen B entries 32 at a time.  Step t: words 2, 0 of its Philox
// block (see mrw_uniform_warp) pick the walker, word 1 the neighbor; lane k
// computes the block of step t0 + k.
template <int MODE>
__device__ __forceinline__ void mrw_degree_warp(const DevGraph &g, uint32_t *vtx, uint4 *rec,
                                                uint32_t R, uint32_t T, uint64_t seed,
                                                uint64_t sample, uint32_t *src, uint32_t *dst,
                                                uint64_t &cnt, bool &bad) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t B = (R + 31) / 32;
  mrw_load_records<MODE, 32>(g, vtx, rec, R, lane);
  __syncwarp();
  uint64_t bsum = 0;  // this lane's walkers
  for (uint32_t i = lane * B; i < min(R, (lane + 1) * B); i++) bsum += rec[i].z;
  for (uint32_t t0 = 0; t0 < T; t0 += 32) {
    const u32x4 mine =
        philox4x32_10(seed, t0 + lane, (uint32_t)sample, (uint32_t)(sample >> 32), TAG_MRW);
    const uint32_t tn = min(32u, T - t0);
    for (uint32_t k = 0; k < tn; k++) {
      const uint32_t rx = __shfl_sync(kFull, mine.x, k), ry = __shfl_sync(kFull, mine.y, k),
                     rz = __shfl_sync(kFull, mine.z, k);
      const uint64_t io = sample * T + t0 + k;
      const uint64_t incl = group_scan<32>(bsum), wsum = __shfl_sync(kFull, incl, 31);
      if (wsum == 0) {  // (warp-uniform)
        if (lane == 0) src[io] = dst[io] = INVALID_VERTEX;
        continue;
      }
      const uint64_t u = mulhi_u64(((uint64_t)rz << 32) | rx, wsum);
      // bucket: the first lane whose inclusive sum exceeds u; then its first walker
      const int Lb = __ffs(__ballot_sync(kFull, incl > u)) - 1;
      uint64_t acc = __shfl_sync(kFull, incl - bsum, Lb);
      const uint32_t b0 = (uint32_t)Lb * B, b1 = min(R, b0 + B);
      uint32_t x = b1 - 1;
      for (uint32_t c0 = b0; c0 < b1; c0 += 32) {  // two passes for R <= 2048
        const uint32_t i = c0 + lane;
        const uint64_t ci = group_scan<32>((uint64_t)(i < b1 ? rec[i].z : 0u));
        const unsigned hit = __ballot_sync(kFull, i < b1 && acc + ci > u);
        if (hit) {
          x = c0 + (uint32_t)(__ffs(hit) - 1);
          break;
        }
        acc += __shfl_sync(kFull, ci, 31);
      }
      int64_t gain = 0;
      if (lane == 0) gain = mrw_move<MODE>(g, vtx, rec, x, ry, src + io, dst + io, cnt, bad);
      gain = __shfl_sync(kFull, gain, 0);
      if (lane == x / B) bsum += gain;
      __syncwarp();
    }
  }
}

// The same by G lanes of a warp, 32 / G samples side by side, for few walkers
// (B = ceil(R / G) a lane) with their state in shared memory.  (Called by
// whole warps; `live`: this group has a sample.)  The lane whose walkers hold
// the pick finds it among them and moves it, so a step is one scan of the
// group's sums, a short search and the two memory reads, with nothing to hand
// round.  (8,192 samples of 80 walkers x 100 steps, R-MAT s22 ef32: 0.191 ms,
// all of them under way at once and bound by the chain of reads, 1.9 us a
// step; 0.216 ms with the walker found and moved by the group together, 0.370
// ms with one sample per warp, of which 4,736 fit.)  Sum: uint32_t where no sum of R degrees reaches 2^32.
template <int MODE, int G, class Sum>
__device__ __forceinline__ void mrw_degree_group(const DevGraph &g, bool live, uint32_t *vtx,
                                                 uint4 *rec, uint32_t R, uint32_t T, uint64_t seed,
                                                 uint64_t sample, uint32_t *src, uint32_t *dst,
                                                 uint64_t &cnt, bool &bad) {
  const uint32_t gl = threadIdx.x & (G - 1);
  const uint32_t B = (R + G - 1) / G, x0 = min(R, gl * B), x1 = min(R, x0 + B);
  if (live) mrw_load_records<MODE, G>(g, vtx, rec, R, gl);
  __syncwarp();
  Sum bsum = 0;  // this lane's walkers [x0, x1)
  if (live)
    for (uint32_t i = x0; i < x1; i++) bsum += rec[i].z;
  for (uint32_t t0 = 0; t0 < T; t0 += G) {
    const u32x4 mine =
        philox4x32_10(seed, t0 + gl, (uint32_t)sample, (uint32_t)(sample >> 32), TAG_MRW);
    const uint32_t tn = min((uint32_t)G, T - t0);
    for (uint32_t k = 0; k < tn; k++) {
      const uint32_t rx = __shfl_sync(kFull, mine.x, k, G), ry = __shfl_sync(kFull, mine.y, k, G),
                     rz = __shfl_sync(kFull, mine.z, k, G);
      const uint64_t io = sample * T + t0 + k;
      const Sum incl = group_scan<G>(bsum), wsum = __shfl_sync(kFull, incl, G - 1, G);
      const Sum u = (Sum)mulhi_u64(((uint64_t)rz << 32) | rx, wsum), before = incl - bsum;
      if (u >= before && u < incl) {  // the pick is among this lane's walkers
        Sum left = u - before;
        uint32_t x = x0;
        for (;; x += 4) {  // four degrees at a time
          uint32_t d[4];
#pragma unroll
          for (int q = 0; q < 4; q++) d[q] = x + q < x1 ? rec[x + q].z : 0xFFFFFFFFu;
          uint32_t past = 0;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (past == (uint32_t)q && left >= d[q]) {
              left -= d[q];
              past++;
            }
          }
          if (past < 4) {
            x += past;
            break;
          }
        }
        bsum += (Sum)mrw_move<MODE>(g, vtx, rec, x, ry, src + io, dst + io, cnt, bad);
      } else if (wsum == 0 && live && gl == 0) {
        src[io] = dst[io] = INVALID_VERTEX;
      }
      __syncwarp();
    }
  }
}

}  // namespace grass
