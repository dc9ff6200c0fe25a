// sample_warp.cuh -- warp-level sampling routines shared by the standalone
// multi-RW kernel and the batched persistent kernel.  Each routine is run by
// all 32 lanes of one warp and needs at most the warp's own shared-memory
// slot (SmemHdr), so a persistent warp can pick up any job type from a work
// queue.
#pragma once
#include "device_common.cuh"

namespace grass {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ void path_store(uint32_t *paths, int layout, uint64_t W, uint32_t L,
                                           uint64_t w, uint32_t s, uint32_t v) {
  if (layout == GRASS_LAYOUT_WALK_MAJOR) store_out_u32(paths + w * (uint64_t)(L + 1) + s, v);
  else store_out_u32(paths + (uint64_t)s * W + w, v);
}

// One step of DEPTH independent walkers: every record load is issued before
// the random words are made, and every sector load before any is decoded, so
// a lane's loads overlap and the Philox rounds run while the records arrive.
// v[k] is the walker's vertex (INVALID_VERTEX: stopped), word(k) its random
// word of the step.
template <int MODE, int DEPTH, class Word>
__device__ __forceinline__ void walk_step(const DevGraph &g, uint32_t (&v)[DEPTH], Word word,
                                          uint64_t &cnt, bool &bad) {
  uint4 rec[DEPTH];
#pragma unroll
  for (int k = 0; k < DEPTH; k++)
    rec[k] = v[k] != INVALID_VERTEX ? graph_record<MODE>(g, v[k]) : make_uint4(0u, 0u, 0u, 0u);
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
// walkers per lane per pass.  Same draws as rw_kernel:
// walker w uses Philox(seed; step>>2, w0+w, .., TAG_RW).
template <int MODE, int DEPTH>
__device__ __forceinline__ void rw_warp(const DevGraph &g, const uint32_t *starts, uint64_t W,
                                        uint32_t L, uint64_t seed, uint64_t w0, int layout,
                                        uint32_t *paths, uint64_t b, uint64_t e, uint64_t &cnt,
                                        bool &bad) {
  const int lane = threadIdx.x & 31;
  for (uint64_t wb = b; wb < e; wb += 32 * DEPTH) {  // warp-uniform
    uint32_t v[DEPTH];
    u32x4 r[DEPTH];
#pragma unroll
    for (int k = 0; k < DEPTH; k++) {
      const uint64_t w = wb + (uint64_t)k * 32 + lane;
      v[k] = INVALID_VERTEX;
      r[k] = u32x4{0, 0, 0, 0};
      if (w < e) {
        const uint32_t s0 = starts[w];
        path_store(paths, layout, W, L, w, 0, s0);
        v[k] = s0 < g.n ? s0 : INVALID_VERTEX;
      }
    }
    for (uint32_t s = 0; s < L; s++) {
      walk_step<MODE, DEPTH>(g, v, [&](int k) {
        if ((s & 3) == 0) {
          const uint64_t id = w0 + wb + (uint64_t)k * 32 + lane;
          r[k] = philox4x32_10(seed, s >> 2, (uint32_t)id, (uint32_t)(id >> 32), TAG_RW);
        }
        return pick(r[k], s & 3);
      }, cnt, bad);
#pragma unroll
      for (int k = 0; k < DEPTH; k++) {
        const uint64_t w = wb + (uint64_t)k * 32 + lane;
        if (w < e) path_store(paths, layout, W, L, w, s + 1, v[k]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// k-hop of one seed (KHopApp, GT/src/apps/khop/khop.cu:1-79, with runtime
// fanouts).  For each hop the frontier is taken in chunks of 32 transits:
// lane p decodes the header of transit p into the warp's shared-memory slot,
// then the chunk's f*32 draws are spread over the lanes.

struct KhopArgs {
  uint32_t hops;
  uint32_t fan[GRASS_MAX_HOPS];
  uint64_t width[GRASS_MAX_HOPS];  // prod_{j<=h} fan[j]
  uint32_t *out[GRASS_MAX_HOPS];
  uint64_t seed;
};

// A warp's frontier group: transit i's record (degree 0: none) and first
// output slot (parent index * fanout).
struct SmemHdr {
  uint4 rec[32];
  uint64_t ob[32];
};

// Word k (0..3) of a Philox block held as four values.
__device__ __forceinline__ uint32_t pick4(uint32_t x, uint32_t y, uint32_t z, uint32_t w, int k) {
  return k == 0 ? x : k == 1 ? y : k == 2 ? z : w;
}

// With parts > 1, `parts` warps share the seed: warp `part` takes the subtrees
// of the first hop's children part, part + parts, ... for every later hop.
// Every part draws the first hop itself (the same values: each writes them,
// only part 0 counts them), so no warp waits for another.  Draws keep their
// Philox slot, so the output is the same for any number of parts.
//
// Draw slot k of hop h (its index in the seed's hop-h output row) uses word
// k & 3 of Philox(seed; k >> 2, s, s >> 32, TAG_KHOP | h).  The frontier is
// taken G transits at a time (G = 32, fewer only for fanouts above 2^27, so
// that a group's draw count fits 32 bits): lane p loads the header of transit
// p, then the group's G f draws are spread over the lanes.  With one part and
// G = 32 a group's slots are contiguous (pc f + j, pc a multiple of 32), so the
// lanes compute the group's Philox blocks once per 128 draws, lane l block l of
// the window, and hand the words out by shuffles; otherwise each draw
// computes its own block.  INFLIGHT: draws a lane has in flight at once (every
// load is issued before any is decoded).  On a CSR a draw is one column load.
template <int MODE, int INFLIGHT = 1>
__device__ __forceinline__ void khop_seed_warp(const DevGraph &g, const uint32_t *seeds,
                                               const KhopArgs &A, uint64_t s, SmemHdr &my,
                                               uint64_t &cnt, bool &bad,
                                               uint32_t part = 0, uint32_t parts = 1) {
  static_assert(INFLIGHT == 1 || INFLIGHT == 2 || INFLIGHT == 4, "INFLIGHT in {1, 2, 4}");
  const int lane = threadIdx.x & 31;
  for (uint32_t hop = 0; hop < A.hops; hop++) {
    const uint32_t f = A.fan[hop];
    const uint64_t Mf = div_magic(f);
    const uint64_t Pall = hop ? A.width[hop - 1] : 1;
    // this part's parents: Q consecutive ones under each of its first-hop children
    const uint64_t Q = hop ? Pall / A.fan[0] : 1;
    const uint64_t mine = hop ? (part < A.fan[0] ? (A.fan[0] - part + parts - 1) / parts : 0) : 1;
    const uint64_t P = mine * Q;
    auto parent = [&](uint64_t k) -> uint64_t {
      return hop ? (part + (k / Q) * parts) * Q + k % Q : 0;
    };
    const bool count = hop || part == 0;
    const bool last_hop = hop + 1 == A.hops;
    const uint32_t G = f < (1u << 27) ? 32u : (uint32_t)max(1ull, 0xFFFFFFFFull / f);
    const bool contig = parts == 1 && G == 32;
    uint32_t *out = A.out[hop] + s * A.width[hop];
    const uint32_t *prev = hop ? A.out[hop - 1] + s * A.width[hop - 1] : nullptr;
    for (uint64_t pc = 0; pc < P; pc += G) {
      const uint64_t p = pc + lane;
      uint32_t t = INVALID_VERTEX;
      uint64_t ob = 0;
      if (lane < (int)G && p < P) {
        const uint64_t par = parent(p);
        ob = par * f;
        t = hop ? prev[par] : seeds[s];
      }
      my.rec[lane] = t < g.n ? graph_record<MODE>(g, t) : make_uint4(0u, 0u, 0u, 0u);
      my.ob[lane] = ob;
      __syncwarp();
      const uint32_t nP = (uint32_t)min((uint64_t)G, P - pc);
      const uint32_t total = nP * f;  // < 2^32 by the choice of G
      const uint64_t sbase = pc * f;  // contiguous groups: slot = sbase + j
      u32x4 rw = u32x4{0, 0, 0, 0};
      for (uint64_t j0 = 0; j0 < total; j0 += 32 * INFLIGHT) {  // warp-uniform
        if (contig && (j0 & 127u) == 0)
          rw = philox4x32_10(A.seed, (uint32_t)(((sbase + j0) >> 2) + (uint64_t)lane), (uint32_t)s,
                             (uint32_t)(s >> 32), TAG_KHOP | hop);
        uint32_t rnd[INFLIGHT];
#pragma unroll
        for (int u = 0; u < INFLIGHT; u++) {
          rnd[u] = 0;
          if (contig) {  // warp-uniform
            // block ((j0 mod 128) + 32 u + lane) / 4 of the window, word lane & 3
            const int src = (int)((((uint32_t)j0 & 127u) + 32u * u + (uint32_t)lane) >> 2);
            const uint32_t x = __shfl_sync(kFull, rw.x, src), y = __shfl_sync(kFull, rw.y, src);
            const uint32_t z = __shfl_sync(kFull, rw.z, src), w = __shfl_sync(kFull, rw.w, src);
            rnd[u] = pick4(x, y, z, w, lane & 3);
          }
        }
        // phase 1: each draw's load; phase 2: its value, stored
        Sec S[INFLIGHT];
        DrawAt at[INFLIGHT];
        uint32_t col[INFLIGHT];
#pragma unroll
        for (int u = 0; u < INFLIGHT; u++) {
          const uint64_t j = j0 + (uint64_t)u * 32 + lane;
          if (j >= total) continue;
          const uint32_t pl = div_by((uint32_t)j, f, Mf);
          const VHdr h = record_header<MODE>(my.rec[pl]);
          col[u] = h.base;  // (degree 1)
          if (MODE == kCsr ? h.d == 0 : h.cb == 0) continue;
          if (!contig) {
            const uint64_t slot = my.ob[pl] + ((uint32_t)j - pl * f);
            rnd[u] = pick(philox4x32_10(A.seed, (uint32_t)(slot >> 2), (uint32_t)s,
                                        (uint32_t)(s >> 32), TAG_KHOP | hop),
                          (int)(slot & 3));
          }
          const uint32_t i = mulhi_u32(rnd[u], h.d);
          if constexpr (MODE == kCsr) {
            col[u] = load_cold_u32(g.cols + h.P + i);
          } else {
            at[u] = draw_at(h, i);
            S[u] = load_sector(g.words, at[u].sec);
          }
        }
#pragma unroll
        for (int u = 0; u < INFLIGHT; u++) {
          const uint64_t j = j0 + (uint64_t)u * 32 + lane;
          if (j >= total) continue;
          const uint32_t pl = div_by((uint32_t)j, f, Mf);
          const VHdr h = record_header<MODE>(my.rec[pl]);
          const uint64_t slot = contig ? sbase + j : my.ob[pl] + ((uint32_t)j - pl * f);
          uint32_t nv = col[u];
          if constexpr (MODE != kCsr)
            if (h.cb) nv = draw_value(S[u], at[u], h);
          const bool ok = nv < g.n;
          if (h.d) {
            bad |= !ok;
            if (ok && count) cnt++;
          }
          nv = h.d && ok ? nv : INVALID_VERTEX;
          if (last_hop) store_out_u32(out + slot, nv);
          else out[slot] = nv;  // read back by the next hop
        }
      }
      __syncwarp();
    }
  }
}

// Start vertex i of a multi-RW job whose roots are drawn from its seed: the
// stream of grass_mrw_roots (word i & 3 of Philox(seed; i >> 2, 0, 0,
// TAG_MRW_ROOT), mapped to [0, n)).
__device__ __forceinline__ uint32_t mrw_root(uint32_t n, uint64_t seed, uint64_t i) {
  const u32x4 r = philox4x32_10(seed, (uint32_t)(i >> 2), 0u, 0u, TAG_MRW_ROOT);
  return mulhi_u32(pick(r, (int)(i & 3)), n);
}

// Multi random walk of one sample (MultiRWApp, GT/src/apps/multiRW/multiRW.cu:3-112).
// The sample's state is vtx[0..R), the walkers' vertices (updated in place),
// and rec[0..R), each walker's 16-byte vertex record (all zero for a vertex
// out of range), in shared or global memory.  Keeping the record makes a
// step cost two dependent DRAM reads (payload, then the new vertex's record)
// instead of three.  Lane j keeps the total degree of walkers [j*B, (j+1)*B),
// B = ceil(R/32); a degree-proportional pick scans the 32 bucket sums with
// shuffles, then the chosen bucket 32 entries at a time.  Step t draws from
// Philox(seed; t, sample, .., TAG_MRW): word 0 (+ word 2 as high half) picks
// the walker, word 1 the neighbor.  Lane k computes the block of step
// t0 + k, so one Philox evaluation per lane serves 32 steps.
template <int MODE>
__device__ __forceinline__ void mrw_warp(const DevGraph &g, uint32_t *vtx, uint4 *rec, uint32_t R,
                                         uint32_t T, int select, uint64_t seed, uint64_t sample,
                                         uint32_t *src, uint32_t *dst, uint64_t &cnt, bool &bad) {
  const int lane = threadIdx.x & 31;
  const uint32_t B = (R + 31) / 32;
  // Records of the start vertices: four independent loads in flight per lane.
  for (uint32_t c0 = 0; c0 < R; c0 += 128) {
    uint4 r[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i = c0 + k * 32 + lane;
      const uint32_t x = i < R ? vtx[i] : INVALID_VERTEX;
      r[k] = x < g.n ? graph_record<MODE>(g, x) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i = c0 + k * 32 + lane;
      if (i < R) rec[i] = r[k];
    }
  }
  __syncwarp();
  uint64_t bsum = 0;  // this lane's bucket
  for (uint32_t i = lane * B; i < min(R, (lane + 1) * B); i++) bsum += rec[i].z;
  uint64_t wsum = bsum;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(kFull, wsum, o);
  for (uint32_t t0 = 0; t0 < T; t0 += 32) {
    const u32x4 mine =
        philox4x32_10(seed, t0 + lane, (uint32_t)sample, (uint32_t)(sample >> 32), TAG_MRW);
    const uint32_t tn = min(32u, T - t0);
    for (uint32_t k = 0; k < tn; k++) {
      const uint32_t rx = __shfl_sync(kFull, mine.x, k), ry = __shfl_sync(kFull, mine.y, k),
                     rz = __shfl_sync(kFull, mine.z, k);
      const uint64_t io = sample * T + t0 + k;
      uint32_t x;
      if (select == GRASS_SELECT_DEGREE) {
        if (wsum == 0) {
          if (lane == 0) {
            src[io] = INVALID_VERTEX;
            dst[io] = INVALID_VERTEX;
          }
          continue;
        }
        const uint64_t u = mulhi_u64(((uint64_t)rz << 32) | rx, wsum);
        // bucket: first lane whose inclusive prefix exceeds u
        uint64_t incl = bsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint64_t y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        const int Lb = __ffs(__ballot_sync(kFull, incl > u)) - 1;
        uint64_t acc = __shfl_sync(kFull, incl - bsum, Lb);  // prefix before the bucket
        const uint32_t b0 = (uint32_t)Lb * B, b1 = min(R, b0 + B);
        x = b1 - 1;
        for (uint32_t c0 = b0; c0 < b1; c0 += 32) {  // two passes for R <= 2048
          const uint32_t i = c0 + lane;
          const uint64_t d = i < b1 ? rec[i].z : 0u;
          uint64_t ci = d;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(kFull, ci, o);
            if (lane >= o) ci += y;
          }
          const unsigned hit = __ballot_sync(kFull, i < b1 && acc + ci > u);
          if (hit) {
            x = c0 + (uint32_t)(__ffs(hit) - 1);
            break;
          }
          acc += __shfl_sync(kFull, ci, 31);
        }
      } else {
        x = mulhi_u32(rx, R);
      }
      // lane 0 moves walker x
      uint32_t nd = 0, od = 0;
      bool moved = false;
      if (lane == 0) {
        const uint32_t v = vtx[x];
        const uint4 r = rec[x];
        od = r.z;
        src[io] = v;
        if (od == 0) {
          dst[io] = INVALID_VERTEX;
        } else {
          const VHdr h = record_header<MODE>(r);
          const uint32_t nv = neighbor<MODE>(g, h, mulhi_u32(ry, h.d));
          if (nv >= g.n) {
            bad = true;
            dst[io] = INVALID_VERTEX;
          } else {
            dst[io] = nv;
            cnt++;
            const uint4 nr = graph_record<MODE>(g, nv);
            vtx[x] = nv;
            rec[x] = nr;
            nd = nr.z;
            moved = true;
          }
        }
      }
      moved = __shfl_sync(kFull, moved, 0);
      if (moved) {
        nd = __shfl_sync(kFull, nd, 0);
        od = __shfl_sync(kFull, od, 0);
        if (lane == (int)(x / B)) bsum = bsum - od + nd;
        wsum = wsum - od + nd;
      }
      __syncwarp();
    }
  }
}

}  // namespace grass
