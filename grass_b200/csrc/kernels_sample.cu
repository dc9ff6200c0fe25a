// kernels_sample.cu -- random walk, k-hop and multi-RW kernels over the
// compressed graph, plus the uncompressed-CSR baselines with the same RNG.
//
// The reference runs every app step as a separate transit-parallel pass:
// sample kernel, then a global radix sort inverting sample->transit, run-
// length encoding, a scan and a kernel-type partition, with blocking syncs in
// between (GT/src/grass.cu:1573-1998).  For fanout-1 walks nothing is shared
// between walkers on the same transit, so here one launch runs all steps:
// each thread owns DEPTH walkers and interleaves them, which keeps DEPTH
// independent decode chains in flight per thread.
#include "graph.h"
#include "launch_rules.h"
#include "mrw_cta.cuh"
#include "sample_warp.cuh"

#include <mutex>

// Resident 512-thread blocks per SM each walk kernel is compiled for (its
// register budget).  With two or four walkers a lane the compressed walk needs
// more than the 64 registers of two blocks (it spilled 160 and 748 bytes) and is
// compiled for one: 1M walkers x 40, R-MAT s22 ef32, step-major, ms with two /
// one: two walkers 1.15 / 1.01, four 1.31 / 1.09; 4,096 walkers, us: 48 / 36 and
// 107 / 50 (with the grid of rw_launch_depth).
#ifndef GRASS_RW_MIN_BLOCKS
#define GRASS_RW_MIN_BLOCKS 2
#endif
#ifndef GRASS_RW_CSR_MIN_BLOCKS
#define GRASS_RW_CSR_MIN_BLOCKS 2
#endif

namespace grass {

namespace {

__device__ __forceinline__ void store_path(uint32_t *paths, int layout, uint64_t W, uint32_t L,
                                           uint64_t w, uint32_t s, uint32_t v) {
  if (layout == GRASS_LAYOUT_WALK_MAJOR) store_out_u32(paths + w * (uint64_t)(L + 1) + s, v);
  else store_out_u32(paths + (uint64_t)s * W + w, v);
}

// w0: walker id of starts[0] -- draws use walker id w0 + w, so a batch split
// into chunks produces the same walks as one launch.
template <int MODE, int DEPTH>
__global__ void __launch_bounds__(512, DEPTH == 1 ? GRASS_RW_MIN_BLOCKS : 1) rw_kernel(DevGraph g, const uint32_t *__restrict__ starts,
                                                 uint64_t W, uint32_t L, uint64_t seed,
                                                 uint64_t w0, int layout,
                                                 uint32_t *__restrict__ paths,
                                                 unsigned long long *edges, unsigned int *err) {
  extern __shared__ uint32_t path_stage[];  // walk-major: kPathStageWords<DEPTH> words a warp
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  uint32_t *stage = path_stage + (threadIdx.x >> 5) * kPathStageWords<DEPTH>;
  uint64_t cnt = 0;
  bool bad = false;
  for (uint64_t wb = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); wb < W;
       wb += nthreads * DEPTH) {  // warp-uniform
    if (layout == GRASS_LAYOUT_WALK_MAJOR)
      rw_pass<MODE, DEPTH, true>(g, starts, W, L, seed, w0, paths, wb, nthreads, W, stage, cnt, bad);
    else
      rw_pass<MODE, DEPTH, false>(g, starts, W, L, seed, w0, paths, wb, nthreads, W, stage, cnt, bad);
  }
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// ---------------------------------------------------------------------------
// Second-order (node2vec) walk.  One walker per thread.  Try k of step s
// draws Philox(seed; s, w, w >> 32, TAG_N2V | k): word 0 picks the candidate
// from N(v), word 1 is compared with the candidate's acceptance threshold
// (return to u, a neighbor of u, or farther).  The membership test searches
// u's sorted neighbor list (has_neighbor).
struct N2vArgs {
  uint32_t L, max_tries;
  int layout;
  uint64_t seed, w0;
  uint64_t t_ret, t_in, t_out;  // acceptance thresholds in [0, 2^32]
};

// The head of the first slot of sector q (from the vertex's first): one field
// of at most 32 bits at the sector's first bit.
__device__ __forceinline__ uint32_t sector_head(const DevGraph &g, const VHdr &h, uint32_t q) {
  return shr_clamp(ldw(g.words + (uint64_t)(h.sec + q) * 8), 32u - h.a);
}

// The last index in [lo, hi] whose key is <= x, given key(lo) <= x, for
// nondecreasing keys: a binary search, one probe per round.  (An 8-way
// search, seven independent probes per round, was slower: with a million
// walkers in flight latency is hidden anyway, and it loads more.)
template <class Key>
__device__ __forceinline__ uint32_t last_le(uint32_t lo, uint32_t hi, uint32_t x, Key key) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo + 1) / 2;
    if (key(mid) <= x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The same with P independent probes a round, for keys that lie side by side
// in memory: with 3 for the fences and for a line's sectors the walk below took
// 1.28 ms instead of 1.43; with 5, 7 and 15 for the fences 1.28, 1.29 and 1.46.
template <int P, class Key>
__device__ __forceinline__ uint32_t last_le_wide(uint32_t lo, uint32_t hi, uint32_t x, Key key) {
  while (lo < hi) {
    const uint32_t n = hi - lo;  // candidates above lo, cut into P + 1 parts
    uint32_t nlo = lo, nhi = hi;
    bool le[P];
#pragma unroll
    for (int i = 1; i <= P; i++) le[i - 1] = key(lo + (n * i + P) / (P + 1)) <= x;
#pragma unroll
    for (int i = 1; i <= P; i++) {
      const uint32_t p = lo + (n * i + P) / (P + 1);
      if (le[i - 1]) nlo = p;
    }
#pragma unroll
    for (int i = P; i >= 1; i--) {
      const uint32_t p = lo + (n * i + P) / (P + 1);
      if (!le[i - 1]) nhi = p - 1;
    }
    lo = nlo;
    hi = nhi;
  }
  return lo;
}

// Whether x is a neighbor of the vertex of header h.  Compressed: a search for
// the one sector that can hold x, over the fences (see build_fences_kernel) for
// its line and over the line's sectors' first heads, then for the slot and the
// neighbor inside that sector, in registers.  CSR: a search of the row.
template <int MODE>
__device__ __forceinline__ bool has_neighbor(const DevGraph &g, const VHdr &h, uint32_t x) {
  if (h.d == 0) return false;
  if constexpr (MODE == kCsr) {
    if (neighbor<MODE>(g, h, 0) > x) return false;
    const uint32_t i = last_le(0u, h.d - 1, x, [&](uint32_t k) { return neighbor<MODE>(g, h, k); });
    return neighbor<MODE>(g, h, i) == x;
  } else {
    if (x <= h.base || h.cb == 0) return x == h.base;
    const uint32_t y = x - h.base;
    const uint32_t slots = div_small(h.d - 1, h.T) + 1;
    uint32_t q = 0, last = div_small(slots - 1, h.K);  // sectors, from the vertex's first
    const uint32_t l0 = h.sec / 4, l1 = (h.sec + last) / 4;
    if (g.fences && l1 > l0) {
      // (fence l0 is the line's owner's, never read: the probes are above it)
      const uint32_t l = last_le_wide<3>(l0, l1, y, [&](uint32_t k) { return ldw(g.fences + k); });
      q = l > l0 ? l * 4 - h.sec : 0;
      last = min(last, l * 4 + 3 - h.sec);
    }
    q = last_le_wide<3>(q, last, y, [&](uint32_t k) { return sector_head(g, h, k); });
    const Sec A = load_sector(g.words, h.sec + q);
    const uint32_t c0 = q * h.K, n = min(h.K, slots - c0);
    auto head = [&](uint32_t c) { return sec_field(A, h.off + c * h.cb, h.a); };
    const uint32_t c = last_le(0u, n - 1, y, head);
    const uint32_t at = h.off + c * h.cb, z = y - sec_field(A, at, h.a);  // the offset looked for
    if (z == 0) return true;
    auto offset = [&](uint32_t id) {  // of index id in the slot
      return sec_field(A, at + h.a + (id - 1) * h.b, id ? h.b : 0u);
    };
    return offset(last_le(0u, min(h.T, h.d - (c0 + c) * h.T) - 1, z, offset)) == z;
  }
}

// Fences for the membership search: word l is the head of the first slot in
// 128-byte line l where that line begins inside a vertex of several sectors
// (other words are not written).  A search over a hub's heads took 3.6 reads
// that missed L2, 12 in all; the fences are 1/32 of the slots' size, a hub's
// lie side by side, and what they leave is one line.  Built by the first
// node2vec call on a graph; one warp per vertex.
__global__ void __launch_bounds__(256) build_fences_kernel(DevGraph g, uint32_t *fences) {
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t v = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; v < g.n; v += nwarps) {
    const VHdr h = record_header<kSlots>(load_record(g.recs + v));
    if (h.d < 2) continue;
    const uint32_t last = div_small(div_small(h.d - 1, h.T), h.K);
    for (uint32_t l = h.sec / 4 + 1 + (threadIdx.x & 31); l <= (h.sec + last) / 4; l += 32)
      fences[l] = sector_head(g, h, l * 4 - h.sec);
  }
}

// Resident 256-thread blocks per SM the node2vec kernels are compiled for: the
// walk waits on dependent sector reads, so resident warps matter more than
// registers until those spill.  262,144 walkers x 80, p = 1, q = 0.5, R-MAT s22
// ef32: 1.45 ms at 4 blocks, 1.56 at 5, 1.86 at 6 (now 1.28 at 4, 54
// registers).  The CSR kernel needs no cap (42 registers).
#ifndef GRASS_N2V_MIN_BLOCKS
#define GRASS_N2V_MIN_BLOCKS 4
#endif
#ifndef GRASS_N2V_CSR_MIN_BLOCKS
#define GRASS_N2V_CSR_MIN_BLOCKS 1
#endif

// A lane goes its own way through tries, steps and walkers: a turn of the loop
// is one candidate for every lane, a first try for most, and the lanes that
// search do so together.  (With the tries of a step in a loop of their own, all
// lanes waited for the last one's: 2.43 against 2.14 ms; 1.45 with the fences and
// 1.28 with three probes a round.  41 M of its reads miss L2; at the rate of
// random reads they take 0.9.)
template <int MODE>
__global__ void __launch_bounds__(256, MODE == kCsr ? GRASS_N2V_CSR_MIN_BLOCKS : GRASS_N2V_MIN_BLOCKS) n2v_kernel(DevGraph g, const uint32_t *__restrict__ starts,
                                                  uint64_t W, N2vArgs a,
                                                  uint32_t *__restrict__ paths,
                                                  unsigned long long *edges, unsigned int *err) {
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t_lo = min(a.t_in, a.t_out), t_hi = max(a.t_in, a.t_out);
  uint64_t cnt = 0;
  bool bad = false;
  uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;  // the lane's walker
  uint32_t s = a.L, k = 0;  // its step and try (s == L: take the next walker)
  uint32_t v = INVALID_VERTEX, u = INVALID_VERTEX;
  uint4 rv = make_uint4(0, 0, 0, 0), ru = rv;  // records of v and of the vertex before it
  bool fresh = false;  // v's record is not loaded yet
  bool first = true;
  for (;;) {  // warp-uniform: one candidate for every lane
    while (s == a.L && w < W) {  // (a loop for walks of no steps)
      if (!first) w += nthreads;
      first = false;
      if (w >= W) break;
      const uint32_t s0 = starts[w];
      store_path(paths, a.layout, W, a.L, w, 0, s0);
      v = s0 < g.n ? s0 : INVALID_VERTEX;
      u = INVALID_VERTEX;
      s = k = 0;
      fresh = true;
    }
    const bool live = w < W;
    if (!__any_sync(kFull, live)) break;
    if (live && fresh) {
      rv = walk_record<MODE>(g, v);
      fresh = false;
      if (rv.z == 0) {  // the walk stops
        for (; s < a.L; s++) store_path(paths, a.layout, W, a.L, w, s + 1, INVALID_VERTEX);
      }
    }
    if (live && s < a.L) {
      const uint64_t id = a.w0 + w;
      const u32x4 r = philox4x32_10(a.seed, s, (uint32_t)id, (uint32_t)(id >> 32), TAG_N2V | k);
      const VHdr h = record_header<MODE>(rv);
      const uint32_t x = neighbor<MODE>(g, h, mulhi_u32(r.x, h.d));
      const uint64_t y = r.y;
      // below both thresholds the candidate is taken, at or above both it is
      // not, whether or not it is a neighbor of u: only in between does the
      // membership search run (never when t_in == t_out, i.e. q = 1)
      bool take = s == 0 || k + 1 == a.max_tries;  // (first step: uniform)
      if (!take) {
        if (x == u) take = y < a.t_ret;
        else if (y < t_lo) take = true;
        else if (y < t_hi) take = y < (has_neighbor<MODE>(g, record_header<MODE>(ru), x) ? a.t_in : a.t_out);
      }
      k++;
      if (take) {
        const bool ok = x < g.n;
        bad |= !ok;
        cnt += ok;
        u = v;
        ru = rv;
        v = ok ? x : INVALID_VERTEX;
        store_path(paths, a.layout, W, a.L, w, s + 1, v);
        s++;
        k = 0;
        fresh = true;
      }
    }
  }
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// Independent random 4-byte reads: each thread draws xorshift64 indices into
// buf[0, mask] and keeps 8 loads in flight; the sum goes to *sink so the loads
// are not dropped.  Used to measure the device's random-read ceiling.
__global__ void __launch_bounds__(256) random_read_kernel(const uint32_t *__restrict__ buf,
                                                          uint64_t mask, uint64_t per_thread,
                                                          uint64_t seed,
                                                          unsigned long long *sink) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint64_t x = (seed + 1) * 0x9E3779B97F4A7C15ull ^ (tid + 1) * 0xBF58476D1CE4E5B9ull;
  uint32_t acc = 0;
  for (uint64_t r = 0; r < per_thread; r += 8) {
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      x ^= x << 13;
      x ^= x >> 7;
      x ^= x << 17;
      v[k] = __ldg(buf + (x & mask));
    }
#pragma unroll
    for (int k = 0; k < 8; k++) acc += v[k];
  }
  acc = __reduce_add_sync(0xFFFFFFFFu, acc);
  if ((threadIdx.x & 31) == 0) atomicAdd(sink, (unsigned long long)acc);
}

// Replays a walk (same stream as rw_kernel) and sums, per draw, the
// algorithmic bytes 16 (vertex record) + ceil(slot bits read / 8) + 4
// (path entry) and the 32-byte sectors the reads span (+1 for the record).
// out[0] = bytes, out[1] = sectors, out[2] = draws.  Start entries add 4
// bytes each.
__global__ void __launch_bounds__(256) rw_account_kernel(DevGraph g,
                                                         const uint32_t *__restrict__ starts,
                                                         uint64_t W, uint32_t L, uint64_t seed,
                                                         unsigned long long *out) {
  uint64_t bytes = 0, sect = 0, draws = 0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < W;
       w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = starts[w];
    bytes += 4;
    if (v >= g.n) v = INVALID_VERTEX;
    u32x4 r{0, 0, 0, 0};
    for (uint32_t s = 0; s < L; s++) {
      if ((s & 3) == 0) r = philox4x32_10(seed, s >> 2, (uint32_t)w, (uint32_t)(w >> 32), TAG_RW);
      bytes += 4;
      if (v == INVALID_VERTEX) continue;
      const VHdr h = header<kSlots>(g, v);
      if (h.d == 0) {
        v = INVALID_VERTEX;
        continue;
      }
      const uint32_t i = mulhi_u32(pick(r, s & 3), h.d);
      // the slot's head and, past its first neighbor, one offset; nothing for degree 1
      const uint32_t bits = h.a + (i % h.T ? h.b : 0u);
      bytes += 16 + (bits + 7) / 8;
      sect += 1 + (h.cb ? 1 : 0);
      draws++;
      const uint32_t nv = neighbor<kSlots>(g, h, i);
      v = nv < g.n ? nv : INVALID_VERTEX;
    }
  }
  warp_add_u64(&out[0], bytes);
  warp_add_u64(&out[1], sect);
  warp_add_u64(&out[2], draws);
}

template <int DEPTH>
__global__ void __launch_bounds__(512, GRASS_RW_CSR_MIN_BLOCKS) rw_csr_kernel(DevCsr c, const uint32_t *__restrict__ starts,
                                                     uint64_t W, uint32_t L, uint64_t seed,
                                                     uint64_t w0, int layout,
                                                     uint32_t *__restrict__ paths,
                                                     unsigned long long *edges) {
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  uint64_t cnt = 0;
  for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; base < W;
       base += nthreads * DEPTH) {
    uint32_t v[DEPTH];
    u32x4 r[DEPTH];
#pragma unroll
    for (int k = 0; k < DEPTH; k++) {
      const uint64_t w = base + k * nthreads;
      v[k] = INVALID_VERTEX;
      r[k] = u32x4{0, 0, 0, 0};
      if (w < W) {
        const uint32_t s0 = starts[w];
        store_path(paths, layout, W, L, w, 0, s0);
        v[k] = s0 < c.n ? s0 : INVALID_VERTEX;
      }
    }
    for (uint32_t s = 0; s < L; s++) {
#pragma unroll
      for (int k = 0; k < DEPTH; k++) {
        const uint64_t w = base + k * nthreads;
        if ((s & 3) == 0) {
          const uint64_t id = w0 + w;
          r[k] = philox4x32_10(seed, s >> 2, (uint32_t)id, (uint32_t)(id >> 32), TAG_RW);
        }
        if (v[k] != INVALID_VERTEX) {
          uint64_t b, e;
          csr_row(c.rowptr, v[k], b, e);
          const uint64_t d = e - b;
          if (d == 0) {
            v[k] = INVALID_VERTEX;
          } else {
            v[k] = load_cold_u32(c.cols + b + mulhi_u32(pick(r[k], s & 3), (uint32_t)d));
            cnt++;
          }
        }
        if (w < W) store_path(paths, layout, W, L, w, s + 1, v[k]);
      }
    }
  }
  warp_add_u64(edges, cnt);
}

// ---------------------------------------------------------------------------
// Draws a lane of the standalone k-hop has in flight at once, and the k-hop
// kernels' resident blocks per SM (256 threads each).  Measured on R-MAT s22
// ef32, 65,536 seeds x (25, 10), us: one draw, 4 blocks 232, 5 blocks 253; two
// draws, 4 blocks 249 (they spill), 3 blocks 244; four draws, 2 blocks 240.  The
// CSR's draws need no sector in registers: two.
#ifndef GRASS_KHOP_INFLIGHT
#define GRASS_KHOP_INFLIGHT 1
#endif
#ifndef GRASS_KHOP_CSR_INFLIGHT
#define GRASS_KHOP_CSR_INFLIGHT 2
#endif
#ifndef GRASS_KHOP_MIN_BLOCKS
#define GRASS_KHOP_MIN_BLOCKS 4
#endif

// k-hop.  One warp per seed (khop_seed_warp).

template <int MODE>
__global__ void __launch_bounds__(256, GRASS_KHOP_MIN_BLOCKS) khop_kernel(DevGraph g, const uint32_t *__restrict__ seeds,
                                                   uint64_t S, KhopArgs A,
                                                   unsigned long long *edges, unsigned int *err) {
  __shared__ SmemHdr sh[8];
  SmemHdr &my = sh[threadIdx.x >> 5];
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t cnt = 0;
  bool bad = false;
  for (uint64_t s = warp; s < S; s += nwarps)
    khop_seed_warp<MODE, GRASS_KHOP_INFLIGHT>(g, seeds, A, s, my, cnt, bad);
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// The CSR twin of khop_kernel: the same warp routine and draws, one column
// load per draw.
__global__ void __launch_bounds__(256, GRASS_KHOP_MIN_BLOCKS) khop_csr_kernel(DevCsr c, const uint32_t *__restrict__ seeds,
                                                       uint64_t S, KhopArgs A,
                                                       unsigned long long *edges) {
  __shared__ SmemHdr sh[8];
  SmemHdr &my = sh[threadIdx.x >> 5];
  DevGraph g{};
  g.n = c.n;
  g.mode = GRASS_MODE_CSR_INTERNAL;
  g.rowptr = c.rowptr;
  g.cols = c.cols;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t cnt = 0;
  bool bad = false;
  for (uint64_t s = warp; s < S; s += nwarps)
    khop_seed_warp<kCsr, GRASS_KHOP_CSR_INFLIGHT>(g, seeds, A, s, my, cnt, bad);
  warp_add_u64(edges, cnt);
}

// ---------------------------------------------------------------------------
// Multi random walk.

// Uniform selection, one warp per sample, the walkers' vertices in shared
// memory (SMEM) or in place.
template <int MODE, bool SMEM>
__device__ __forceinline__ void mrw_uniform_samples(const DevGraph &g, uint32_t *roots, uint64_t S,
                                                    uint32_t R, uint32_t T, uint64_t seed,
                                                    uint32_t *src, uint32_t *dst,
                                                    uint32_t *smem, uint64_t &cnt, bool &bad) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t s = warp; s < S; s += nwarps) {
    uint32_t *rt = roots + s * R;
    if constexpr (SMEM) {
      for (uint32_t i = lane; i < R; i += 32) smem[i] = rt[i];
      __syncwarp();
      mrw_uniform_warp<MODE>(g, smem, R, T, seed, s, src, dst, cnt, bad);
      for (uint32_t i = lane; i < R; i += 32) rt[i] = smem[i];
      __syncwarp();
    } else {
      mrw_uniform_warp<MODE>(g, rt, R, T, seed, s, src, dst, cnt, bad);
    }
  }
}

// Resident 256-thread blocks per SM: every lane waits on dependent record and
// sector reads, so resident warps pay (65,536 samples of 80 x 100 on R-MAT s22
// ef32: 246 us at 4 blocks, 251 at 6, 212 at 8, 32 registers; the 7 M reads that miss L2
// take 155 at the rate of random reads).
#ifndef GRASS_MRW_MIN_BLOCKS
#define GRASS_MRW_MIN_BLOCKS 8
#endif

template <int MODE>
__global__ void __launch_bounds__(256, GRASS_MRW_MIN_BLOCKS) mrw_kernel(DevGraph g, uint32_t *__restrict__ roots,
                                                  uint64_t S, uint32_t R, uint32_t T, uint64_t seed,
                                                  uint32_t *__restrict__ src,
                                                  uint32_t *__restrict__ dst,
                                                  unsigned long long *edges, unsigned int *err) {
  extern __shared__ uint32_t walkers[];  // R words a warp
  uint64_t cnt = 0;
  bool bad = false;
  mrw_uniform_samples<MODE, true>(g, roots, S, R, T, seed, src, dst,
                                  walkers + (threadIdx.x >> 5) * R, cnt, bad);
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// The same with more walkers than shared memory holds.
template <int MODE>
__global__ void __launch_bounds__(256) mrw_global_kernel(DevGraph g, uint32_t *roots, uint64_t S,
                                                         uint32_t R, uint32_t T, uint64_t seed,
                                                         uint32_t *__restrict__ src,
                                                         uint32_t *__restrict__ dst,
                                                         unsigned long long *edges,
                                                         unsigned int *err) {
  uint64_t cnt = 0;
  bool bad = false;
  mrw_uniform_samples<MODE, false>(g, roots, S, R, T, seed, src, dst, nullptr, cnt, bad);
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// Degree-proportional selection, G lanes per sample (8, or 32 with more walkers
// than a lane should search).  With rec == nullptr the state (R records, then R
// vertices a sample) lives in shared memory, else (G = 32) the records in rec
// (S R of them) and the vertices in place.
#ifndef GRASS_MRW_DEGREE_MIN_BLOCKS
#define GRASS_MRW_DEGREE_MIN_BLOCKS 4
#endif
template <int MODE, int G, class Sum>
__global__ void __launch_bounds__(256, GRASS_MRW_DEGREE_MIN_BLOCKS)
    mrw_degree_kernel(DevGraph g, uint32_t *roots, uint4 *rec, uint64_t S, uint32_t R, uint32_t T,
                      uint64_t seed, uint32_t *__restrict__ src, uint32_t *__restrict__ dst,
                      unsigned long long *edges, unsigned int *err) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr uint32_t P = 32 / G;  // samples per warp
  const uint32_t gl = threadIdx.x & (G - 1), grp = threadIdx.x / G;
  uint4 *srec = reinterpret_cast<uint4 *>(smem) + (uint64_t)grp * R;
  uint32_t *svtx = reinterpret_cast<uint32_t *>(smem + (uint64_t)(blockDim.x / G) * R * 16) + (uint64_t)grp * R;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t cnt = 0;
  bool bad = false;
  for (uint64_t s0 = warp * P; s0 < S; s0 += nwarps * P) {  // warp-uniform
    const uint64_t s = s0 + (threadIdx.x & 31) / G;
    const bool live = s < S;
    uint32_t *rt = roots + s * R;
    if (G == 32 && rec) {
      mrw_degree_warp<MODE>(g, rt, rec + s * R, R, T, seed, s, src, dst, cnt, bad);
      continue;
    }
    if (live)
      for (uint32_t i = gl; i < R; i += G) svtx[i] = rt[i];
    __syncwarp();
    if constexpr (G == 32)
      mrw_degree_warp<MODE>(g, svtx, srec, R, T, seed, s, src, dst, cnt, bad);
    else
      mrw_degree_group<MODE, G, Sum>(g, live, svtx, srec, R, T, seed, s, src, dst, cnt, bad);
    if (live)
      for (uint32_t i = gl; i < R; i += G) rt[i] = svtx[i];
    __syncwarp();
  }
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

// Multi random walk, one block per sample, walkers in parallel (mrw_cta.cuh);
// scratch holds `stride` bytes per block, reused for its samples.
template <int MODE, int NW>
__global__ void __launch_bounds__(32 * NW) mrw_cta_kernel(DevGraph g, uint32_t *__restrict__ roots,
                                                      uint64_t S, uint32_t R, uint32_t T,
                                                      uint32_t select, uint64_t seed,
                                                      uint32_t *__restrict__ src,
                                                      uint32_t *__restrict__ dst,
                                                      unsigned char *scratch, uint64_t stride,
                                                      unsigned long long *edges,
                                                      unsigned int *err) {
  __shared__ CtaSmem<NW> sm;
  unsigned char *scr = scratch + blockIdx.x * stride;
  uint64_t cnt = 0;
  bool bad = false;
  for (uint64_t s = blockIdx.x; s < S; s += gridDim.x)
    mrw_cta_sample<MODE, NW>(g, roots + s * R, src + s * T, dst + s * T, R, T, select, seed, s,
                             scr, sm, cnt, bad);
  warp_add_u64(edges, cnt);
  if (bad && err) atomicOr(err, 1u);
}

__global__ void starts_kernel(uint64_t n, uint64_t count, uint64_t seed, uint32_t tag,
                              uint32_t *out) {
  const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q * 4 < count; q += nt) {
    const u32x4 r = philox4x32_10(seed, (uint32_t)q, 0, 0, tag);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint64_t i = q * 4 + k;
      if (i < count) out[i] = mulhi_u32(pick(r, k), (uint32_t)n);
    }
  }
}

unsigned grid_warps(uint64_t units, int units_per_block, int device, int per_sm) {
  const uint64_t need = (units + units_per_block - 1) / units_per_block;
  const uint64_t cap = (uint64_t)sm_count(device) * per_sm;
  return (unsigned)std::max<uint64_t>(1, std::min(need, cap));
}

int cur_dev() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

}  // namespace

void launch_uniform_starts(uint64_t n, uint64_t count, uint64_t seed, uint32_t *out,
                           cudaStream_t s, bool mrw_roots) {
  if (!count) return;
  starts_kernel<<<grid_warps((count + 3) / 4, 256, cur_dev(), 8), 256, 0, s>>>(
      n, count, seed, mrw_roots ? TAG_MRW_ROOT : TAG_START, out);
  count_launch();
}

// Launch through cudaLaunchKernelEx so the L2 window is a per-launch
// attribute: the caller's stream keeps its own access policy.
template <class... ExpTypes, class... ActTypes>
static void launch_with_window(void (*kern)(ExpTypes...), unsigned grid, unsigned block,
                               size_t smem, cudaStream_t s, const L2Window &win,
                               ActTypes &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (win.on()) {
    attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
    attr[0].val.accessPolicyWindow.base_ptr = const_cast<void *>(win.base);
    attr[0].val.accessPolicyWindow.num_bytes = win.bytes;
    attr[0].val.accessPolicyWindow.hitRatio = win.hit_ratio;
    attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  cudaLaunchKernelEx(&cfg, kern, std::forward<ActTypes>(args)...);
}

int apply_tuning(int device, const grass_tuning &t, const void *base, size_t bytes,
                 L2Window &win) {
  win = L2Window();
  if (t.l2_fetch_bytes) {
    cudaError_t e = cudaDeviceSetLimit(cudaLimitMaxL2FetchGranularity, t.l2_fetch_bytes);
    if (e != cudaSuccess) return cuda_fail(e, "cudaLimitMaxL2FetchGranularity");
  }
  if (t.l2_persist && base && bytes) {
    int max_persist = 0, max_window = 0;
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, device);
    cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, device);
    if (max_persist > 0 && max_window > 0) {
      const size_t carve = std::min<size_t>((size_t)max_persist, bytes);
      cudaError_t e = cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, carve);
      if (e != cudaSuccess) return cuda_fail(e, "cudaLimitPersistingL2CacheSize");
      size_t got = 0;
      cudaDeviceGetLimit(&got, cudaLimitPersistingL2CacheSize);
      win.base = base;
      win.bytes = std::min<size_t>(bytes, (size_t)max_window);
      win.hit_ratio = (float)std::min(1.0, (double)got / (double)win.bytes);
    }
  }
  return GRASS_OK;
}

// Defaults measured on B200 (R-MAT s22 ef32, 1M walkers x 80, step-major
// paths): the compressed walk is fastest with one walker per thread, the CSR
// walk 0.5% faster with four.  Blocks of 64 threads spread few walkers over more
// SMs and leave a place sooner (us at 64 / 256 threads: 4,096 x 80 on s22 63 /
// 75, on s16 54.7 / 55.1; 1M x 80 2014 / 2032); 512 resident threads a block
// pair (64 registers) beat 1536 (40: 2.09 -> 2.15 ms).  A caller that bounds the
// blocks per SM and not their threads means blocks of 256 (1M x 40 at two of
// them: 1.10 ms, at two of 64 threads 3.16).
grass_tuning resolve_tuning(const grass_tuning &t, int kind) {
  grass_tuning r = t;
  if (!r.rw_depth) r.rw_depth = kind == 2 ? 4 : 1;
  if (!r.rw_threads) r.rw_threads = kind == 2 || r.rw_blocks_per_sm ? 256 : 64;
  return r;  // rw_blocks_per_sm == 0: as many as are resident
}

// Grid for a grid-stride kernel: the requested blocks per SM, capped by
// what the occupancy calculator says is resident, times the SM count, and
// no more blocks than there is work for.
template <class K>
static unsigned resident_grid(K kern, int threads, size_t smem, uint32_t want_per_sm,
                              uint64_t units, uint64_t units_per_block) {
  int per_sm = resident_blocks((const void *)kern, threads, smem);
  if (want_per_sm && (int)want_per_sm < per_sm) per_sm = (int)want_per_sm;
  const uint64_t need = (units + units_per_block - 1) / units_per_block;
  const uint64_t cap = (uint64_t)sm_count(cur_dev()) * per_sm;
  return (unsigned)std::max<uint64_t>(1, std::min(need, cap));
}

template <int DEPTH>
static void rw_launch_depth(const DevGraph &g, const grass_rw_params &p, const uint32_t *starts,
                            uint64_t W, uint32_t *paths, unsigned long long *edges,
                            unsigned int *err, cudaStream_t s, const grass_tuning &t,
                            const L2Window &win, uint64_t w0) {
  auto kern = rw_kernel<kSlots, DEPTH>;
  const size_t smem = p.layout == GRASS_LAYOUT_WALK_MAJOR
                          ? (size_t)t.rw_threads / 32 * kPathStageWords<DEPTH> * 4 : 0;
  static_assert(512 / 32 * kPathStageWords<DEPTH> * 4 <= 48 * 1024, "no opt-in needed");
  // (a lane takes a second walker only where all resident lanes have one)
  const unsigned grid = resident_grid(kern, (int)t.rw_threads, smem, t.rw_blocks_per_sm, W,
                                      t.rw_threads);
  launch_with_window(kern, grid, t.rw_threads, smem, s, win, g, starts, W, p.length, p.seed, w0,
                     (int)p.layout, paths, edges, err);
}

static void rw_dispatch(const DevGraph &g, const grass_rw_params &p, const uint32_t *starts,
                        uint64_t W, uint32_t *paths, unsigned long long *edges,
                        unsigned int *err, cudaStream_t s, const grass_tuning &t,
                        const L2Window &win, uint64_t w0) {
  switch (t.rw_depth) {
    case 1: rw_launch_depth<1>(g, p, starts, W, paths, edges, err, s, t, win, w0); break;
    case 4: rw_launch_depth<4>(g, p, starts, W, paths, edges, err, s, t, win, w0); break;
    default: rw_launch_depth<2>(g, p, starts, W, paths, edges, err, s, t, win, w0);
  }
}

void launch_rw(const DevGraph &g, const grass_rw_params &p, const uint32_t *starts, uint64_t W,
               uint32_t *paths, unsigned long long *edges, unsigned int *err, cudaStream_t s,
               const grass_tuning &tin, const L2Window &win, uint64_t w0) {
  if (!W) return;
  const grass_tuning t = resolve_tuning(tin, g.mode);
  rw_dispatch(g, p, starts, W, paths, edges, err, s, t, win, w0);
  count_launch();
}

uint64_t launch_random_read(const uint32_t *buf, uint64_t n_words, uint64_t reads, uint64_t seed,
                            unsigned long long *sink, cudaStream_t s) {
  const unsigned grid = (unsigned)sm_count(cur_dev()) * 8;
  const uint64_t threads = (uint64_t)grid * 256;
  const uint64_t per_thread = ((reads + threads - 1) / threads + 7) / 8 * 8;
  random_read_kernel<<<grid, 256, 0, s>>>(buf, n_words - 1, per_thread, seed, sink);
  count_launch();
  return per_thread * threads;
}

void launch_rw_account(const DevGraph &g, const grass_rw_params &p, const uint32_t *starts,
                       uint64_t W, unsigned long long *out, cudaStream_t s) {
  if (!W) return;
  const unsigned grid = grid_warps(W, 256, cur_dev(), 8);
  rw_account_kernel<<<grid, 256, 0, s>>>(g, starts, W, p.length, p.seed, out);
  count_launch();
}

void launch_rw_csr(const DevCsr &c, const grass_rw_params &p, const uint32_t *starts,
                   uint64_t W, uint32_t *paths, unsigned long long *edges, cudaStream_t s,
                   const grass_tuning &tin, const L2Window &win, uint64_t w0) {
  if (!W) return;
  const grass_tuning t = resolve_tuning(tin, 2);
  const uint32_t L = p.length;
  const int lay = (int)p.layout;
  const int T = (int)t.rw_threads;
  switch (t.rw_depth) {
    case 1: {
      const unsigned grid = resident_grid(rw_csr_kernel<1>, T, 0, t.rw_blocks_per_sm, W, T);
      launch_with_window(rw_csr_kernel<1>, grid, T, 0, s, win, c, starts, W, L, p.seed, w0, lay,
                         paths, edges);
      break;
    }
    case 4: {
      const unsigned grid = resident_grid(rw_csr_kernel<4>, T, 0, t.rw_blocks_per_sm, W, T * 4);
      launch_with_window(rw_csr_kernel<4>, grid, T, 0, s, win, c, starts, W, L, p.seed, w0, lay,
                         paths, edges);
      break;
    }
    default: {
      const unsigned grid = resident_grid(rw_csr_kernel<2>, T, 0, t.rw_blocks_per_sm, W, T * 2);
      launch_with_window(rw_csr_kernel<2>, grid, T, 0, s, win, c, starts, W, L, p.seed, w0, lay,
                         paths, edges);
    }
  }
  count_launch();
}

static KhopArgs khop_args(const grass_khop_params &p, uint32_t *const *hop_out) {
  KhopArgs A{};
  A.hops = p.hops;
  uint64_t w = 1;
  for (uint32_t h = 0; h < p.hops; h++) {
    A.fan[h] = p.fanouts[h];
    w *= p.fanouts[h];
    A.width[h] = w;
    A.out[h] = hop_out[h];
  }
  A.seed = p.seed;
  return A;
}

void launch_khop(const DevGraph &g, const grass_khop_params &p, const uint32_t *seeds,
                 uint64_t S, uint32_t *const *hop_out, unsigned long long *edges,
                 unsigned int *err, cudaStream_t s) {
  if (!S) return;
  const KhopArgs A = khop_args(p, hop_out);
  const unsigned grid = grid_warps(S, 8, cur_dev(), 8);
  khop_kernel<kSlots><<<grid, 256, 0, s>>>(g, seeds, S, A, edges, err);
  count_launch();
}

uint64_t fence_words(uint64_t n_words) { return n_words / 32 + 1; }

void launch_build_fences(const DevGraph &g, uint32_t *fences, cudaStream_t s) {
  build_fences_kernel<<<grid_warps(g.n, 8, cur_dev(), 8), 256, 0, s>>>(g, fences);
  count_launch();
}

void launch_node2vec(const DevGraph &g, const grass_node2vec_params &p, const uint64_t t[3],
                     const uint32_t *starts, uint64_t W, uint32_t *paths,
                     unsigned long long *edges, unsigned int *err, cudaStream_t s, uint64_t w0) {
  if (!W) return;
  N2vArgs a;
  a.L = p.length;
  a.max_tries = p.max_tries;
  a.layout = (int)p.layout;
  a.seed = p.seed;
  a.w0 = w0;
  a.t_ret = t[0];
  a.t_in = t[1];
  a.t_out = t[2];
  const unsigned grid = grid_warps(W, 256, cur_dev(), 8);
  if (g.mode == GRASS_MODE_CSR_INTERNAL)
    n2v_kernel<kCsr><<<grid, 256, 0, s>>>(g, starts, W, a, paths, edges, err);
  else
    n2v_kernel<kSlots><<<grid, 256, 0, s>>>(g, starts, W, a, paths, edges, err);
  count_launch();
}

void launch_khop_csr(const DevCsr &c, const grass_khop_params &p, const uint32_t *seeds,
                     uint64_t S, uint32_t *const *hop_out, unsigned long long *edges,
                     cudaStream_t s) {
  if (!S) return;
  const KhopArgs A = khop_args(p, hop_out);
  khop_csr_kernel<<<grid_warps(S, 8, cur_dev(), 8), 256, 0, s>>>(c, seeds, S, A, edges);
  count_launch();
}

// Warps per block (a power of two up to 8) for `warps` warps of work, each
// with `bytes` of shared memory: at most 48 KB a block, and no more warps than
// spread the work over the SMs.
static int mrw_block_warps(uint64_t warps, size_t bytes) {
  int w = 8;
  while (w > 1 && (w * bytes > 48 * 1024 || warps < (uint64_t)sm_count(cur_dev()) * w)) w /= 2;
  return w;
}

// Shape of mrw_degree_kernel<.., G, ..> for S samples of R walkers: warps per
// block, bytes of shared memory per warp (0: the state is in global memory), blocks.
struct DegreeShape {
  int w;
  size_t per_warp;
  unsigned grid;
};
template <int G>
static DegreeShape mrw_degree_shape(uint64_t S, uint32_t R) {
  const uint64_t warps = (S + 32 / G - 1) / (32 / G);
  DegreeShape d;
  d.per_warp = (size_t)R * 20 * (32 / G);
  if (d.per_warp > 48 * 1024) d.per_warp = 0;  // too many walkers for shared memory (G = 32)
  d.w = mrw_block_warps(warps, d.per_warp);
  d.grid = grid_warps(warps, d.w, cur_dev(), 64 / d.w);
  return d;
}
// Samples of that shape that are resident at once.
template <int G, class Sum>
static uint64_t mrw_degree_resident(uint64_t S, uint32_t R) {
  const DegreeShape d = mrw_degree_shape<G>(S, R);
  return (uint64_t)sm_count(cur_dev()) * d.w * (32 / G) *
         std::min(64 / d.w, resident_blocks((const void *)mrw_degree_kernel<kSlots, G, Sum>,
                                            d.w * 32, d.per_warp * d.w));
}

template <int G, class Sum>
static int launch_mrw_degree(const DevGraph &g, const grass_mrw_params &p, uint32_t *roots,
                             uint64_t S, uint32_t *src, uint32_t *dst, unsigned long long *edges,
                             unsigned int *err, cudaStream_t s) {
  const DegreeShape d = mrw_degree_shape<G>(S, p.walkers);
  uint4 *rec = nullptr;
  if (!d.per_warp) {
    cudaError_t e =
        scratch_alloc(reinterpret_cast<void **>(&rec), S * (uint64_t)p.walkers * sizeof(uint4), s);
    if (e != cudaSuccess) return cuda_fail(e, "multi-RW scratch");
  }
  mrw_degree_kernel<kSlots, G, Sum><<<d.grid, d.w * 32, d.per_warp * d.w, s>>>(
      g, roots, rec, S, p.walkers, p.steps, p.seed, src, dst, edges, err);
  count_launch();
  if (rec) scratch_free(rec, s);
  return GRASS_OK;
}

int launch_mrw(const DevGraph &g, const grass_mrw_params &p, uint32_t *roots, uint64_t S,
               uint32_t *src, uint32_t *dst, unsigned long long *edges, unsigned int *err,
               uint32_t max_degree, cudaStream_t s) {
  if (!S || !p.steps) return GRASS_OK;
  // Block per sample (walkers in parallel) for continuous-time selection, and
  // for uniform selection where a block ends a long chain sooner than a warp
  // (same output); the rules and their measurements are in launch_rules.h.
  const bool ct = p.select == GRASS_SELECT_DEGREE_CT, wide = ct && p.walkers > kWideWalkers;
  const int threads = mrw_block_threads(S, p.walkers, ct, sm_count(cur_dev()));
  auto cta = wide ? mrw_cta_kernel<kSlots, 32> : mrw_cta_kernel<kSlots, 16>;
  uint64_t resident = 0;
  if (p.select != GRASS_SELECT_DEGREE)
    resident = (uint64_t)sm_count(cur_dev()) * resident_blocks((const void *)cta, threads, 0);
  if (ct || (p.select == GRASS_SELECT_UNIFORM &&
             mrw_uniform_by_blocks(S, p.walkers, p.steps, threads, resident))) {
    const uint64_t stride = mrw_sample_scratch(p.walkers, p.steps, p.select);
    uint64_t grid = std::min<uint64_t>(S, resident);
    unsigned char *scr = nullptr;
    cudaError_t e = scratch_alloc(reinterpret_cast<void **>(&scr), grid * stride, s);
    while (e == cudaErrorMemoryAllocation && grid > 1) {  // a block takes one sample after another
      cudaGetLastError();
      grid /= 2;
      e = scratch_alloc(reinterpret_cast<void **>(&scr), grid * stride, s);
    }
    if (e != cudaSuccess) return cuda_fail(e, "multi-RW scratch");
    cta<<<(unsigned)grid, threads, 0, s>>>(
        g, roots, S, p.walkers, p.steps, p.select, p.seed, src, dst, scr, stride, edges, err);
    count_launch();
    scratch_free(scr, s);
    return GRASS_OK;
  }
  if (p.select == GRASS_SELECT_DEGREE) {
    const bool wide = (uint64_t)p.walkers * max_degree >> 32;  // (sums of 64 bits)
    bool groups = p.walkers <= kSurelyGroups;
    if (!groups && p.walkers <= kGroupWalkers)
      groups = mrw_degree_by_groups(S, p.walkers, p.steps,
                                    wide ? mrw_degree_resident<8, uint64_t>(S, p.walkers)
                                         : mrw_degree_resident<8, uint32_t>(S, p.walkers),
                                    mrw_degree_resident<32, uint64_t>(S, p.walkers));
    if (!groups)
      return launch_mrw_degree<32, uint64_t>(g, p, roots, S, src, dst, edges, err, s);
    if (wide)
      return launch_mrw_degree<8, uint64_t>(g, p, roots, S, src, dst, edges, err, s);
    return launch_mrw_degree<8, uint32_t>(g, p, roots, S, src, dst, edges, err, s);
  }
  const bool fits = p.walkers <= 48 * 1024 / 4;
  const size_t per_warp = fits ? (size_t)p.walkers * 4 : 0;
  const int w = mrw_block_warps(S, per_warp);
  auto kern = fits ? mrw_kernel<kSlots> : mrw_global_kernel<kSlots>;
  kern<<<grid_warps(S, w, cur_dev(), 64 / w), w * 32, per_warp * w, s>>>(
      g, roots, S, p.walkers, p.steps, p.seed, src, dst, edges, err);
  count_launch();
  return GRASS_OK;
}

}  // namespace grass
