// device_common.cuh -- device-side view of a compressed graph and the GT/LE
// decoders used by every kernel.
//
// Stream words: the .graph file's bytes in big-endian order per 32-bit word
// (GT/src/grass.cu:1147-1159), stored byte-swapped in HBM so that a word read
// is the next 32 stream bits MSB-first.  Two zero guard words follow the last
// word, so a 64-bit window read never leaves the allocation.
#pragma once
#include <stdint.h>

#include "rng.h"

namespace grass {

constexpr uint32_t INVALID_VERTEX = 0xFFFFFFFFu;

// A graph as the samplers see it: compressed (words and records: the slot
// layout below, the same for a GT and an LE file) or an uncompressed CSR
// (mode 2, GRASS_MODE_CSR_INTERNAL: rowptr and cols), so that one sampler
// template serves both sides of a comparison.  mode names the file format;
// load-time kernels are templated on it, samplers on kSlots or kCsr.
struct DevGraph {
  const uint32_t *__restrict__ words;
  const uint4 *__restrict__ recs;        // n vertex records (sampling, decode)
  const uint64_t *__restrict__ offsets;  // n + 1 bit offsets (load time only)
  uint32_t n;
  int32_t mode;
  const uint64_t *__restrict__ rowptr;   // mode 2
  const uint32_t *__restrict__ cols;     // mode 2
  const uint32_t *__restrict__ fences;   // node2vec: a head per 128-byte line (or null)
};
constexpr int GRASS_MODE_CSR_INTERNAL = 2;
// Sampler template argument MODE.
constexpr int kSlots = 1;  // slot layout
constexpr int kCsr = 2;    // uncompressed CSR

struct DevCsr {
  const uint64_t *__restrict__ rowptr;
  const uint32_t *__restrict__ cols;
  uint32_t n;
};

__device__ __forceinline__ uint32_t ldw(const uint32_t *p) { return __ldg(p); }

// A field of width w in [1, 32] at bit offset off
// (the reference's get_32b(off) >> (32 - w), GT/src/bcg.cuh:64-70, 90-95).
__device__ __forceinline__ uint32_t read_field(const uint32_t *w, uint64_t off, int width) {
  const uint32_t *q = w + (off >> 5);
  uint32_t win = __funnelshift_l(ldw(q + 1), ldw(q), (uint32_t)off & 31u);
  return width ? win >> (32 - width) : 0u;
}

// Sequential MSB-first reader: the top `nb` bits of `buf` are unread stream
// bits, the rest are zero; one 32-bit word is pulled when nb <= 32.
struct BitCur {
  const uint32_t *p;
  uint64_t buf;
  int nb;
  __device__ __forceinline__ void init(const uint32_t *w, uint64_t off) {
    const uint32_t *q = w + (off >> 5);
    uint32_t s = (uint32_t)off & 31u;
    buf = (((uint64_t)ldw(q) << 32) | ldw(q + 1)) << s;
    nb = 64 - (int)s;
    p = q + 2;
  }
  __device__ __forceinline__ void fill() {
    if (nb <= 32) {
      buf |= (uint64_t)ldw(p) << (32 - nb);
      p++;
      nb += 32;
    }
  }
  // width in [1, 32]
  __device__ __forceinline__ uint32_t get(int width) {
    fill();
    uint32_t v = (uint32_t)(buf >> (64 - width));
    buf <<= width;
    nb -= width;
    return v;
  }
  // Elias-gamma of x+1, returns x (GT/src/bcg.cuh:82-107): zeros z, then
  // z+1 bits.  z is clamped to 31 as the reference's 32-bit window implies;
  // headers are validated once at load, so sampling kernels see z <= 31.
  __device__ __forceinline__ uint32_t gamma() {
    fill();
    int z = min(__clzll(buf), 31);
    buf <<= z;
    nb -= z;
    fill();
    uint32_t v = (uint32_t)(buf >> (63 - z));
    buf <<= (z + 1);
    nb -= z + 1;
    return v - 1u;
  }
  __device__ __forceinline__ uint64_t pos(const uint32_t *w) const {
    return (uint64_t)(p - w) * 32u - (uint64_t)nb;
  }
};

// One 32-byte sector of the slots as eight words, each the next 32 stream bits
// MSB first.  It is read by one 256-bit load: random reads are limited by the
// number of requests (43 G/s on a 1 GB footprint whether a request brings 4
// or 32 bytes), so a sector read as two 16-byte halves costs twice.
struct Sec {
  uint32_t w[8];
};

// L2 eviction priorities.  Every draw reads one entry of a small hot table
// (vertex records, or the CSR's row pointers: tens of MB, i.e. L2-sized)
// and one or two random sectors of a large cold array (the stream, or CSR
// columns: far larger than L2).  Without hints the cold reads evict the hot
// table between its uses and every draw pays a DRAM access for it.
//   hot table  -> evict_last
//   cold reads -> GRASS_COLD_POLICY (0: normal, 1: evict_first)
//   path/frontier stores -> GRASS_ST_POLICY (0: normal, 1: evict_first)
#ifndef GRASS_HOT_POLICY
#define GRASS_HOT_POLICY 1
#endif
#ifndef GRASS_COLD_POLICY
#define GRASS_COLD_POLICY 0
#endif
#ifndef GRASS_ST_POLICY
#define GRASS_ST_POLICY 1
#endif

__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// The loads below are inline PTX, marked volatile: a non-volatile asm
// statement counts as a pure function of its inputs, so the compiler may
// execute it speculatively -- hoisted above the branch that guards its
// address (a record load for an invalid vertex id, say) -- and fault.
__device__ __forceinline__ uint4 load_record(const uint4 *p) {
  uint4 r;
#if GRASS_HOT_POLICY
  asm volatile("ld.global.nc.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(p), "l"(policy_evict_last()));
#else
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(p));
#endif
  return r;
}

// A 4-byte cold read (CSR column).
__device__ __forceinline__ uint32_t load_cold_u32(const uint32_t *p) {
#if GRASS_COLD_POLICY
  uint32_t v;
  asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(policy_evict_first()));
  return v;
#else
  return __ldg(p);
#endif
}

// Store of an output entry that is not read again by the kernel.
__device__ __forceinline__ void store_out_u32(uint32_t *p, uint32_t v) {
#if GRASS_ST_POLICY
  asm volatile("st.global.L2::cache_hint.u32 [%0], %1, %2;" ::"l"(p), "r"(v),
               "l"(policy_evict_first())
               : "memory");
#else
  *p = v;
#endif
}

__device__ __forceinline__ Sec load_sector(const uint32_t *words, uint32_t sector) {
  const uint32_t *p = words + (uint64_t)sector * 8;
  Sec r;
#if GRASS_COLD_POLICY
  asm volatile("ld.global.nc.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
#else
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
#endif
      : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]),
        "=r"(r.w[6]), "=r"(r.w[7])
      : "l"(p));
  return r;
}

// x >> n for n in [0, 32] (32 gives 0).
__device__ __forceinline__ uint32_t shr_clamp(uint32_t x, uint32_t n) {
  return __funnelshift_rc(x, 0u, n);
}

// The `width` (0..32) bits at bit `off` of a sector, the field inside it.
// Registers cannot be indexed, so the field's two words are picked by a tree
// of selects on the word index's bits (5 + 3 + 2), then one funnel shift.
__device__ __forceinline__ uint32_t sec_field(const Sec &A, uint32_t off, uint32_t width) {
  const bool k4 = off & 128u, k2 = off & 64u, k1 = off & 32u;
  const uint32_t t0 = k4 ? A.w[4] : A.w[0], t1 = k4 ? A.w[5] : A.w[1], t2 = k4 ? A.w[6] : A.w[2],
                 t3 = k4 ? A.w[7] : A.w[3], t4 = k4 ? 0u : A.w[4];
  const uint32_t u0 = k2 ? t2 : t0, u1 = k2 ? t3 : t1, u2 = k2 ? t4 : t2;
  const uint32_t hi = k1 ? u1 : u0, lo = k1 ? u2 : u1;
  return shr_clamp(__funnelshift_l(lo, hi, off), 32u - width);  // (shifts by off mod 32)
}

__device__ __forceinline__ uint32_t isqrt_u32(uint32_t x) {
  uint32_t r = (uint32_t)__fsqrt_rn((float)x);
  if ((uint64_t)r * r > x) r--;
  if ((uint64_t)(r + 1) * (r + 1) <= x) r++;
  return r;
}

// ---- the files' own formats (load time only) ----
// Decoded stream header of a vertex.  a = GT head_bit / LE rock_bit, b = GT
// body_bit / LE sea_bit; bn/bl/om = GT block_num/block_len/om_num or LE
// chunk_num/chunk_len/om_num (decoder convention, LE/src/bcg.cuh:141-146);
// fp = first_pos, or for LE degree 1 the single neighbor.
struct DiskHdr {
  uint64_t P;  // bit offset of the payload
  uint32_t v, d, bn, bl, om, fp;
  int a, b;
};

// GT header: BCGVertex ctor, GT/src/bcg.cuh:109-136 (isqrt instead of
// sqrt((float)d); equal for every degree the compressor can emit below 2^24).
__device__ __forceinline__ DiskHdr gt_header(const DevGraph &g, uint32_t v) {
  DiskHdr h;
  BitCur c;
  c.init(g.words, g.offsets[v]);
  h.v = v;
  h.d = c.gamma();
  h.a = (int)c.gamma();
  h.b = (int)c.gamma();
  h.fp = c.gamma();
  h.P = c.pos(g.words);
  uint32_t s = isqrt_u32(h.d);
  if (s * s == h.d) {
    h.bn = h.bl = s;
    h.om = 0;
  } else {
    h.bn = s + 1;
    h.bl = h.d / h.bn;
    h.om = h.d - h.bn * h.bl;
  }
  return h;
}

// GT block geometry: block blk starts at
// P + blk (a + (bl - 1) b) + min(blk, om) b (GT/src/bcg.cuh:153-163).
__device__ __forceinline__ uint64_t gt_disk_block_pos(const DiskHdr &h, uint32_t blk) {
  return h.P + (uint64_t)blk * ((uint64_t)h.a + (uint64_t)(h.bl - 1) * h.b) +
         (uint64_t)min(blk, h.om) * h.b;
}

// Geometry of an LE vertex of degree d >= 2: chunk_num, chunk_len, om
// (decoder convention, LE/src/bcg.cuh:141-146).
__device__ __forceinline__ void le_disk_geometry(uint32_t d, uint32_t &bn, uint32_t &bl,
                                                 uint32_t &om) {
  const uint32_t D = d - 1;
  const uint32_t s = isqrt_u32(D);
  const uint32_t o = D - s * s;
  bn = s + (o > s ? 1u : 0u);
  bl = D / bn;
  om = D - bn * bl;
}

// LE header: BCGVertex ctor, LE/src/bcg.cuh:130-152.
__device__ __forceinline__ DiskHdr le_header(const DevGraph &g, uint32_t v) {
  DiskHdr h;
  BitCur c;
  c.init(g.words, g.offsets[v]);
  h.v = v;
  h.d = c.gamma();
  h.a = h.b = 0;
  h.bn = h.bl = h.om = h.fp = 0;
  if (h.d == 0) {
    h.P = 0;
    return h;
  }
  uint32_t r = c.gamma();
  if (h.d == 1) {
    h.fp = r;  // degree 1: the field holds the neighbor itself
    h.P = 0;
    return h;
  }
  h.a = (int)r;
  h.b = (int)c.gamma();
  h.fp = c.gamma();
  h.P = c.pos(g.words);
  le_disk_geometry(h.d, h.bn, h.bl, h.om);
  return h;
}

// Stream headers (gamma decode at offsets[v]); used at load time only.
template <int MODE>
__device__ __forceinline__ DiskHdr stream_header(const DevGraph &g, uint32_t v) {
  if constexpr (MODE == 0) return gt_header(g, v);
  else return le_header(g, v);
}

// A stream header as a 16-byte load-time record: x = payload bit offset P, low
// 32 bits; y = P bits 32..47 | a << 16 (6 bits) | b << 22 (6 bits); z = degree;
// w = first_pos, or for LE degree 1 the single neighbor.
__device__ __forceinline__ uint4 pack_record(const DiskHdr &h) {
  uint4 r;
  r.x = (uint32_t)h.P;
  r.y = ((uint32_t)(h.P >> 32) & 0xFFFFu) | ((uint32_t)h.a & 63u) << 16 |
        ((uint32_t)h.b & 63u) << 22;
  r.z = h.d;
  r.w = h.fp;
  return r;
}

// Header of a GT vertex from its load-time record.
__device__ __forceinline__ DiskHdr gt_disk_record_header(const uint4 r, uint32_t v) {
  DiskHdr h;
  h.v = v;
  h.P = (uint64_t)r.x | ((uint64_t)(r.y & 0xFFFFu) << 32);
  h.a = (int)((r.y >> 16) & 63u);
  h.b = (int)((r.y >> 22) & 63u);
  h.d = r.z;
  h.fp = r.w;
  const uint32_t s = isqrt_u32(h.d);
  if (s * s == h.d) {
    h.bn = h.bl = s;
    h.om = 0;
  } else {
    h.bn = s + 1;
    h.bl = h.d / h.bn;
    h.om = h.d - h.bn * h.bl;
  }
  return h;
}

// Header of an LE vertex from its load-time record.
__device__ __forceinline__ DiskHdr le_disk_record_header(const uint4 r, uint32_t v) {
  DiskHdr h;
  h.v = v;
  h.P = (uint64_t)r.x | ((uint64_t)(r.y & 0xFFFFu) << 32);
  h.a = (int)((r.y >> 16) & 63u);
  h.b = (int)((r.y >> 22) & 63u);
  h.d = r.z;
  h.fp = r.w;
  h.bn = h.bl = h.om = 0;
  if (h.d > 1) le_disk_geometry(h.d, h.bn, h.bl, h.om);
  return h;
}

// ---- sector slots: the device layout of both formats ----
// On disk a vertex is ~sqrt(d) blocks (GT) or chunks (LE) of ~sqrt(d)
// neighbors, so a random draw in a hub touches several 32-byte sectors: GT
// adds up to sqrt(d) gaps (GT/src/bcg.cuh:153-168), LE reads its rock pair
// and its sea from two places (LE/src/bcg.cuh:195-261).  At load every
// vertex of either format is re-chunked for the device: chunk c holds
// neighbors cT .. cT + T - 1 in a slot
//   [head n_cT - n_0 (a bits)][offsets n_i - n_cT (b bits) of i = cT+1 ..]
// of cb = a + (T - 1) b bits that never crosses a sector: it starts at
// P + (c / K) 256 + (c % K) cb, with K <= 63 slots per sector.  A vertex whose
// slots fit in one sector is packed without alignment (and lies inside one
// sector), a larger one starts on a sector.  All differences are mod 2^32, so
// any list is kept bit for bit.
//
// So a draw reads its record and one sector, and of that two fields whatever
// its index in the slot: neighbor = n_0 + head + offset.  (The slots held the
// files' own codes before: GT's gaps, which a draw has to add up, and LE's
// left rock, right rock and signed sea, interpolated with a division.  That
// took 286 instructions a draw of the walk.  R-MAT s22 ef32, 1M x 80: 2.07 ms
// against LE 2.23 ms; a small walk, all latency, 54 against 103 us; node2vec
// 2.43 against 3.48 ms.)  T in 1..32 is chosen per vertex
// for the fewest bits, about 3 on average: R-MAT s21 ef32 takes 19.9 bits an
// edge, where LE's code on the same slots took 21.3 and GT's 18.5; all T equal
// to 1 would take 21.8, powers of two 20.8.
//
// Record (16 B): x = P low 32 bits; y = P bits 32..39 | a << 8 | b << 14 |
// T << 20 | K << 26; z = degree; w = n_0.  A vertex of degree 1 has a = b = 0:
// its neighbor is in the record and it has no slot.
struct VHdr {
  uint32_t sec, off;  // kSlots: P's sector and bit in it
  uint64_t P;         // kCsr: first entry of the row
  uint32_t d, base;   // degree, n_0
  uint32_t a, b, T, K, cb;
};

__device__ __forceinline__ uint4 pack_slot_record(uint64_t P, uint32_t a, uint32_t b, uint32_t T,
                                                  uint32_t K, uint32_t d, uint32_t n0) {
  return make_uint4((uint32_t)P,
                    ((uint32_t)(P >> 32) & 0xFFu) | (a & 63u) << 8 | (b & 63u) << 14 |
                        (T & 63u) << 20 | (K & 63u) << 26,
                    d, n0);
}

template <int MODE>
__device__ __forceinline__ VHdr record_header(const uint4 r) {
  VHdr h{};
  h.d = r.z;
  if constexpr (MODE == kCsr) {
    h.P = (uint64_t)r.x | ((uint64_t)(r.y & 0xFFFFu) << 32);
  } else {
    h.sec = __funnelshift_r(r.x, r.y, 8);
    h.off = r.x & 255u;
    h.a = (r.y >> 8) & 63u;
    h.b = (r.y >> 14) & 63u;
    h.T = (r.y >> 20) & 63u;
    h.K = r.y >> 26;
    h.cb = h.a + (h.T - 1u) * h.b;
    h.base = r.w;
  }
  return h;
}

// Exact x / d for x < 2^31 (degrees are below it) and the layout's small
// divisors 1 <= d < 64 (chunk length T, slots per sector K): with 2^(s-1) < d
// <= 2^s and m = ceil(2^(31+s) / d) < 2^32, x m / 2^(31+s) = x / d + x e /
// (d 2^(31+s)) with e < d <= 2^s, and x e / 2^(31+s) < 1 keeps the quotient.
// One 8-byte table entry (through L1) and a 32-bit multiply-high of 2x.
struct DivMagic64 {
  uint2 m[64];  // {m, s}
};
__host__ __device__ constexpr DivMagic64 make_div_magic64() {
  DivMagic64 t{};
  for (uint32_t d = 1; d < 64; d++) {
    uint32_t s = 0;
    while ((1u << s) < d) s++;
    t.m[d].x = (uint32_t)(((1ull << (31 + s)) + d - 1) / d);
    t.m[d].y = s;
  }
  return t;
}
__device__ const DivMagic64 kDivMagic64 = make_div_magic64();
__device__ __forceinline__ uint32_t div_small(uint32_t x, uint32_t d) {
  const uint2 m = __ldg(&kDivMagic64.m[d]);
  return __umulhi(x + x, m.x) >> m.y;
}

// Where a draw's slot is: sector, bit in it, index in the slot.
struct DrawAt {
  uint32_t sec, off, id;
};
__device__ __forceinline__ DrawAt slot_at(const VHdr &h, uint32_t c) {
  const uint32_t q = div_small(c, h.K);
  return DrawAt{h.sec + q, h.off + (c - q * h.K) * h.cb, 0u};
}
__device__ __forceinline__ DrawAt draw_at(const VHdr &h, uint32_t i) {
  const uint32_t c = div_small(i, h.T);
  DrawAt at = slot_at(h, c);
  at.id = i - c * h.T;
  return at;
}
// The drawn neighbor from its slot's sector.
__device__ __forceinline__ uint32_t draw_value(const Sec &A, const DrawAt &at, const VHdr &h) {
  return h.base + sec_field(A, at.off, h.a) +
         sec_field(A, at.off + h.a + (at.id - 1u) * h.b, at.id ? h.b : 0u);
}

// [rowptr[v], rowptr[v+1]) of a CSR with one 32-byte load (two when the pair
// straddles a sector, v % 4 == 3).  rowptr must be allocated in whole
// sectors with one spare sector (see grass_csr allocation).
__device__ __forceinline__ void csr_row(const uint64_t *rowptr, uint32_t v, uint64_t &b,
                                        uint64_t &e) {
  const uint64_t *p = rowptr + (v & ~3u);
  uint64_t a0, a1, a2, a3;
#if GRASS_HOT_POLICY
  asm volatile("ld.global.nc.L2::evict_last.v4.b64 {%0,%1,%2,%3}, [%4];"
      : "=l"(a0), "=l"(a1), "=l"(a2), "=l"(a3)
      : "l"(p));
#else
  asm volatile("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];"
      : "=l"(a0), "=l"(a1), "=l"(a2), "=l"(a3)
      : "l"(p));
#endif
  const uint32_t k = v & 3u;
  b = k == 0 ? a0 : k == 1 ? a1 : k == 2 ? a2 : a3;
  e = k == 0 ? a1 : k == 1 ? a2 : k == 2 ? a3 : __ldg(p + 4);
}

// The 16-byte record of vertex v; for a CSR (mode 2) one is made from its
// row pointers: {start low 32 bits, start bits 32..47, degree, 0}.
template <int MODE>
__device__ __forceinline__ uint4 graph_record(const DevGraph &g, uint32_t v) {
  if constexpr (MODE == kCsr) {
    uint64_t b, e;
    csr_row(g.rowptr, v, b, e);
    return make_uint4((uint32_t)b, (uint32_t)(b >> 32) & 0xFFFFu, (uint32_t)(e - b), 0u);
  } else {
    return load_record(g.recs + v);
  }
}

template <int MODE>
__device__ __forceinline__ VHdr header(const DevGraph &g, uint32_t v) {
  return record_header<MODE>(graph_record<MODE>(g, v));
}

__device__ __forceinline__ uint32_t record_degree(const DevGraph &g, uint32_t v) {
  return __ldg(&g.recs[v].z);
}

template <int MODE>
__device__ __forceinline__ uint32_t neighbor(const DevGraph &g, const VHdr &h, uint32_t i) {
  if constexpr (MODE == kCsr) {
    return load_cold_u32(g.cols + h.P + i);
  } else {
    if (h.cb == 0) return h.base;  // degree 1
    const DrawAt at = draw_at(h, i);
    return draw_value(load_sector(g.words, at.sec), at, h);
  }
}

// End bit of a vertex's on-disk payload given its stream header (load-time
// validation).  For the files the reference compressor writes this is offsets[v+1]
// (GT/chunk_compress/compressor.hpp:297-349, LE/chunk_compress/compressor.hpp:329-390).
template <int MODE>
__device__ __forceinline__ uint64_t payload_end(const DevGraph &g, const DiskHdr &h) {
  if constexpr (MODE == 0) {
    return gt_disk_block_pos(h, h.bn);
  } else {
    if (h.d <= 1) return 0;  // caller checks via the header cursor instead
    return h.P + (uint64_t)(h.bn + 1) * h.a + (uint64_t)(h.d - h.bn - 1) * (h.b + 1);
  }
}

// Warp-aggregated add of a per-thread counter into a device u64.
__device__ __forceinline__ void warp_add_u64(unsigned long long *dst, uint64_t v) {
  if (!dst) return;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, (unsigned long long)v);
}

}  // namespace grass
