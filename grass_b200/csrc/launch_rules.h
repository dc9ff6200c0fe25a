// launch_rules.h -- which multi-RW kernel runs a call and in what shape: host
// arithmetic on sizes and on how many samples are resident at once, without
// anything of CUDA (tests compile it by itself).  Figures: one B200, R-MAT s22 ef32.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace grass {

// A number of threads as a block size: whole warps, between `least` and `most`.
inline int block_size(uint64_t threads, int least, int most) {
  return (int)std::min<uint64_t>(most, std::max<uint64_t>(least, (threads + 31) / 32 * 32));
}

// Continuous-time multi-RW of at most kWideWalkers walkers takes the kernel of
// 116 registers, of more the one of 64 registers and up to 1024 threads (2000
// walkers x 10,000 steps, 1 / 51 samples: 246 / 320 us, with 512 threads 279 /
// 400; with few walkers the registers pay: 80 x 100, 2000 samples 279 us against
// 331).
constexpr uint32_t kWideWalkers = 512;

// Threads of a block that takes one sample of R walkers, of S samples on `sms`
// SMs, in a launch of its own (mrw_cta_kernel).  Continuous time: a thread a
// walker is fastest while every sample has an SM to itself.  With more samples
// blocks of 160 threads pay, three of which are resident where one of 288 to 512
// is.  us with a thread a walker / 160 threads / half a thread a walker and the
// radix sort: 257 walkers x 400 steps, 148 samples 73 / 85 / 145, 300 130 / 92 /
// 153, 8192 3022 / 1613 / 1984; 512 x 400, 148 56 / 89 / 111, 300 119 / 98 / 195,
// 8192 2463 / 1838 / 2851.
inline int mrw_block_threads(uint64_t S, uint32_t R, bool continuous, int sms) {
  if (!continuous) return block_size(R / 2, 128, 512);
  if (R > kWideWalkers) return block_size(R, 128, 1024);
  return block_size(R, 128, S <= (uint64_t)sms ? 512 : 160);
}

// Threads of a block of the batch's block-level kernel, which takes `samples`
// multi-RW samples of up to R walkers (a thread a walker, 64 registers).  Two
// blocks of 512 fit on an SM.  With more samples than that, the blocks are half as
// wide as the walkers and 256 threads at most, and more of them are resident.  us
// in a batch at 512 threads / here, of 256 threads before block-level items had a
// kernel of their own, LE, R-MAT s22 ef32: uniform, 10,000 samples of 20 walkers x 30
// 281 / 84 / 225, 2000 of 80 x 100 71 / 34 / 64, 500 of 2000 x 500 57 / 56 / 92;
// continuous time, the same, 1390 / 473 / 1362, 317 / 143 / 343, 203 / 187 / 361.
// 51 samples of 2000 x 10,000, at 512 / 256: 106 / 169, 406 / 636.
inline int batch_block_threads(uint64_t samples, uint32_t R, int sms) {
  return samples <= 2 * (uint64_t)sms ? block_size(R, 128, 512) : block_size(R / 2, 128, 256);
}

// Rounds of `resident` samples at a time that S samples take.
inline uint64_t sample_rounds(uint64_t S, uint64_t resident) {
  return (S + resident - 1) / std::max<uint64_t>(resident, 1);
}

// Whether S samples of uniform multi-RW (R walkers, T steps) run as blocks of
// `threads` threads, `resident` of them at a time, or as warps: the output is
// the same.  A warp takes 32 steps of a sample a round and needs about T / 10 us
// for as many samples as fit.  A round of blocks takes about 11 us to set up,
// more with many walkers, and then T steps shared by its threads or, with few
// walkers, by the walkers (a step's figures are tenths of a microsecond); it
// also wants a chain long enough for the walkers that share it.  The constants
// are a fit to 3,000 pairs of times, S 1-2000, R 8-5000, T 100-10,000, within
// 0.6 % of the better one on average.  us, block / warp: 80 walkers x 300 steps,
// 148 / 600 samples: 27 / 32, 41 / 34; x 1024, 600 / 2000: 111 / 120, 232 / 144.
// 1000 x 100, 1: 17 / 17; x 500, 148 / 300: 27 / 40, 44 / 48; x 3000, 600 / 2000:
// 181 / 332, 484 / 434.  2000 x 10,000, 600 / 2000: 486 / 988, 1341 / 1343.  8 x
// 2000, 148: 421 / 307.
inline bool mrw_uniform_by_blocks(uint64_t S, uint32_t R, uint32_t T, int threads,
                                  uint64_t resident) {
  if (R < 12 || T < 120.0 + 8000.0 / R) return false;
  const double step = std::max(43.0 / threads, 0.9 - R / 100.0);
  return (double)sample_rounds(S, resident) * (110.0 + R / 30.0 + step * T) <= T;
}

// Whether S samples of degree-proportional multi-RW (R walkers of at most
// kGroupWalkers, T steps) run as groups of eight lanes or as warps, given how many
// of each are resident.  A step of a group costs less with few walkers a lane to
// search, and its samples take four times fewer warps, but fewer of them fit with
// many walkers, and there are fewer loads under way for the first records.  us,
// groups / warps, 100 steps: 80 walkers, 1500 / 8192 samples 106 / 131, 184 / 361;
// 160, 121 / 133, 222 / 365; 192, 128 / 134, 232 / 366; 208 (7104 groups
// resident), 131 / 134, 413 / 369; 256, 141 / 136, 430 / 376.  192 walkers, 12,000
// samples, 5 / 10 / 50 steps: 77 / 50, 98 / 75, 246 / 285.  (A lone sample has its
// warp to itself: 256 walkers x 300, 293 / 313, where 148 take 374 / 320.)  Up to
// kSurelyGroups walkers groups are never slower by more than 2 us, and a launch
// does not ask what is resident.
constexpr uint32_t kGroupWalkers = 256, kSurelyGroups = 128;
inline bool mrw_degree_by_groups(uint64_t S, uint32_t R, uint32_t T, uint64_t groups,
                                 uint64_t warps) {
  return S == 1 || (double)sample_rounds(S, groups) * T * (410 + R) + 0.0025 * (double)S * R <=
                       (double)sample_rounds(S, warps) * T * 600;
}

}  // namespace grass
