// batch.h -- work items of the batched persistent kernel (internal).
#pragma once
#include <vector>

#include "graph.h"
#include "launch_rules.h"
#include "mrw_cta.cuh"
#include "sample_warp.cuh"

namespace grass {

// Device-side job descriptor.
struct BatchJob {
  uint32_t type, count;
  uint64_t seed;
  const uint32_t *in;
  uint32_t *roots, *out0, *out1;
  unsigned char *mscr;  // multi-RW scratch: mstride bytes per sample
  uint64_t mstride;
  unsigned long long *edges;
  uint32_t length, layout, walkers, steps, select;
  uint32_t gen_roots;  // multi-RW: draw the start vertices first (as grass_mrw_roots)
  KhopArgs khop;
};

// One work item: items [begin, end) of job `job` (walkers, seeds or samples).
struct BatchTask {
  uint32_t job, pad;
  uint64_t begin, end;
};

// The work items by kind, in this order: ends of the block-level multi-RW
// samples, the sequential multi-RW samples, the k-hop seeds and the walker
// tiles.  parts: warps per k-hop seed; walkers: the most of a block-level sample.
struct BatchRanges {
  uint32_t cta, mrw, khop, rw, parts, walkers;
};
// Words of the device queue: a counter per kind, zero before a run.
constexpr uint32_t kQueueWords = 4;

// Zero fields of a config take the defaults for this decode mode.
grass_batch_config resolve_batch_config(const grass_batch_config &c, int mode);

// Walk jobs of at most this many walkers are split into one-pass work items.
// Measured in the serving loop (R-MAT s24 ef16, results in device memory):
// p50 at 2 k req/s 0.73 ms against 1.01 ms, p99 at 80 % of peak 3.3 ms
// against 3.65 ms, peak 75 k against 76 k req/s; the 256-job batch within 1 %.
#ifndef GRASS_BATCH_SMALL_RW
#define GRASS_BATCH_SMALL_RW 2048
#endif

// Walkers per work item of a walk job of `count` walkers (resolved config):
// a small job takes one pass per item (32 x depth walkers), so that its
// walkers run side by side instead of in sequential passes of one warp.
inline uint64_t rw_tile(uint64_t count, const grass_batch_config &c) {
  const uint64_t pass = 32ull * c.depth;
  return count <= GRASS_BATCH_SMALL_RW && c.walker_tile > pass ? pass : c.walker_tile;
}

// Multi-RW scratch bytes of a job (count samples of mrw_sample_scratch).
inline uint64_t mrw_job_scratch(const grass_job &j) {
  return j.type == GRASS_JOB_MRW ? (uint64_t)j.count * mrw_sample_scratch(j.walkers, j.steps, j.select)
                                 : 0;
}

// Fills a device job descriptor from a job (mscr: mrw_job_scratch(j) bytes
// for a multi-RW job, else null).
BatchJob make_batch_job(const grass_job &j, unsigned char *mscr);

// Appends the work items of job index `ji`, split per config, to the queues:
// block-level items (multi-RW samples whose walkers move in parallel,
// selections 0 and 2), then warp-level items (sequential multi-RW samples,
// k-hop seed groups, walker tiles).
void split_job(const grass_job &j, uint32_t ji, const grass_batch_config &c,
               std::vector<BatchTask> &cta, std::vector<BatchTask> &mrw,
               std::vector<BatchTask> &khop, std::vector<BatchTask> &rw);

// Walkers of a job's block-level samples (0: it has none).
inline uint32_t block_walkers(const grass_job &j) {
  return j.type == GRASS_JOB_MRW && j.select != GRASS_SELECT_DEGREE ? j.walkers : 0;
}

inline BatchRanges batch_ranges(const std::vector<BatchTask> &cta, const std::vector<BatchTask> &mrw,
                                const std::vector<BatchTask> &khop,
                                const std::vector<BatchTask> &rw, const grass_batch_config &c,
                                uint32_t walkers) {
  BatchRanges r;
  r.cta = (uint32_t)cta.size();
  r.mrw = r.cta + (uint32_t)mrw.size();
  r.khop = r.mrw + (uint32_t)khop.size();
  r.rw = r.khop + (uint32_t)rw.size();
  r.parts = c.warps_per_vertex;
  r.walkers = walkers;
  return r;
}

// Kernels that launch_batch launches for the work items.
inline uint64_t batch_kernels(const BatchRanges &r) { return (r.cta > 0) + (r.rw > r.cta); }

// A stream and events beside a batch's stream, for its block-level items.
struct BatchSide {
  cudaStream_t st = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  cudaError_t create();  // once; a second call does nothing
  void destroy();
};

// Launches the persistent kernels on graph `dg` (compressed or CSR) of device
// `device` over the work items of `ranges`: block-level and warp-level items have
// a kernel each, which run side by side where both kinds are present (side,
// created here, joins stream s again; null: one after the other on s).  d_queue:
// kQueueWords zeroed words.  Corrupt payloads set bit 0 of *d_err.
int launch_batch(const DevGraph &dg, int device, const BatchJob *d_jobs, const BatchTask *d_tasks,
                 const BatchRanges &ranges, unsigned int *d_queue, unsigned long long *d_total,
                 unsigned int *d_err, cudaStream_t s, BatchSide *side,
                 const grass_batch_config &c);

}  // namespace grass
