// Batched rank launcher (host side).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace modlin {

// One matrix of a batch: n x n row-major residues at device pointer m
// (clobbered), field constants inline so one launch mixes primes.
struct RankJob {
  uint64_t p, mu_lo, mu_hi, safe_batch;
  uint64_t* m;
  int64_t n;
  int64_t slot;  // output index
};

// Largest side the batched kernel takes (its row permutation lives in shared
// memory); larger matrices go through the single-matrix engine.
constexpr int64_t kRankBatchMaxN = 8192;
constexpr int64_t kRankBatchWideN = 384;

struct RankBatchShape {
  int threads, blocks;
};
// Launch shape for `count` jobs of sides up to max_n; blocks 0 on an error.
RankBatchShape rank_batch_shape(int64_t count, int64_t max_n, int num_sms);
// Relative running time of a job.
double rank_batch_cost(uint64_t p, int64_t n);
cudaError_t launch_rank_batch(const RankJob* d_jobs, int64_t count, unsigned long long* d_next, int64_t max_n,
                              const RankBatchShape& shape, int64_t* d_out, cudaStream_t st);

}  // namespace modlin
