// Batched rank launcher (host side).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

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
  int cluster;     // CTAs per team
  int64_t shared;  // jobs (the first ones) that teams take
  int64_t max_n;
};
// Launch shape for jobs sorted longest first; blocks 0 on an error.
RankBatchShape rank_batch_shape(const std::vector<RankJob>& jobs, int num_sms);
// Relative running time of a job.
double rank_batch_cost(uint64_t p, int64_t n);
constexpr int kRankBatchCounters = 2;  // job counters at d_next
cudaError_t launch_rank_batch(const RankJob* d_jobs, int64_t count, unsigned long long* d_next,
                              const RankBatchShape& shape, int64_t* d_out, cudaStream_t st);
// The same for a shape with teams, and the teams of 2, 4 and 8 CTAs that the
// current device holds at a time.
struct RankTeams {
  int n[3];
};
cudaError_t launch_rank_team(const RankJob* d_jobs, int64_t count, unsigned long long* d_next,
                             const RankBatchShape& shape, int64_t* d_out, cudaStream_t st);
RankTeams rank_team_resident(int num_sms);

}  // namespace modlin
