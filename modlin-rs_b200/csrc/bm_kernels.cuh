// Linear-complexity launchers (host side).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "field.cuh"

namespace modlin {

// One sequence of a batch: field constants inline so a launch mixes primes.
struct BmJob {
  uint64_t p, mu_lo, mu_hi, safe_batch;
  const uint64_t* s;  // device pointer, n residues
  int64_t n;
  int64_t slot;       // output index
};

// 64-bit words of the two residual arrays of an n-residue sequence as byte
// planes, `limbs` each.
MODLIN_HD constexpr int64_t bm_words(int limbs, int64_t n) { return 2 * limbs * ((n + 160 + 15) / 16 * 16) / 8; }
int64_t bm_smem_words(uint64_t p, int64_t n);  // for p's limbs
int64_t bm_workspace_words(int64_t n);         // for any p

// threads: a multiple of 32 from 128 to 512. gws: workspace of
// bm_smem_words(p, n) words when that is more than smem_words.
cudaError_t launch_bm_block(const BmJob& job, uint64_t* gws, int64_t smem_words, int threads, int64_t* d_out,
                            cudaStream_t st);
cudaError_t launch_bm_batch(const BmJob* d_jobs, int64_t count, unsigned long long* d_next, uint64_t* gws,
                            int64_t gws_words, int64_t smem_words, int blocks, int threads, int64_t* d_out,
                            cudaStream_t st);
int bm_batch_max_blocks_per_sm(int threads, int64_t smem_words);
// Loads the module of bm_block_kernel on the current device now (a lazily
// loaded module would otherwise be loaded, and its memory allocated, at the
// first launch).
cudaError_t bm_block_prepare();

// One long sequence on up to `ctas` CTAs (cooperative launch; at least two),
// or on one thread-block cluster of 16 CTAs (8 where 16 cannot be launched).
// ws: bm_long_bytes(p, n) bytes. spin: cycles a CTA waits, beyond what a sweep of
// the sequence may take, before it gives up and sets the error word (at
// bm_long_err_offset() in ws); skip_cta (>= 0, tests only): that CTA does not
// signal, and spin is all that a CTA waits.
size_t bm_long_bytes(uint64_t p, int64_t n);
int bm_long_err_offset();
cudaError_t launch_bm_long(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, int num_sms, void* ws,
                           long long spin, int skip_cta, int64_t* d_out, cudaStream_t st);
cudaError_t launch_bm_cluster(const FieldParams& fp, const uint64_t* s, int64_t n, void* ws, long long spin,
                              int64_t* d_out, cudaStream_t st);
constexpr int64_t kBmClusterMaxN = 409600;

}  // namespace modlin
