// Batched rank: thousands of matrices of uneven sides and primes in one
// persistent launch (the CLI's `reps` loop, src/main.rs:82, with every job
// in flight at once).
//
// One CTA eliminates one matrix at a time, pulling jobs (largest first) from a
// device counter. The row order is a logical permutation in shared memory
// instead of physical swaps (src/fp.rs:158-162). Per 64-column panel:
//  * Block step, when the 64 x 64 block P of the next 64 rows is invertible:
//    its rows and columns are the panel's pivots, and the rest becomes the
//    Schur complement: H = -X P^-1 for the panel X below P (written over X),
//    then C += H U tile by tile. P^-1 by inv64, the products as 64 x 64 x 64
//    limb products on the tensor cores (mma_limbs.cuh).
//  * Otherwise (dependent columns, the last ragged panel, p = 2) the reference's
//    panel (src/fp.rs:125-200) and the update of the rest as in a block step
//    (rank_batch_dev.cuh).
// When an update leaves nothing nonzero, the rank is what has been counted.
// Every residue is exact, so the rank is the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <functional>
#include <queue>
#include <vector>

#include "launch.cuh"
#include "rank_batch_dev.cuh"

namespace modlin {

namespace {

// One block step at (r0, c0); false when P is not invertible (nothing has
// changed but the order of the 64 rows). any: something right of and below
// the block is nonzero afterwards.
// Bound: 8 x 64 x 64 limb-product instructions per tile and 2^61 - 1 (8192 of
// an SM's cycles), the epilogue and the conversions for fewer limbs.
template <class F, int LIMBS, int kT>
__device__ __forceinline__ bool block_step_body(const F& f, uint64_t* __restrict__ m, const int n, int* perm,
                                                BatchSmem& S, uint8_t* a2, int r0, int c0, bool& any) {
  const LimbRed<F, LIMBS> red(f);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t p = f.modulus();
  uint64_t* M = reinterpret_cast<uint64_t*>(S.a);
  InvScratch<LIMBS>& I = *reinterpret_cast<InvScratch<LIMBS>*>(S.b);
  for (int q = tid; q < kP * kP; q += kT) M[(q >> 6) * kInvLd + (q & 63)] = m[(int64_t)perm[r0 + (q >> 6)] * n + c0 + (q & 63)];
  __syncthreads();
  if (!inv64<F, LIMBS, kT>(f, red, M, I)) return false;
  uint64_t fac[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) fac[u] = I.fac[u];
  const int moved = tid < kP ? perm[r0 + I.order[tid]] : 0;
  __syncthreads();
  if (tid < kP) perm[r0 + tid] = moved;
  // Right operand: -P^-1, plane row = column of P^-1.
  for (int q = tid; q < kP * 16; q += kT) {
    const int i = q & 63, k4 = 4 * (q >> 6);
    const uint64_t fk = k4 < 32 ? (k4 < 16 ? fac[0] : fac[1]) : (k4 < 48 ? fac[2] : fac[3]);
    uint64_t v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = f.mul(M[(k4 + u) * kInvLd + i], fk);
      v[u] = v[u] ? p - v[u] : 0;
    }
    mml::put_planes4<LIMBS>(S.b + i * kStride + k4, kPlane, v);
  }
  const int rb = r0 + kP, cb = c0 + kP;
  // This warp's tiles: rows 16 rg .. +16, kTiles groups of 8 columns from cg0.
  constexpr int kTiles = 32 / (kT / 32), kRound = kT / 16;
  const int rg = warp & 3, cg0 = (warp >> 2) * kTiles;
  const int g = lane >> 2, t2 = 2 * (lane & 3);
  // Left operand: rows rt .. rt + 63 of the panel, through registers.
  constexpr int kN = kP / kRound;
  const auto load_rows = [&](int rt, uint64_t (&v)[kN][4]) {
#pragma unroll
    for (int w = 0; w < kN; ++w) {
      const int i = (tid >> 4) + kRound * w, k4 = 4 * (tid & 15);
      const uint64_t* src = rt + i < n ? m + (int64_t)perm[rt + i] * n + c0 + k4 : nullptr;
#pragma unroll
      for (int u = 0; u < 4; ++u) v[w][u] = src ? src[u] : 0;
    }
  };
  const auto put_rows = [&](uint8_t* dst, const uint64_t (&v)[kN][4]) {
#pragma unroll
    for (int w = 0; w < kN; ++w)
      mml::put_planes4<LIMBS>(dst + ((tid >> 4) + kRound * w) * kStride + 4 * (tid & 15), kPlane, v[w]);
  };
  // The next tile's rows are loaded during this one's products where the
  // registers allow; with two buffers one barrier a tile is enough.
  constexpr bool kTwo = kT == 512, kEarly = LIMBS <= 4;
  uint8_t* const bufs[2] = {S.a, kTwo ? a2 : S.a};
  uint32_t acc[2 * LIMBS - 1][4];
  uint64_t lv[kN][4];
  if (cb < n && rb < n && kEarly) load_rows(rb, lv);
  for (int rt = rb, k = 0; rt < n && cb < n; rt += kP, k ^= 1) {  // H over X
    if (!kEarly) load_rows(rt, lv);
    if (!kTwo || rt == rb) __syncthreads();  // the last product has read the buffer (or P^-1)
    put_rows(bufs[k], lv);
    __syncthreads();
    if (kEarly && rt + kP < n) load_rows(rt + kP, lv);
    const int ra = rt + 16 * rg + g, rz = ra + 8;
    uint64_t* pa = ra < n ? m + (int64_t)perm[ra] * n + c0 : nullptr;
    uint64_t* pz = rz < n ? m + (int64_t)perm[rz] * n + c0 : nullptr;
#pragma unroll 1
    for (int q = 0; q < kTiles; ++q) {
      block_tile<LIMBS>(acc, bufs[k], S.b, rg, cg0 + q);
      const int c = 8 * (cg0 + q) + t2;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint64_t* dst = e < 2 ? pa : pz;
        const uint64_t v = red.residue(acc, e);
        if (dst) dst[c + (e & 1)] = v;
      }
    }
  }
  // Trailing update by strips of kCols column tiles whose right operands fill
  // region b: the left operand's load and the barriers are shared by them.
  constexpr int kCols = LIMBS == 8 || !kTwo ? 1 : LIMBS == 4 ? 2 : 4;
  bool nz = false;
  for (int ct = cb; ct < n; ct += kP * kCols) {
    __syncthreads();
    constexpr int kRows4 = kT / 64;
#pragma unroll 1
    for (int s = 0; s < kCols; ++s) {
      uint64_t uv[kN][4];
      const int col = ct + kP * s + (tid & 63);
#pragma unroll
      for (int w = 0; w < kN; ++w)  // U: plane row = column
#pragma unroll
        for (int u = 0; u < 4; ++u)
          uv[w][u] = col < n ? m[(int64_t)perm[r0 + 4 * ((tid >> 6) + kRows4 * w) + u] * n + col] : 0;
#pragma unroll
      for (int w = 0; w < kN; ++w)
        mml::put_planes4<LIMBS>(S.b + s * LIMBS * kPlane + (tid & 63) * kStride + 4 * ((tid >> 6) + kRows4 * w),
                                kPlane, uv[w]);
    }
    if (kEarly) load_rows(rb, lv);
    for (int rt = rb, k = 0; rt < n; rt += kP, k ^= 1) {
      const int ra = rt + 16 * rg + g, rz = ra + 8;
      uint64_t* pa = ra < n ? m + (int64_t)perm[ra] * n : nullptr;
      uint64_t* pz = rz < n ? m + (int64_t)perm[rz] * n : nullptr;
      // C of this warp's tiles is loaded before the left operand where
      // registers allow, else before each tile's products (which cover it).
      constexpr bool kAhead = LIMBS <= 4;
      constexpr int kAll = kTiles * kCols;
      uint64_t cv[kAhead ? kAll : 1][4];
      const auto column = [&](int q) { return ct + kP * (q / kTiles) + 8 * (cg0 + q % kTiles) + t2; };
      const auto load_c = [&](int q, uint64_t (&x)[4]) {
        const int c = column(q);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint64_t* src = e < 2 ? pa : pz;
          x[e] = src && c + (e & 1) < n ? src[c + (e & 1)] : 0;
        }
      };
      if (kAhead) {
#pragma unroll
        for (int q = 0; q < kAll; ++q) load_c(q, cv[q]);
      }
      if (!kEarly) load_rows(rt, lv);
      if (!kTwo && rt > rb) __syncthreads();
      put_rows(bufs[k], lv);
      __syncthreads();
      if (kEarly && rt + kP < n) load_rows(rt + kP, lv);
#pragma unroll(kAhead ? kAll : 1)
      for (int q = 0; q < kAll; ++q) {
        const int c = column(q);
        uint64_t(&x)[4] = cv[kAhead ? q : 0];
        if (!kAhead) load_c(q, x);
        block_tile<LIMBS>(acc, bufs[k], S.b + q / kTiles * LIMBS * kPlane, rg, cg0 + q % kTiles);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint64_t* dst = e < 2 ? pa : pz;
          const uint64_t v = red.plus(x[e], acc, e);
          if (dst && c + (e & 1) < n) {
            dst[c + (e & 1)] = v;
            nz |= v != 0;
          }
        }
      }
    }
  }
  any = __syncthreads_or(nz);
  return true;
}

// As a function of its own its registers are the products' (148 matrices of side
// 512 mod 65521: 795 -> 770 us); only four limbs on 512 threads are faster
// within rank_one (979 us, 1027 on their own).
template <class F, int LIMBS, int kT>
__device__ __noinline__ bool block_step_call(const F& f, uint64_t* __restrict__ m, const int n, int* perm,
                                             BatchSmem& S, uint8_t* a2, int r0, int c0, bool& any) {
  return block_step_body<F, LIMBS, kT>(f, m, n, perm, S, a2, r0, c0, any);
}
template <class F, int LIMBS, int kT>
__device__ __forceinline__ bool block_step(const F& f, uint64_t* __restrict__ m, const int n, int* perm, BatchSmem& S,
                                           uint8_t* a2, int r0, int c0, bool& any) {
  if constexpr (LIMBS == 4 && kT == 512)
    return block_step_body<F, LIMBS, kT>(f, m, n, perm, S, a2, r0, c0, any);
  else
    return block_step_call<F, LIMBS, kT>(f, m, n, perm, S, a2, r0, c0, any);
}

// The CTA's shared memory: BatchSmem, the left operand's second buffer (one CTA
// an SM), the row order.
extern __shared__ __align__(16) unsigned char rb_smem[];
template <int NT>
struct OneCta {
  static constexpr int kT = NT;
  static __device__ __forceinline__ BatchSmem& smem() { return *reinterpret_cast<BatchSmem*>(rb_smem); }
  static __device__ __forceinline__ uint8_t* a2() { return rb_smem + sizeof(BatchSmem); }
  static __device__ __forceinline__ int* perm() { return reinterpret_cast<int*>(a2() + (NT == 512 ? kRegion : 0)); }
};

template <class F, int LIMBS, int kT>
__device__ __noinline__ int rank_one(const F& f, uint64_t* __restrict__ m, const int n, int* perm, BatchSmem& S,
                                     uint8_t* a2) {
  const int tid = threadIdx.x;
  const uint64_t p = f.modulus();
  for (int i = tid; i < n; i += kT) perm[i] = i;
  __syncthreads();
  int r0 = 0;
  for (int c0 = 0; c0 < n && r0 < n; c0 += kP) {
    const int W = min(kP, n - c0);
    const int tries = block_tries(p, n - r0);
    if (W == kP && n - r0 >= kP && tries > 0) {
      // A block without a pivot is tried again with the next 64 rows.
      bool any = false, step = false;
      for (int t = 1;; ++t) {
        step = block_step<F, LIMBS, kT>(f, m, n, perm, S, a2, r0, c0, any);
        if (step || t == tries || n - r0 < (t + 1) * kP) break;
        if (tid < kP) {
          const int o = perm[r0 + tid];
          perm[r0 + tid] = perm[r0 + t * kP + tid];
          perm[r0 + t * kP + tid] = o;
        }
        __syncthreads();
      }
      if (step) {
        r0 += kP;
        if (!any) break;
        continue;
      }
      __syncthreads();
    }
    const int pb = eliminate_panel<F, LIMBS, OneCta<kT>>(f, m, n, r0, c0, W);
    if (pb == 0) continue;
    const int jend = c0 + W;
    bool nz = false;
    if (jend < n && r0 + pb < n) {
      panel_rows<F, OneCta<kT>>(f, m, n, r0, pb, c0);
      nz = update_rest<F, LIMBS, OneCta<kT>>(f, m, n, r0, pb, r0 + pb, kP, c0, jend);
    }
    r0 += pb;
    if (!__syncthreads_or(nz)) break;
  }
  return r0;
}

// NT = 256: two CTAs an SM; 512: one.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
    rank_batch_kernel(const RankJob* __restrict__ jobs, int64_t count, unsigned long long* next, int64_t* out) {
  BatchSmem& S = OneCta<NT>::smem();
  uint8_t* a2 = OneCta<NT>::a2();
  int* perm = OneCta<NT>::perm();
  for (;;) {
    if (threadIdx.x == 0) S.job = (long long)atomicAdd(next, 1ULL);
    __syncthreads();
    const long long q = S.job;
    __syncthreads();
    if (q >= count) break;
    const RankJob J = jobs[q];
    const FieldParams fp{J.p, J.mu_lo, J.mu_hi, J.safe_batch};
    int r;
    if (J.p == kM61) {
      r = rank_one<FpM61, 8, NT>(FpM61(fp), J.m, (int)J.n, perm, S, a2);
    } else if (J.p < (1ULL << 32)) {
      const FpSmall f(fp);
      r = J.p <= (1ULL << 8)    ? rank_one<FpSmall, 1, NT>(f, J.m, (int)J.n, perm, S, a2)
          : J.p <= (1ULL << 16) ? rank_one<FpSmall, 2, NT>(f, J.m, (int)J.n, perm, S, a2)
                                : rank_one<FpSmall, 4, NT>(f, J.m, (int)J.n, perm, S, a2);
    } else {
      const FpBarrett f(fp);
      r = rank_one<FpBarrett, 8, NT>(f, J.m, (int)J.n, perm, S, a2);
    }
    if (threadIdx.x == 0) out[J.slot] = r;
    __syncthreads();
  }
}

}  // namespace

static size_t rank_batch_smem_bytes(int threads, int64_t max_n) {
  return sizeof(BatchSmem) + (threads == 512 ? kRegion : 0) + (size_t)max_n * sizeof(int);
}

// The kernels' dynamic shared memory cap is set once per device to what the largest side
// needs, so launches of any batch (graph-captured ones included) need no
// attribute call.
static cudaError_t rank_batch_attr() {
  static PerDevice narrow, wide;
  const cudaError_t e = allow_smem(narrow, rank_batch_kernel<256>, rank_batch_smem_bytes(256, kRankBatchMaxN));
  return e != cudaSuccess ? e : allow_smem(wide, rank_batch_kernel<512>, rank_batch_smem_bytes(512, kRankBatchMaxN));
}

// Threads per CTA: 512 when every matrix has an SM to itself, or the largest
// are long enough to set the end of the batch.
static int batch_threads(int64_t count, int64_t max_n, int num_sms) {
  return count <= num_sms || max_n >= kRankBatchWideN ? 512 : 256;
}

// Running time of a job on a team of `size`, relative to one CTA: the block
// inverses are not shared. Their part measured 0.22 and 0.53 at sides 1024 and
// 512 of 16 bits, 0.17 and 0.44 of 31, 0.12 and 0.32 over 2^61 - 1.
static double team_time(const RankJob& j, int size) {
  const double k = j.p < (1ULL << 16) ? 240 : j.p < (1ULL << 32) ? 200 : 150;
  const double fixed = std::min(1.0, k / (double)j.n);
  return fixed + (1 - fixed) / size;
}

// About the end of a batch (jobs longest first, costs `cost`) whose first
// `shared` jobs go to `teams` teams of `size` CTAs and the others, `rest` in
// all, to the CTAs as they become free. Above `best`: a lower bound of it.
static double batch_end(const std::vector<RankJob>& jobs, const std::vector<double>& cost, size_t shared, int size,
                        int teams, double rest, double best) {
  double sum = 0;
  for (size_t i = 0; i < shared; ++i) sum += cost[i] * team_time(jobs[i], size);
  const double area = (sum * size + rest) / (teams * size);
  if (area >= best) return area;
  std::priority_queue<double, std::vector<double>, std::greater<double>> t(std::greater<double>(),
                                                                           std::vector<double>(teams, 0.0));
  double last = area;
  for (size_t i = 0; i < shared; ++i) {
    const double e = t.top() + cost[i] * team_time(jobs[i], size);
    t.pop();
    t.push(e);
    last = std::max(last, e);
  }
  if (shared < cost.size()) last = std::max(last, t.top() + cost[shared]);
  return last;
}

RankBatchShape rank_batch_shape(const std::vector<RankJob>& jobs, int num_sms) {
  RankBatchShape B{};
  const int64_t count = (int64_t)jobs.size();
  if (count == 0 || rank_batch_attr() != cudaSuccess) return B;
  B.max_n = 1;
  double total = 0, longest = 0;
  for (const RankJob& j : jobs) {
    B.max_n = std::max(B.max_n, j.n);
    const double c = rank_batch_cost(j.p, j.n);
    total += c;
    longest = std::max(longest, c);
  }
  B.threads = batch_threads(count, B.max_n, num_sms);
  B.cluster = 1;
  const size_t smem = rank_batch_smem_bytes(B.threads, B.max_n);
  int nb = 0;
  if (B.threads == 512)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rank_batch_kernel<512>, 512, smem);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rank_batch_kernel<256>, 256, smem);
  B.blocks = (int)std::min<int64_t>(count, (int64_t)nb * num_sms);
  // Teams when the longest job is more than an SM's share of the batch (it
  // would be the batch's end): of the candidates, the one with the earliest
  // end, when that is 15 % before the end without. 512 matrices of sides 64 to
  // 1024 over four primes: 12.9 ms without, 9.4 with; 40 of side 1024 over
  // 2^61 - 1: 11.0 and 6.3; 100 of them stay without. Sides below 4 tiles gain
  // nothing.
  const double share = total / num_sms;
  if (B.threads != 512 || nb < 1 || longest <= share) return B;
  std::vector<double> cost(count);
  for (int64_t i = 0; i < count; ++i) cost[i] = rank_batch_cost(jobs[i].p, jobs[i].n);
  const RankTeams resident = rank_team_resident(num_sms);
  const int* teams = resident.n;
  double best = 0.85 * longest;
  for (int k = 0; k < 3; ++k) {
    if (teams[k] < 1) continue;
    int64_t shared = 0;
    double rest = total;
    for (const double over : {2.0, 1.5, 1.0, 0.75, 0.5}) {
      const int64_t before = shared;
      for (; shared < count && cost[shared] > over * share && jobs[shared].n >= 4 * kP; ++shared) rest -= cost[shared];
      if (shared == before) continue;
      const double end = batch_end(jobs, cost, (size_t)shared, 2 << k, teams[k], rest, best);
      if (end < best) {
        best = end;
        B.cluster = 2 << k;
        B.shared = shared;
        B.blocks = teams[k] * B.cluster;
      }
    }
  }
  return B;
}

cudaError_t launch_rank_batch(const RankJob* d_jobs, int64_t count, unsigned long long* d_next,
                              const RankBatchShape& B, int64_t* d_out, cudaStream_t st) {
  if (B.shared) return launch_rank_team(d_jobs, count, d_next, B, d_out, st);
  const size_t smem = rank_batch_smem_bytes(B.threads, B.max_n);
  cudaError_t e = rank_batch_attr();
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(d_next, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  if (B.threads == 512)
    rank_batch_kernel<512><<<B.blocks, 512, smem, st>>>(d_jobs, count, d_next, d_out);
  else
    rank_batch_kernel<256><<<B.blocks, 256, smem, st>>>(d_jobs, count, d_next, d_out);
  return cudaGetLastError();
}

// Modular multiply-adds of a limb class relative to one-limb primes, roughly:
// the batch takes its longest jobs first.
double rank_batch_cost(uint64_t p, int64_t n) {
  const double w = p < (1ULL << 16) ? 1.0 : p < (1ULL << 32) ? 1.45 : p == kM61 ? 2.65 : 5.0;
  return w * (double)n * n * (n + 200);
}

}  // namespace modlin
