// Batched rank with teams: the longest matrices of a batch are each shared by
// the CTAs of a thread-block cluster, which then take the other matrices one
// by one. For batches whose longest matrix would be their end (the rule is
// rank_batch_shape's).
//
// A team's CTAs each invert the step's block (the same work, no exchange) and
// take every size-th tile of 64 rows of the panel and of the rest; one cluster
// barrier a step orders their writes before the next step's reads. A panel
// without a block step is eliminated by the first CTA alone, its update of the
// rest is again the team's. The control flow is the same in all CTAs of a team:
// they compute what decides it from the same data, which no CTA writes before
// a cluster barrier, or get it from the first. 1016 x 1016 over 2^61 - 1: 11.55
// ms on one CTA, 2.83 on eight.
//
// The steps are those of rank_batch.cu. That kernel stays for batches without
// teams: it is up to 10 % faster there for p < 2^32 (148 of side 512 mod 65521:
// 0.78 ms, 0.84 here).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <climits>
#include <map>
#include <mutex>

#include "launch.cuh"
#include "rank_batch_dev.cuh"

namespace modlin {

namespace cg = cooperative_groups;

namespace {

constexpr int kT = 512;
constexpr int kMaxCluster = 8;  // portable cluster size

// The CTAs of a cluster that work on one matrix: how many (1: no exchange at
// all) and which one this is.
struct Team {
  int size, rank;
};

struct TeamSmem : BatchSmem {
  // Written by the cluster's CTAs: whether something nonzero is left (by
  // parity of the exchange and CTA), and the panel path's pivots.
  int nz[2][kMaxCluster];
  int panel_pivots;
  Team team;
};

// The CTA's shared memory: TeamSmem, the left operand's second buffer, the row
// order.
extern __shared__ __align__(16) unsigned char rb_smem[];
__device__ __forceinline__ TeamSmem& batch_smem() { return *reinterpret_cast<TeamSmem*>(rb_smem); }
__device__ __forceinline__ uint8_t* second_buffer() { return rb_smem + sizeof(TeamSmem); }
__device__ __forceinline__ int* row_order() { return reinterpret_cast<int*>(second_buffer() + kRegion); }
struct TeamCta {
  static constexpr int kT = 512;
  static __device__ __forceinline__ BatchSmem& smem() { return batch_smem(); }
  static __device__ __forceinline__ uint8_t* a2() { return second_buffer(); }
  static __device__ __forceinline__ int* perm() { return row_order(); }
};
using Map = TileMap<kT>;

// Whether any CTA of the team has something nonzero left.
__device__ __forceinline__ bool team_any(TeamSmem& S, int c0, bool any) {
  // Two buffers: the next step's writes come before every CTA has read these
  // (other paths to an exchange have cluster barriers of their own).
  const int parity = (c0 / kP) & 1;
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < S.team.size) cl.map_shared_rank(&S, threadIdx.x)->nz[parity][S.team.rank] = any;
  cl.sync();
  for (int q = 0; q < S.team.size; ++q) any |= S.nz[parity][q] != 0;
  return any;
}

// One block step at (r0, c0); false when P is not invertible (nothing has
// changed but the order of the 64 rows). any: something right of and below
// the block is nonzero afterwards.
// Bound: 8 x 64 x 64 limb-product instructions per tile and 2^61 - 1 (8192 of
// an SM's cycles), the epilogue and the conversions for fewer limbs.
// A team's CTAs each invert P (the same work, no exchange) and take every
// size-th tile of 64 rows: H over their rows of X, then their rows of C. One
// cluster barrier a step orders their writes before the next step's reads.
template <class F, int LIMBS, bool kTeam>
__device__ __noinline__ bool block_step(const F& f, uint64_t* __restrict__ m, const int n, int r0, int c0, bool& any) {
  TeamSmem& S = batch_smem();
  uint8_t* const a2 = second_buffer();
  int* const perm = row_order();
  const int first = kTeam ? kP * S.team.rank : 0;  // of this CTA's row tiles, after the block
  const int stride = kTeam ? kP * S.team.size : kP;
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
  const int rb = r0 + kP + first, cb = c0 + kP;  // this CTA's first row tile
  // This warp's tiles: rows 16 rg .. +16, kTiles groups of 8 columns from cg0.
  constexpr int kTiles = Map::kTiles;
  const int rg = warp & 3, cg0 = (warp >> 2) * kTiles;
  const int g = lane >> 2, t2 = 2 * (lane & 3);
  constexpr int kN = Map::kN;
  // The next tile's rows are loaded during this one's products where the
  // registers allow; with two buffers one barrier a tile is enough.
  constexpr bool kEarly = LIMBS <= 4;
  uint8_t* const bufs[2] = {S.a, a2};
  uint32_t acc[2 * LIMBS - 1][4];
  uint64_t lv[kN][4];
  if (cb < n && rb < n && kEarly) load_rows<kT>(m, n, perm, c0, rb, lv);
  for (int rt = rb, k = 0; rt < n && cb < n; rt += stride, k ^= 1) {  // H over X
    if (!kEarly) load_rows<kT>(m, n, perm, c0, rt, lv);
    if (rt == rb) __syncthreads();  // the last product has read the buffer (or P^-1)
    put_rows<LIMBS, kT>(bufs[k], lv);
    __syncthreads();
    if (kEarly && rt + stride < n) load_rows<kT>(m, n, perm, c0, rt + stride, lv);
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
  const bool nz = rb < n && cb < n &&
                  update_rest<F, LIMBS, TeamCta>(f, m, n, r0, kP, rb, stride, c0, cb);
  any = __syncthreads_or(nz);
  if constexpr (kTeam) any = team_any(S, c0, any);
  return true;
}

template <class F, int LIMBS, bool kTeam>
__device__ __noinline__ int rank_one(const F& f, uint64_t* __restrict__ m, const int n) {
  TeamSmem& S = batch_smem();
  int* const perm = row_order();
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += kT) perm[i] = i;
  __syncthreads();
  int r0 = 0;
  for (int c0 = 0; c0 < n && r0 < n; c0 += kP) {
    const int W = min(kP, n - c0);
    const int tries = block_tries(f.modulus(), n - r0);
    if (W == kP && n - r0 >= kP && tries > 0) {
      // A block without a pivot is tried again with the next 64 rows.
      bool any = false, step = false;
      for (int t = 1;; ++t) {
        step = block_step<F, LIMBS, kTeam>(f, m, n, r0, c0, any);
        if (step || t == tries || n - r0 < (t + 1) * kP) break;
        // The rows of the failed block are written by the next attempt's step.
        if constexpr (kTeam) cg::this_cluster().sync();
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
    int pb = 0;
    // The panel path is the team's first CTA's, which may write once no other
    // reads the block it failed on.
    const bool mine = !kTeam || S.team.rank == 0;
    if constexpr (kTeam) cg::this_cluster().sync();
    const int jend = c0 + W;
    if (mine) {
      pb = eliminate_panel<F, LIMBS, TeamCta>(f, m, n, r0, c0, W);
      if (pb > 0 && jend < n && r0 + pb < n) panel_rows<F, TeamCta>(f, m, n, r0, pb, c0);
    }
    __syncthreads();
    if constexpr (kTeam) {
      // The pivots and the row order for the others.
      cg::cluster_group cl = cg::this_cluster();
      if (mine && tid < S.team.size) cl.map_shared_rank(&S, tid)->panel_pivots = pb;
      cl.sync();
      if (!mine) {
        const int* src = cl.map_shared_rank(perm, 0);
        for (int i = tid; i < n; i += kT) perm[i] = src[i];
      }
      pb = S.panel_pivots;
      cl.sync();
    }
    // The trailing rows, as in a block step.
    if (pb > 0) {
      bool nz = false;
      if (jend < n) {
        const int rb = r0 + pb + (kTeam ? kP * S.team.rank : 0);
        if (rb < n)
          nz = update_rest<F, LIMBS, TeamCta>(f, m, n, r0, pb, rb, kTeam ? kP * S.team.size : kP, c0,
                                         jend);
        nz = __syncthreads_or(nz);
        if constexpr (kTeam) nz = team_any(S, c0, nz);
      }
      r0 += pb;
      if (!nz) break;
    }
  }
  return r0;
}

template <bool kTeam>
__device__ __forceinline__ int rank_any(const RankJob& J) {
  const FieldParams fp{J.p, J.mu_lo, J.mu_hi, J.safe_batch};
  const int n = (int)J.n;
  if (J.p == kM61) return rank_one<FpM61, 8, kTeam>(FpM61(fp), J.m, n);
  if (J.p < (1ULL << 32)) {
    const FpSmall f(fp);
    return J.p <= (1ULL << 8)    ? rank_one<FpSmall, 1, kTeam>(f, J.m, n)
           : J.p <= (1ULL << 16) ? rank_one<FpSmall, 2, kTeam>(f, J.m, n)
                                 : rank_one<FpSmall, 4, kTeam>(f, J.m, n);
  }
  return rank_one<FpBarrett, 8, kTeam>(FpBarrett(fp), J.m, n);
}

// The first `shared` jobs (the longest) go to the clusters; then each CTA takes
// the others one by one, from a second counter.
__global__ void __launch_bounds__(kT, 1)
    rank_team_kernel(const RankJob* __restrict__ jobs, int64_t count, int64_t shared, unsigned long long* next,
                      int64_t* out) {
  TeamSmem& S = batch_smem();
  const Team& team = S.team;
  if (threadIdx.x == 0) {
    S.team.size = (int)cg::this_cluster().num_blocks();
    S.team.rank = (int)cg::this_cluster().block_rank();
  }
  // Every CTA of the cluster has started before the first write to another's
  // shared memory, the job's number below.
  cg::this_cluster().sync();
  for (;;) {
    long long q;
    if (team.size > 1) {
      cg::cluster_group cl = cg::this_cluster();
      if (team.rank == 0 && threadIdx.x == 0) {
        const long long t = (long long)atomicAdd(next, 1ULL);
        for (int c = 0; c < team.size; ++c) cl.map_shared_rank(&S, c)->job = t;
      }
      cl.sync();
      q = S.job;
      cl.sync();  // the next job's number, and the next matrix, come after
      if (q >= shared) {
        // No CTA touches another's shared memory from here on.
        __syncthreads();
        if (threadIdx.x == 0) S.team = Team{1, 0};
        __syncthreads();
        continue;
      }
    } else {
      if (threadIdx.x == 0) S.job = shared + (long long)atomicAdd(next + 1, 1ULL);
      __syncthreads();
      q = S.job;
      __syncthreads();
      if (q >= count) break;
    }
    const RankJob J = jobs[q];
    int r;
    if (team.size > 1)
      r = rank_any<true>(J);
    else
      r = rank_any<false>(J);
    if (threadIdx.x == 0 && team.rank == 0) out[J.slot] = r;
    __syncthreads();
  }
}

}  // namespace

static size_t team_smem_bytes(int64_t max_n) { return sizeof(TeamSmem) + kRegion + (size_t)max_n * sizeof(int); }

static cudaError_t team_attr() {
  static PerDevice once;
  return allow_smem(once, rank_team_kernel, team_smem_bytes(kRankBatchMaxN));
}

static cudaLaunchConfig_t team_config(int size, int blocks, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(512);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Teams of 2, 4 and 8 CTAs that the current device holds at a time (asked once
// per device).
RankTeams rank_team_resident(int num_sms) {
  static std::mutex mu;
  static std::map<int, RankTeams> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || team_attr() != cudaSuccess) {
    cudaGetLastError();
    return RankTeams{};
  }
  std::lock_guard<std::mutex> g(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  RankTeams t{};
  for (int k = 0; k < 3; ++k) {
    cudaLaunchAttribute attr[1];
    const int size = 2 << k;
    const cudaLaunchConfig_t cfg =
        team_config(size, num_sms / size * size, team_smem_bytes(kRankBatchMaxN), nullptr, attr);
    if (cudaOccupancyMaxActiveClusters(&t.n[k], rank_team_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      t.n[k] = 0;
    }
  }
  return known[dev] = t;
}

cudaError_t launch_rank_team(const RankJob* d_jobs, int64_t count, unsigned long long* d_next,
                             const RankBatchShape& B, int64_t* d_out, cudaStream_t st) {
  cudaError_t e = team_attr();
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(d_next, 0, kRankBatchCounters * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = team_config(B.cluster, B.blocks, team_smem_bytes(B.max_n), st, attr);
  return cudaLaunchKernelEx(&cfg, rank_team_kernel, d_jobs, count, B.shared, d_next, d_out);
}

}  // namespace modlin
