// Panel kernels and the plain trailing update of the blocked GPU rank.
// See rank_plain.cuh for the algorithm and its correspondence to the
// reference's src/fp.rs:125-255.
#include <cuda_runtime.h>

#include "block_inv.cuh"
#include "launch.cuh"
#include "rank_plain.cuh"
#include "rank_kernels.cuh"
#include "tc_ptx.cuh"

namespace modlin {

// ---------------------------------------------------------------------------
// window_kernel — one CTA, kWindowThreads threads.
// Candidates: round 0 -> rows [r0, r0 + min(64, n - r0)); later rounds ->
// ps->cand[0 .. min(ps->ncand, 64)). Their panel columns [col, col + W) are
// eliminated in shared memory with first-nonzero pivoting in candidate order
// (src/fp.rs:150-157), fraction-free, while recording for each candidate
// alpha and its coefficients g against this round's new pivots, so that a
// pivot row k satisfies  U_k = alpha_k * row_k - sum_{k2<k} G[k][k2] * U_k2.
// ---------------------------------------------------------------------------
// Issue-bound: 64 x 64 entries, two products and one reduction each, for every
// pivot (ElimField::comb; 64 pivots over 2^61 - 1: 117 us, 127 with two reduced
// products per entry).
template <class F>
__global__ void __launch_bounds__(kWindowThreads) window_kernel(F f, const uint64_t* __restrict__ m, int64_t ld,
                                                                 int32_t n, int32_t r0, int32_t col, int32_t W,
                                                                 int32_t round, PanelState* ps, uint64_t* Upanel,
                                                                 uint64_t* G, const uint64_t* Lbuf,
                                                                 uint8_t* is_pivot) {
  using W64 = typename ElimField<F>::W;
  const ElimField<F> ef(f);
  extern __shared__ __align__(16) uint64_t smem_w[];
  uint64_t(*A)[kPanel] = reinterpret_cast<uint64_t(*)[kPanel]>(smem_w);                  // [64][64]
  uint64_t(*Gc)[kPanel] = reinterpret_cast<uint64_t(*)[kPanel]>(smem_w + kWindow * kPanel);  // [64][64]
  __shared__ uint64_t alph[kWindow];
  __shared__ int32_t rowidx[kWindow], ispiv[kWindow], pivcand[kPanel], pivc[kPanel];
  __shared__ uint32_t ballots[2][2];
  __shared__ int32_t sh_nc, sh_pb_old;
  __shared__ uint64_t sh_mask;

  const int tid = threadIdx.x;
  if (tid == 0) {
    int nc = round == 0 ? min(kWindow, n - r0) : min(ps->ncand, kWindow);
    sh_nc = nc < 0 ? 0 : nc;
    sh_pb_old = ps->pb;
    sh_mask = ps->colmask;
  }
  __syncthreads();
  const int nc = sh_nc, pb_old = sh_pb_old;
  const uint64_t mask0 = sh_mask;
  if (tid < kWindow) {
    rowidx[tid] = tid < nc ? (round == 0 ? r0 + tid : ps->cand[tid]) : -1;
    ispiv[tid] = 0;
    alph[tid] = ef.in(1);
  }
  for (int idx = tid; idx < kWindow * kPanel; idx += blockDim.x) {
    (&Gc[0][0])[idx] = 0;
    (&A[0][0])[idx] = 0;
  }
  __syncthreads();
  for (int idx = tid; idx < nc * W; idx += blockDim.x) {
    const int i = idx / W, c = idx - (idx / W) * W;
    A[i][c] = ef.in(m[(int64_t)rowidx[i] * ld + col + c]);
  }
  __syncthreads();

  int npiv = 0, nb = 0;
  uint64_t newmask = 0;
  const int j = tid >> 3, sub = tid & 7;
  for (int c = 0; c < W; ++c) {
    if ((mask0 >> c) & 1ULL) continue;
    if (tid < kWindow) {
      const bool nz = tid < nc && !ispiv[tid] && !ef.zero(A[tid][c]);
      const uint32_t bal = __ballot_sync(0xffffffffu, nz);
      if ((tid & 31) == 0) ballots[nb & 1][tid >> 5] = bal;
    }
    __syncthreads();
    const uint32_t b0 = ballots[nb & 1][0], b1 = ballots[nb & 1][1];
    ++nb;
    const int piv = b0 ? __ffs(b0) - 1 : (b1 ? 31 + __ffs(b1) : -1);
    if (piv < 0) continue;
    const int t = npiv++;
    newmask |= 1ULL << c;
    const W64 e = A[piv][c];
    W64 h = 0;
    if (j < nc && j != piv && !ispiv[j]) h = A[j][c];
    __syncwarp();
    if (!ef.zero(h)) {
      const W64 nh = ef.neg(h);
      for (int cc = c + 1 + sub; cc < W; cc += 8) A[j][cc] = ef.comb(e, A[j][cc], nh, A[piv][cc]);
      for (int t2 = sub; t2 < t; t2 += 8) Gc[j][t2] = ef.comb(e, Gc[j][t2], ef.neg(0), 0);
      if (sub == 0) {
        alph[j] = ef.comb(e, alph[j], ef.neg(0), 0);
        Gc[j][t] = h;
        A[j][c] = 0;
      }
    }
    if (tid == 0) {
      ispiv[piv] = 1;
      pivcand[t] = piv;
      pivc[t] = c;
    }
    __syncthreads();
  }
  __syncthreads();

  // Outputs: pivot bookkeeping, reduced pivot rows, transformation rows.
  for (int t = tid; t < npiv; t += blockDim.x) {
    const int k = pb_old + t, i = pivcand[t];
    ps->prow[k] = rowidx[i];
    ps->pcol[k] = col + pivc[t];
    ps->alpha[k] = ef.out(alph[i]);
    const uint64_t pv = ef.out(A[i][pivc[t]]);
    ps->inv[k] = std::is_same<F, FpM61>::value ? fp_inv_m61(pv) : fp_inv(f, pv);
    is_pivot[rowidx[i]] = 1;
  }
  for (int idx = tid; idx < npiv * kPanel; idx += blockDim.x) {
    const int t = idx / kPanel, cc = idx % kPanel;
    Upanel[(int64_t)(pb_old + t) * kPanel + cc] = cc < W ? ef.out(A[pivcand[t]][cc]) : 0;
  }
  for (int idx = tid; idx < npiv * kPanel; idx += blockDim.x) {
    const int t = idx / kPanel, k2 = idx % kPanel, k = pb_old + t, i = pivcand[t];
    uint64_t v = 0;
    if (k2 < pb_old)
      v = f.mul(ef.out(alph[i]), Lbuf[(int64_t)(rowidx[i] - r0) * kPanel + k2]);
    else if (k2 < k)
      v = ef.out(Gc[i][k2 - pb_old]);
    G[(int64_t)k * kPanel + k2] = v;
  }
  if (tid == 0) {
    ps->pb = pb_old + npiv;
    ps->colmask = mask0 | newmask;
    ps->ncand = 0;
  }
}

// ---------------------------------------------------------------------------
// bulk_kernel — a warp per active non-pivot row: reference-style elimination
// of this round's new pivots pb_lo .. ps->pb from the row's panel part
// (f = e * inv, row -= f * U_k; src/fp.rs:163-175), multipliers to Lbuf,
// residual written back and, if nonzero, the row offered as a candidate.
// ---------------------------------------------------------------------------
// The pivot rows are normalised when they are loaded (U_k * inv_k), so a row's
// dependent chain is one shuffle and one multiply-add per pivot; the
// multipliers are formed afterwards (64 pivots over 2^61 - 1: 6 us for 436 rows,
// 24 with the multiplier on the chain; 60 and 79 us for 5950 rows).
template <class F>
__global__ void __launch_bounds__(256) bulk_kernel(F f, uint64_t* __restrict__ m, int64_t ld, int32_t n, int32_t r0,
                                                    int32_t col, int32_t W, int32_t pb_lo, PanelState* ps,
                                                    const uint64_t* __restrict__ Upanel, uint64_t* Lbuf,
                                                    const uint8_t* __restrict__ is_pivot) {
  using W64 = typename ElimField<F>::W;
  const ElimField<F> ef(f);
  __shared__ W64 Us[kPanel][kPanel];
  __shared__ uint64_t invs[kPanel];
  __shared__ int32_t pcs[kPanel];
  const int pb_hi = ps->pb;
  const int nk = pb_hi - pb_lo;
  for (int t = threadIdx.x; t < nk; t += blockDim.x) {
    invs[t] = ps->inv[pb_lo + t];
    pcs[t] = ps->pcol[pb_lo + t] - col;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nk * kPanel; idx += blockDim.x) {
    const int t = idx / kPanel, c = idx % kPanel;
    Us[t][c] = ef.in(c < W ? f.mul(Upanel[(int64_t)(pb_lo + t) * kPanel + c], invs[t]) : 0);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps_total = gridDim.x * (blockDim.x >> 5);
  const W64 one = ef.in(1);
  for (int r = r0 + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps_total) {
    if (is_pivot[r]) continue;
    uint64_t* row = m + (int64_t)r * ld + col;
    W64 x0 = ef.in(lane < W ? row[lane] : 0);
    W64 x1 = ef.in(lane + 32 < W ? row[lane + 32] : 0);
    W64 e0 = 0, e1 = 0;  // entries eliminated by pivots lane and lane + 32
    for (int t = 0; t < nk; ++t) {
      const int pc = pcs[t];
      const W64 e = __shfl_sync(0xffffffffu, pc < 32 ? x0 : x1, pc & 31);
      if (t < 32) {
        if (lane == t) e0 = e;
      } else if (lane == t - 32) {
        e1 = e;
      }
      const W64 ne = ef.neg(e);
      x0 = ef.comb(one, x0, ne, Us[t][lane]);
      x1 = ef.comb(one, x1, ne, Us[t][lane + 32]);
    }
    uint64_t* L = Lbuf + (int64_t)(r - r0) * kPanel + pb_lo;
    if (lane < nk) L[lane] = f.mul(ef.out(e0), invs[lane]);
    if (lane + 32 < nk) L[lane + 32] = f.mul(ef.out(e1), invs[lane + 32]);
    const uint64_t y0 = ef.out(x0), y1 = ef.out(x1);
    if (nk > 0) {
      if (lane < W) row[lane] = y0;
      if (lane + 32 < W) row[lane + 32] = y1;
    }
    const bool nz = __any_sync(0xffffffffu, (y0 | y1) != 0);
    if (nz && lane == 0) {
      const int s = atomicAdd(&ps->ncand, 1);
      if (s < kWindow) ps->cand[s] = r;
    }
  }
}

// ---------------------------------------------------------------------------
// couple_kernel — U block (src/fp.rs:184-200): for every trailing column c,
// U_k[c] = alpha_k * row_{prow_k}[c] - sum_{k2<k} G[k][k2] * U_k2[c],
// sequential in k. Eight threads share a column's sum (a CTA takes 32
// columns), lazy accumulation and a shuffle reduction per k: the chain of 64
// steps of up to 8 products each binds it (over 2^61 - 1 11 us for 436 columns,
// 118 with a thread per column; 65 and 142 us for 5950 columns).
// ---------------------------------------------------------------------------
constexpr int kCoupleCols = 32, kCoupleSplit = 8;
template <class F>
__global__ void __launch_bounds__(256) couple_kernel(F f, const uint64_t* __restrict__ m, int64_t ld, int32_t n,
                                                      int32_t jend, const PanelState* __restrict__ ps,
                                                      const uint64_t* __restrict__ G, uint64_t* Ubuf, int64_t ldU) {
  extern __shared__ __align__(16) uint64_t smem_c[];
  uint64_t(*Us)[kCoupleCols] = reinterpret_cast<uint64_t(*)[kCoupleCols]>(smem_c);  // alpha_k row_k, then U_k
  uint64_t(*Gs)[kPanel] = reinterpret_cast<uint64_t(*)[kPanel]>(smem_c + kPanel * kCoupleCols);
  const int pb = ps->pb;
  const int64_t c0 = (int64_t)jend + (int64_t)blockIdx.x * kCoupleCols;
  for (int idx = threadIdx.x; idx < pb * kPanel; idx += blockDim.x) Gs[idx / kPanel][idx % kPanel] = G[idx];
  for (int idx = threadIdx.x; idx < pb * kCoupleCols; idx += blockDim.x) {
    const int k = idx / kCoupleCols;
    const int64_t c = c0 + idx % kCoupleCols;
    Us[k][idx % kCoupleCols] = c < n ? f.mul(ps->alpha[k], m[(int64_t)ps->prow[k] * ld + c]) : 0;
  }
  __syncthreads();
  // A column's threads are neighbours in a warp.
  const int t = threadIdx.x / kCoupleSplit, q = threadIdx.x % kCoupleSplit;
  const uint64_t sb = f.safe_batch();
  for (int k = 1; k < pb; ++k) {
    u128 acc = 0;
    uint64_t cnt = 0;
    for (int k2 = q; k2 < k; k2 += kCoupleSplit) {  // at most 8 products
      acc += f.prod(Gs[k][k2], Us[k2][t]);
      if (++cnt == sb) {
        acc = f.reduce(acc);  // counts as one product
        cnt = 1;
      }
    }
    uint64_t part = f.reduce(acc);
#pragma unroll
    for (int o = 1; o < kCoupleSplit; o <<= 1) part = f.add(part, __shfl_xor_sync(0xffffffffu, part, o));
    if (q == 0) Us[k][t] = f.sub(Us[k][t], part);
    __syncwarp();
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < pb * kCoupleCols; idx += blockDim.x) {
    const int64_t c = c0 + idx % kCoupleCols;
    if (c < n) Ubuf[(int64_t)(idx / kCoupleCols) * ldU + c] = Us[idx / kCoupleCols][idx % kCoupleCols];
  }
}

// ---------------------------------------------------------------------------
// move_rows_kernel — compaction of the active block: a non-pivot row that sits
// in [r0, r0 + pb) is copied (trailing part and multiplier row) into the slot
// of a pivot row that sits in [r0 + pb, n). blockIdx.y = move.
// ---------------------------------------------------------------------------
__global__ void move_rows_kernel(uint64_t* m, int64_t ld, int32_t n, int32_t jend, const int2* moves,
                                 uint64_t* Lbuf, int32_t r0, int32_t pb) {
  const int2 mv = moves[blockIdx.y];
  const int64_t src = mv.x, dst = mv.y;
  for (int64_t c = (int64_t)jend + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
    m[dst * ld + c] = m[src * ld + c];
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < pb; k += blockDim.x)
      Lbuf[(dst - r0) * kPanel + k] = Lbuf[(src - r0) * kPanel + k];
}

__global__ void clear_pivot_flags_kernel(const PanelState* ps, uint8_t* is_pivot) {
  const int k = threadIdx.x;
  if (k < ps->pb) is_pivot[ps->prow[k]] = 0;
}

// ---------------------------------------------------------------------------
// trailing_plain_kernel — A[rbeg.., jend..cend) -= L * U mod p on the integer
// pipes (src/fp.rs:208-248): 64x64 output tile per CTA, 4x4 per thread,
// u128 accumulators, one reduction per safe_batch products. The operands of
// the whole depth K are staged in shared memory by bulk copies
// (cp.async.bulk, completion counted on one mbarrier) that warp 0 issues:
// the tile's 64 rows of L (row stride 64, so one contiguous block) and K rows
// of 64 columns of U (one 512-byte copy each). U rows that are not 16-byte
// aligned or run past cend, and an unaligned L, are loaded by the threads.
// The mbarrier wait is bounded; on expiry the CTA records err[0] = 1, waits
// (bounded) for its own copies and returns without writing C.
// ---------------------------------------------------------------------------
constexpr int kPlainSmem = 2 * 64 * 64 * 8;  // L tile + U tile

template <class F>
__global__ void __launch_bounds__(256) trailing_plain_kernel(F f, uint64_t* __restrict__ m, int64_t ld, int32_t rbeg,
                                                              int32_t n, int32_t jend, int32_t cend,
                                                              const uint64_t* __restrict__ Lbuf, int32_t r0,
                                                              const uint64_t* __restrict__ Ubuf, int64_t ldU,
                                                              int32_t K, int* err) {
  extern __shared__ __align__(128) uint64_t smem_plain[];
  uint64_t* Ls = smem_plain;            // [64][64]: tile row ri, depth k
  uint64_t* Us = smem_plain + 64 * 64;  // [64][64]: depth k, tile column ci
  __shared__ __align__(8) uint64_t bar;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t rt = (int64_t)rbeg + (int64_t)blockIdx.y * 64;
  const int64_t ct = (int64_t)jend + (int64_t)blockIdx.x * 64;
  const int rows = n - rt < 64 ? (int)(n - rt) : 64;
  const uint64_t* lsrc = Lbuf + (rt - r0) * kPanel;
  const bool bulk_l = ((uintptr_t)lsrc & 15) == 0;
  const bool bulk_u = ct + 64 <= cend && ((uintptr_t)(Ubuf + ct) & 15) == 0 && (ldU & 1) == 0;
  const uint32_t bytes = (bulk_l ? (uint32_t)rows * 512u : 0u) + (bulk_u ? (uint32_t)K * 512u : 0u);
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid < 32 && bytes) {
    if (tid == 0) tc::mbar_arrive_expect_tx(&bar, bytes);
    __syncwarp();
    if (bulk_l && tid == 0) tc::bulk_g2s(Ls, lsrc, (uint32_t)rows * 512u, &bar);
    if (bulk_u)
      for (int k = tid; k < K; k += 32) tc::bulk_g2s(Us + k * 64, Ubuf + (int64_t)k * ldU + ct, 512u, &bar);
  }
  if (!bulk_l)
    for (int idx = tid; idx < rows * 64; idx += 256) Ls[idx] = lsrc[(idx >> 6) * kPanel + (idx & 63)];
  if (!bulk_u)
    for (int idx = tid; idx < K * 64; idx += 256) {
      const int k = idx >> 6, ci = idx & 63;
      Us[idx] = ct + ci < cend ? Ubuf[(int64_t)k * ldU + ct + ci] : 0;
    }
  bool ok = true;
  if (bytes) ok = tc::mbar_wait(&bar, 0, err);
  if (!__syncthreads_and(ok)) {
    if (tid == 0) {
      atomicExch(err, 1);
      if (bytes) tc::mbar_wait(&bar, 0, err + 1);  // this CTA's copies land before it exits
    }
    return;
  }
  const uint64_t sb = f.safe_batch();
  uint64_t tot[4][4];
  u128 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      tot[i][q] = 0;
      acc[i][q] = 0;
    }
  uint64_t cnt = 0;
  for (int k = 0; k < K; ++k) {
    uint64_t a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = Ls[(ty + 16 * i) * 64 + k];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = Us[k * 64 + tx + 16 * q];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][q] += f.prod(a[i], b[q]);
    if (++cnt == sb) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          tot[i][q] = f.add(tot[i][q], f.reduce(acc[i][q]));
          acc[i][q] = 0;
        }
      cnt = 0;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t r = rt + ty + 16 * i;
    if (r >= n) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t c = ct + tx + 16 * q;
      if (c < cend) {
        uint64_t* p = m + r * ld + c;
        *p = f.sub(*p, f.add(tot[i][q], f.reduce(acc[i][q])));
      }
    }
  }
}

// ---------------------------------------------------------------------------
// plain_mac_peak_kernel — the roofline of trailing_plain_kernel: its inner
// loop (4x4 u128 accumulators per thread, operands read from shared memory,
// one reduction per safe_batch products) run `iters` times over a 64-deep
// tile that stays in shared memory, with no global traffic. The sums are
// written out so that nothing is optimised away.
// ---------------------------------------------------------------------------
template <class F>
__global__ void __launch_bounds__(256) plain_mac_peak_kernel(F f, int iters, uint64_t* out) {
  extern __shared__ __align__(128) uint64_t smem_peak[];
  uint64_t* Ls = smem_peak;
  uint64_t* Us = smem_peak + 64 * 64;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const uint64_t p = f.modulus();
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    Ls[idx] = (0x9E3779B97F4A7C15ull * (uint64_t)(idx + 1 + blockIdx.x)) % p;
    Us[idx] = (0xBF58476D1CE4E5B9ull * (uint64_t)(idx + 7)) % p;
  }
  __syncthreads();
  const uint64_t sb = f.safe_batch();
  uint64_t tot[4][4];
  u128 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      tot[i][q] = 0;
      acc[i][q] = 0;
    }
  uint64_t cnt = 0;
  for (int it = 0; it < iters; ++it)
    for (int k = 0; k < 64; ++k) {
      uint64_t a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = Ls[(ty + 16 * i) * 64 + k];
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = Us[k * 64 + tx + 16 * q];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] += (u128)a[i] * b[q];
      if (++cnt == sb) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            tot[i][q] = f.add(tot[i][q], f.reduce(acc[i][q]));
            acc[i][q] = 0;
          }
        cnt = 0;
      }
    }
  uint64_t s = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) s ^= f.add(tot[i][q], f.reduce(acc[i][q]));
  out[(int64_t)blockIdx.x * 256 + tid] = s;
}

template <class F>
cudaError_t launch_plain_mac_peak(const F& f, int blocks, int iters, uint64_t* out, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(plain_mac_peak_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kPlainSmem);
  if (e != cudaSuccess) return e;
  plain_mac_peak_kernel<F><<<blocks, 256, kPlainSmem, st>>>(f, iters, out);
  return cudaGetLastError();
}

template <class F>
int plain_blocks_per_sm() {
  cudaFuncSetAttribute(trailing_plain_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPlainSmem);
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, trailing_plain_kernel<F>, 256, kPlainSmem);
  return nb;
}

// ---------------------------------------------------------------------------
// gj64_inverse — one CTA of kInvThreads (8 per block row): the inverse of
// the 64 x 64 block P = A[r0 .. r0+64, col .. col+64), or status = 1 when P
// is singular. In-place fraction-free Gauss-Jordan: at
// column c with pivot row `piv` (the first row not yet used whose entry is
// nonzero) every other row j becomes e * row_j - h * row_piv (e = P[piv][c],
// h = P[j][c]: one reduction of the two-product sum per entry), and column c,
// now zero outside the pivot, stores column `piv` of the accumulated row
// operations E instead (-h s and s in the pivot row, s = the scale row piv
// took while it was not a pivot). Row j's remaining left entry d_j is tracked
// apart. At the end P^-1 [pc_j][i] = E[j][i] / d_j with
// E[j][i] stored at column pc_i. One block barrier per column: the owner of
// column c+1 in each row flags a nonzero entry before it, and every warp then
// finds the pivot by itself with a ballot over the flags.
// Output: Vneg[c][i] = -(P^-1)[c][i] (row c = panel column, column i =
// block row), the B operand of the multiplier GEMM H = X_P * P^-1.
// ---------------------------------------------------------------------------
template <class F>
__device__ void gj64_inverse(const F& f, const uint64_t* __restrict__ m, int64_t ld, int32_t r0, int32_t col,
                             uint64_t* __restrict__ Vneg, int* status, const Guard& g, uint64_t* smem_inv) {
  uint64_t(*M)[kPanel + 1] = reinterpret_cast<uint64_t(*)[kPanel + 1]>(smem_inv);
  __shared__ uint64_t d[kPanel], dinv[kPanel], sc[kPanel];
  __shared__ int32_t pc[kPanel];
  __shared__ uint8_t nz[2][kPanel];  // nz[c & 1][j]: row j's entry in column c is nonzero
  const uint64_t p = f.modulus();
  constexpr int kRow = kInvThreads / kPanel;  // threads per block row
  const int tid = threadIdx.x, j = tid / kRow, s = tid % kRow;
#pragma unroll
  for (int q = 0; q < kPanel / kRow; ++q) M[j][s + kRow * q] = m[(int64_t)(r0 + j) * ld + col + s + kRow * q];
  if (s == 0) {
    d[j] = 0;
    sc[j] = 1;
    nz[0][j] = M[j][0] != 0;  // written by this thread just above
  }
  __syncthreads();
  const int lane = tid & 31;
  unsigned long long used = 0;  // rows that are pivots already (same in every thread)
  int last_piv = -1;     // the previous column's pivot row: its column gets E's entry now
  uint64_t last_sc = 0;  // that entry: the pivot row's scale
  for (int c = 0; c < kPanel; ++c) {
    // Deferred from the previous column, after every thread has read the
    // pivot value there; only this thread reads this entry before the next
    // barrier.
    if (j == last_piv && s == (c - 1) % kRow) M[j][c - 1] = last_sc;
    // Every warp finds the pivot itself: the first row not yet used with a
    // nonzero entry in column c (a ballot over the 64 rows' flags, set before
    // the barrier by the thread that owns column c of each row).
    const bool lo = !((used >> lane) & 1) && nz[c & 1][lane];
    const bool hi = !((used >> (lane + 32)) & 1) && nz[c & 1][lane + 32];
    const uint32_t b0 = __ballot_sync(0xffffffffu, lo), b1 = __ballot_sync(0xffffffffu, hi);
    if ((b0 | b1) == 0) {  // no pivot in column c: P is singular
      if (tid == 0) {
        if (status) *status = 1;
        if (g.bad) atomicMin(g.bad, g.step + 1);  // the chain of step g.step + 1 failed
      }
      return;
    }
    const int piv = b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
    const uint64_t e = M[piv][c];
    const uint64_t spiv = sc[piv];  // E[piv][piv]: the scale row piv took while unused
    const uint64_t h = j != piv ? M[j][c] : 0;
    __syncwarp();  // every read of M[j][c] precedes its overwrite below
    if (h != 0) {
      const uint64_t nh = p - h;
#pragma unroll
      for (int q = 0; q < kPanel / kRow; ++q) {
        const int k = s + kRow * q;
        M[j][k] = f.reduce2(f.prod(e, M[j][k]) + f.prod(nh, M[piv][k]));
      }
      if (s == c % kRow) M[j][c] = f.mul(nh, spiv);  // column c now holds E's column piv
      if (s == 0) {
        if ((used >> j) & 1)
          d[j] = f.mul(e, d[j]);
        else
          sc[j] = f.mul(e, sc[j]);
      }
    }
    if (j == piv && s == 0) {
      d[j] = e;
      pc[j] = c;
    }
    const int cn = c + 1;
    if (cn < kPanel && s == cn % kRow) nz[cn & 1][j] = M[j][cn] != 0;
    last_piv = piv;
    last_sc = spiv;
    used |= 1ULL << piv;
    __syncthreads();
  }
  if (j == last_piv && s == (kPanel - 1) % kRow) M[j][kPanel - 1] = last_sc;
  if (tid < kPanel) dinv[tid] = fp_inv_binary(d[tid], p);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPanel / kRow; ++q) {
    const int i = s + kRow * q;
    const uint64_t v = f.mul(M[j][pc[i]], dinv[j]);
    Vneg[(int64_t)pc[j] * kPanel + i] = v ? p - v : 0;
  }
}


// ---------------------------------------------------------------------------
// block_inverse_kernel — one CTA: inv64 (block_inv.cuh), or on its failure (a
// 16-column block without a pivot) the pivoting Gauss-Jordan over all 64 rows,
// so the result never depends on the path. Output as gj64_inverse. On the
// look-ahead chain: the latency of 64 dependent column steps (~400 cycles
// each) and the K = 16 products between them. Measured over 2^61 - 1 28 us
// (75 as a recursive inverse with all products on the integer pipes), mod
// 65521 32 us (76; 347 by the pivoting Gauss-Jordan with 128-bit
// reductions).
// ---------------------------------------------------------------------------
template <class F, int LIMBS>
__device__ bool inv64_block(const F& f, const uint64_t* __restrict__ m, int64_t ld, int32_t r0, int32_t col,
                            uint64_t* __restrict__ Vneg, uint64_t* smem) {
  const LimbRed<F, LIMBS> red(f);
  const uint64_t p = f.modulus();
  uint64_t* M = smem;
  InvScratch<LIMBS>& S = *reinterpret_cast<InvScratch<LIMBS>*>(smem + kPanel * kInvLd);
  for (int t = threadIdx.x; t < kPanel * kPanel; t += kInvThreads)
    M[(t >> 6) * kInvLd + (t & 63)] = m[(int64_t)(r0 + (t >> 6)) * ld + col + (t & 63)];
  __syncthreads();
  if (!inv64<F, LIMBS, kInvThreads>(f, red, M, S)) return false;
  for (int t = threadIdx.x; t < kPanel * kPanel; t += kInvThreads) {
    const int c = t >> 6, i = t & 63;
    const uint64_t v = f.mul(M[c * kInvLd + i], S.fac[c >> 4]);
    Vneg[c * kPanel + S.order[i]] = v ? p - v : 0;
  }
  return true;
}

template <class F>
__global__ void __launch_bounds__(kInvThreads) block_inverse_kernel(F f, const uint64_t* __restrict__ m, int64_t ld,
                                                                     int32_t r0, int32_t col,
                                                                     uint64_t* __restrict__ Vneg, int* status,
                                                                     int reset_status, Guard g) {
  extern __shared__ __align__(16) uint64_t smem_inv[];
  pdl_wait();
  if (guard_skip(g)) return;  // an earlier step of the pipeline failed
  if (reset_status && status && threadIdx.x == 0) *status = 0;
  bool ok;
  if constexpr (std::is_same<F, FpSmall>::value) {
    const uint64_t p = f.modulus();
    ok = p <= (1ULL << 8)    ? inv64_block<F, 1>(f, m, ld, r0, col, Vneg, smem_inv)
         : p <= (1ULL << 16) ? inv64_block<F, 2>(f, m, ld, r0, col, Vneg, smem_inv)
                             : inv64_block<F, 4>(f, m, ld, r0, col, Vneg, smem_inv);
  } else {
    ok = inv64_block<F, 8>(f, m, ld, r0, col, Vneg, smem_inv);
  }
  if (ok) return;
  // With no status word to fill (a chain of the block pipeline) the answer
  // may be "not inverted": such a panel takes the general path. Over a large
  // prime an invertible block fails with probability 64 / p, so the pivoting
  // elimination is left out (a 64 x 64 matrix of rank 32 over 2^61 - 1: 239 us
  // with it, 188 without).
  if (!status && f.modulus() >> 20) {
    if (threadIdx.x == 0 && g.bad) atomicMin(g.bad, g.step + 1);
    return;
  }
  __syncthreads();
  gj64_inverse(f, m, ld, r0, col, Vneg, status, g, smem_inv);
}

// ---------------------------------------------------------------------------
// small_gemm64_kernel — C = D - A * B (negate) or C = D + A * B on 64 x 64
// blocks mod p (D may be null: zero), or the copy C = D when A is null; up to
// kSgMaxProbs independent problems per launch, 16 CTAs of 256 threads each,
// one 16 x 16 output tile per CTA, so the products spread over the SMs a
// finished trailing update leaves free. On the chain between two block steps:
// limb products on the tensor cores (mma_limbs.cuh), a warp per 16 x 8 tile and
// 32 of the inner dimension, the parts added afterwards. Over 2^61 - 1 4.4 us
// on average (K = 64 and 128); 5.5 and 10 with a thread per output.
// ---------------------------------------------------------------------------
constexpr int kSgTile = 16;
constexpr int kSgStride = 2 * kPanel + 16;  // bytes per row of a limb plane
struct SgBatch {
  SgProb p[kSgMaxProbs];
  Guard g;
};
template <class F, int LIMBS>
__global__ void __launch_bounds__(256) small_gemm64_kernel(F f, SgBatch batch) {
  __shared__ __align__(16) uint8_t As[LIMBS][kSgTile][kSgStride], Bs[LIMBS][kSgTile][kSgStride];
  __shared__ uint64_t part[8][4][32];
  pdl_wait();
  if (guard_skip(batch.g)) return;
  const SgProb& P = batch.p[blockIdx.x >> 4];
  const int tid = threadIdx.x, i = tid >> 4, j = tid & 15, lane = tid & 31, warp = tid >> 5;
  const int ti = (blockIdx.x >> 2) & 3, tj = blockIdx.x & 3;
  const int r = ti * kSgTile + i, c = tj * kSgTile + j;
  if (!P.A) {  // copy
    P.C[(int64_t)r * P.ldc + c] = P.D[(int64_t)r * P.ldd + c];
    return;
  }
  const int K = P.k == 2 * kPanel ? 2 * kPanel : kPanel;
  constexpr int kPl = kSgTile * kSgStride;
  uint64_t va[2][4], vb[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = 4 * (j + 16 * h);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      va[h][u] = k < K ? P.A[(int64_t)(ti * kSgTile + i) * P.lda + k + u] : 0;
      vb[h][u] = 4 * (i + 16 * h) < K ? P.B[(int64_t)(4 * (i + 16 * h) + u) * P.ldb + tj * kSgTile + j] : 0;
    }
  }
  const uint64_t d = P.D ? P.D[(int64_t)r * P.ldd + c] : 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    mml::put_planes4<LIMBS>(&As[0][i][4 * (j + 16 * h)], kPl, va[h]);
    mml::put_planes4<LIMBS>(&Bs[0][j][4 * (i + 16 * h)], kPl, vb[h]);
  }
  __syncthreads();
  const LimbRed<F, LIMBS> red(f);
  const int kc = warp >> 1, kcs = K / 32;
  if (kc < kcs) {
    uint32_t acc[2 * LIMBS - 1][4];
    mml::tile_k32<LIMBS, 1, kSgStride>(acc, mml::saddr(As) + 32 * kc, kPl,
                                       mml::saddr(&Bs[0][8 * (warp & 1)][0]) + 32 * kc, kPl);
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][e][lane] = red.residue(acc, e);
  }
  __syncthreads();
  // Entry (i, j): tile column j / 8, lane 4 (i mod 8) + (j mod 8) / 2.
  const int e = (i >> 3) * 2 + (j & 1), ln = 4 * (i & 7) + ((j & 7) >> 1);
  uint64_t v = 0;
  for (int q = 0; q < kcs; ++q) v = f.add(v, part[2 * q + (j >> 3)][e][ln]);
  P.C[(int64_t)r * P.ldc + c] = P.negate ? f.sub(d, v) : f.add(d, v);
}

__global__ void zero_kernel(uint64_t* __restrict__ p, int64_t n, Guard g) {
  pdl_wait();
  if (guard_skip(g)) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = 0;
}

// ---------------------------------------------------------------------------
// any_nonzero_kernel — *flag = 1 when some entry of rows [r0, n), columns
// [c0, n) is nonzero: a zero rest ends the rank (a matrix of recurrence rows is
// zero after its order's pivots). A warp per 256 columns of a row; DRAM-bound,
// and over at once when an entry is found.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) any_nonzero_kernel(const uint64_t* __restrict__ m, int64_t ld, int32_t r0,
                                                          int32_t c0, int32_t n, int* flag) {
  const int lane = threadIdx.x & 31;
  const int64_t per_row = (n - c0 + 255) / 256, items = per_row * (n - r0);
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < items; q += warps) {
    if (*(volatile int*)flag) return;
    const uint64_t* row = m + (r0 + q / per_row) * ld;
    const int64_t c = c0 + (q % per_row) * 256 + lane;
    uint64_t v = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (c + 32 * k < n) v |= row[c + 32 * k];
    if (__any_sync(0xffffffffu, v != 0)) {
      if (lane == 0) atomicExch(flag, 1);
      return;
    }
  }
}

// ---------------------------------------------------------------------------
// Launch wrappers (explicit instantiation for both field policies).
// ---------------------------------------------------------------------------
template <class F>
void launch_window(const F& f, const uint64_t* m, int64_t ld, int n, int r0, int col, int W, int round,
                   PanelState* ps, uint64_t* Upanel, uint64_t* G, const uint64_t* Lbuf, uint8_t* is_pivot,
                   cudaStream_t st) {
  const size_t smem = 2 * kWindow * kPanel * sizeof(uint64_t);
  static PerDevice once;
  allow_smem(once, window_kernel<F>, smem);
  window_kernel<F><<<1, kWindowThreads, smem, st>>>(f, m, ld, n, r0, col, W, round, ps, Upanel, G, Lbuf, is_pivot);
}

template <class F>
void launch_bulk(const F& f, uint64_t* m, int64_t ld, int n, int r0, int col, int W, int pb_lo, PanelState* ps,
                 const uint64_t* Upanel, uint64_t* Lbuf, const uint8_t* is_pivot, int num_sms, cudaStream_t st) {
  const int rows = n - r0;
  int blocks = (rows + 7) / 8;
  const int cap = num_sms * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  bulk_kernel<F><<<blocks, 256, 0, st>>>(f, m, ld, n, r0, col, W, pb_lo, ps, Upanel, Lbuf, is_pivot);
}

template <class F>
void launch_couple(const F& f, const uint64_t* m, int64_t ld, int n, int jend, const PanelState* ps,
                   const uint64_t* G, uint64_t* Ubuf, int64_t ldU, cudaStream_t st) {
  const int cols = n - jend;
  const size_t smem = (size_t)(kPanel * kCoupleCols + kPanel * kPanel) * sizeof(uint64_t);
  static PerDevice once;
  allow_smem(once, couple_kernel<F>, smem);
  couple_kernel<F><<<(cols + kCoupleCols - 1) / kCoupleCols, 256, smem, st>>>(f, m, ld, n, jend, ps, G, Ubuf, ldU);
}

void launch_moves(uint64_t* m, int64_t ld, int n, int jend, const int2* moves, int nmoves, uint64_t* Lbuf, int r0,
                  int pb, cudaStream_t st) {
  if (nmoves <= 0) return;
  const int cols = n - jend;
  int bx = (cols + 255) / 256;
  if (bx > 64) bx = 64;
  if (bx < 1) bx = 1;
  move_rows_kernel<<<dim3(bx, nmoves), 256, 0, st>>>(m, ld, n, jend, moves, Lbuf, r0, pb);
}

void launch_clear_flags(const PanelState* ps, uint8_t* is_pivot, cudaStream_t st) {
  clear_pivot_flags_kernel<<<1, kPanel, 0, st>>>(ps, is_pivot);
}

template <class F>
void launch_trailing_plain(const F& f, uint64_t* m, int64_t ld, int rbeg, int rend, int jend, int cend,
                           const uint64_t* Lbuf, int r0, const uint64_t* Ubuf, int64_t ldU, int K, int* err,
                           cudaStream_t st) {
  if (rbeg >= rend || jend >= cend || K <= 0) return;
  static PerDevice once;
  allow_smem(once, trailing_plain_kernel<F>, kPlainSmem);
  dim3 grid((cend - jend + 63) / 64, (rend - rbeg + 63) / 64);
  trailing_plain_kernel<F><<<grid, 256, kPlainSmem, st>>>(f, m, ld, rbeg, rend, jend, cend, Lbuf, r0, Ubuf, ldU, K,
                                                           err);
}

template <class F>
void launch_block_inverse(const F& f, const uint64_t* m, int64_t ld, int r0, int col, uint64_t* Vneg, int* status,
                          cudaStream_t st, bool reset_status, const Guard& g) {
  const size_t smem = kPanel * kInvLd * 8 + sizeof(InvScratch<8>);  // more than the pivoting path's kPanel * (kPanel + 1) words
  static PerDevice once;
  allow_smem(once, block_inverse_kernel<F>, smem);
  launch_k(block_inverse_kernel<F>, dim3(1), dim3(kInvThreads), smem, st, 1, f, m, ld, (int32_t)r0, (int32_t)col,
           Vneg, status, reset_status ? 1 : 0, g);
}

template <class F>
void launch_small_gemm64_batch(const F& f, const SgProb* probs, int count, cudaStream_t st, const Guard& g) {
  SgBatch b = {};
  b.g = g;
  for (int i = 0; i < count && i < kSgMaxProbs; ++i) b.p[i] = probs[i];
  const int n = count < kSgMaxProbs ? count : kSgMaxProbs;
  const dim3 grid(16 * n);
  if constexpr (std::is_same<F, FpSmall>::value) {
    const uint64_t p = f.modulus();
    if (p <= (1ULL << 8))
      launch_k(small_gemm64_kernel<F, 1>, grid, dim3(256), 0, st, 1, f, b);
    else if (p <= (1ULL << 16))
      launch_k(small_gemm64_kernel<F, 2>, grid, dim3(256), 0, st, 1, f, b);
    else
      launch_k(small_gemm64_kernel<F, 4>, grid, dim3(256), 0, st, 1, f, b);
  } else {
    launch_k(small_gemm64_kernel<F, 8>, grid, dim3(256), 0, st, 1, f, b);
  }
}

template <class F>
void launch_small_gemm64(const F& f, const uint64_t* A, int64_t lda, const uint64_t* B, int64_t ldb, const uint64_t* D,
                         int64_t ldd, uint64_t* C, int64_t ldc, bool negate, cudaStream_t st, const Guard& g) {
  const SgProb pr = {A, B, D, C, lda, ldb, ldd, ldc, negate ? 1 : 0, kPanel};
  launch_small_gemm64_batch<F>(f, &pr, 1, st, g);
}

void launch_zero(uint64_t* p, int64_t n, cudaStream_t st, const Guard& g) {
  if (n <= 0) return;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 1184) blocks = 1184;
  launch_k(zero_kernel, dim3((unsigned)blocks), dim3(256), 0, st, 1, p, n, g);
}

cudaError_t launch_any_nonzero(const uint64_t* m, int64_t ld, int r0, int c0, int n, int* flag, int num_sms,
                               cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  any_nonzero_kernel<<<num_sms * 8, 256, 0, st>>>(m, ld, r0, c0, n, flag);
  return cudaGetLastError();
}

#define INSTANTIATE(F)                                                                                          \
  template void launch_small_gemm64<F>(const F&, const uint64_t*, int64_t, const uint64_t*, int64_t,            \
                                       const uint64_t*, int64_t, uint64_t*, int64_t, bool, cudaStream_t,        \
                                       const Guard&);                                                           \
  template void launch_block_inverse<F>(const F&, const uint64_t*, int64_t, int, int, uint64_t*, int*,          \
                                        cudaStream_t, bool, const Guard&);                                      \
  template void launch_small_gemm64_batch<F>(const F&, const SgProb*, int, cudaStream_t, const Guard&);         \
  template void launch_window<F>(const F&, const uint64_t*, int64_t, int, int, int, int, int, PanelState*,       \
                                 uint64_t*, uint64_t*, const uint64_t*, uint8_t*, cudaStream_t);                \
  template void launch_bulk<F>(const F&, uint64_t*, int64_t, int, int, int, int, int, PanelState*,              \
                               const uint64_t*, uint64_t*, const uint8_t*, int, cudaStream_t);                  \
  template void launch_couple<F>(const F&, const uint64_t*, int64_t, int, int, const PanelState*,               \
                                 const uint64_t*, uint64_t*, int64_t, cudaStream_t);                            \
  template void launch_trailing_plain<F>(const F&, uint64_t*, int64_t, int, int, int, int, const uint64_t*, int, \
                                         const uint64_t*, int64_t, int, int*, cudaStream_t);                        \
  template cudaError_t launch_plain_mac_peak<F>(const F&, int, int, uint64_t*, cudaStream_t);                      \
  template int plain_blocks_per_sm<F>();

INSTANTIATE(FpBarrett)
INSTANTIATE(FpSmall)
INSTANTIATE(FpM61)

}  // namespace modlin
