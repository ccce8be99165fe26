// What the batched rank's kernels share: tile layout, sums, shared memory.
#pragma once
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <type_traits>

#include "block_inv.cuh"
#include "field.cuh"
#include "mma_limbs.cuh"
#include "rank_batch.cuh"

namespace modlin {

namespace {

constexpr int kP = 64;  // panel width
constexpr int kG = 8;   // rows per warp in flight during the in-panel elimination
constexpr int kStride = 80;                // bytes per row of a 64-deep limb plane
constexpr int kPlane = kP * kStride;       // one limb plane of a 64 x 64 tile
constexpr int kRegion = 8 * kPlane;        // 8 limb planes: 40 KiB

// Lazy accumulation of products of residues: u128 sums reduced once per
// safe_batch products in general; for p < 2^32 a product fits in 32 x 32 ->
// 64 bits, so the sums stay in a u64 and are reduced once per
// floor((2^64 - 1) / (p - 1)^2) products (at least 1; p < 2^31 gives >= 4).
// A reduced sum (< p) counts as one product.
template <class F>
struct Acc {
  using T = u128;
  __device__ static T prod(const F& f, uint64_t a, uint64_t b) { return f.prod(a, b); }
  __device__ static uint64_t reduce(const F& f, T x) { return f.reduce(x); }
  __device__ static uint64_t batch(const F& f) { return f.safe_batch(); }
};
template <>
struct Acc<FpSmall> {
  using T = uint64_t;
  __device__ static T prod(const FpSmall&, uint64_t a, uint64_t b) { return (uint64_t)(uint32_t)a * (uint32_t)b; }
  __device__ static uint64_t reduce(const FpSmall& f, T x) { return f.reduce64(x); }
  __device__ static uint64_t batch(const FpSmall& f) {
    const uint64_t q = f.modulus() - 1;
    return q <= 1 ? UINT64_MAX : UINT64_MAX / (q * q);
  }
};

// Regions of shared memory: `a` holds the block being inverted, then the left
// operand's planes, or LF on the panel path; `b` the inverse's scratch, then
// the right operand's planes, or Us; `a2` (one CTA an SM) the left operand's
// second buffer.
struct BatchSmem {
  alignas(16) uint8_t b[kRegion];
  alignas(16) uint8_t a[kRegion];
  uint64_t prow[kP];  // pivot row's panel segment, scaled
  int pcol[kP];
  int red[16];
  int found;
  long long job;
};
static_assert(sizeof(InvScratch<8>) <= kRegion && kP * kInvLd * 8 <= kRegion && kP * (kP + 1) * 8 <= kRegion, "");

// Diagonal sums of the 16 x 8 tile (row group rg, column group cg) of the
// 64 x 64 product of the planes at A and B.
template <int LIMBS>
__device__ __forceinline__ void block_tile(uint32_t (&acc)[2 * LIMBS - 1][4], const uint8_t* A, const uint8_t* B,
                                           int rg, int cg) {
  mml::tile_k32<LIMBS, 2, kStride>(acc, mml::saddr(A) + rg * 16 * kStride, kPlane, mml::saddr(B) + cg * 8 * kStride,
                                   kPlane);
}

// A kernel's shared memory and row map: SM::kT threads, SM::smem(), SM::a2()
// (the left operand's second buffer) and SM::perm() (the row order).

// A warp's tiles of a 64 x 64 output: rows 16 rg .. +16, kTiles groups of 8
// columns from cg0; and a thread's share of a left operand (64 rows of 64).
template <int kT>
struct TileMap {
  static constexpr int kTiles = 32 / (kT / 32), kRound = kT / 16, kN = kP / kRound;
};

// Left operand: rows rt .. rt + 63, columns c0 .. c0 + 63, through registers.
template <int kT>
__device__ __forceinline__ void load_rows(const uint64_t* __restrict__ m, int n, const int* perm, int c0, int rt,
                                          uint64_t (&v)[TileMap<kT>::kN][4]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int w = 0; w < TileMap<kT>::kN; ++w) {
    const int i = (tid >> 4) + TileMap<kT>::kRound * w, k4 = 4 * (tid & 15);
    const uint64_t* src = rt + i < n ? m + (int64_t)perm[rt + i] * n + c0 + k4 : nullptr;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[w][u] = src ? src[u] : 0;
  }
}
template <int LIMBS, int kT>
__device__ __forceinline__ void put_rows(uint8_t* dst, const uint64_t (&v)[TileMap<kT>::kN][4]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int w = 0; w < TileMap<kT>::kN; ++w)
    mml::put_planes4<LIMBS>(dst + ((tid >> 4) + TileMap<kT>::kRound * w) * kStride + 4 * (tid & 15), kPlane, v[w]);
}

// C += H U for the row tiles of 64 at rb, rb + stride, .. and the columns from
// cb: H in columns c0 .. c0 + 63 of those rows, U the first pb of the rows at r0
// (H's other columns are zero). Whether this thread wrote something nonzero.
// A function of its own: its registers are the products'.
template <class F, int LIMBS, class SM>
__device__ __noinline__ bool update_rest(const F& fr, uint64_t* __restrict__ m, const int n, int r0, int pb, int rb,
                                         int stride, int c0, int cb) {
  BatchSmem& S = SM::smem();
  int* const perm = SM::perm();
  const F f = fr;
  const LimbRed<F, LIMBS> red(f);
  constexpr int kT = SM::kT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kTiles = TileMap<kT>::kTiles, kN = TileMap<kT>::kN;
  // The next tile's rows are loaded during this one's products where the
  // registers allow; with two buffers one barrier a tile is enough.
  constexpr bool kTwo = kT == 512, kEarly = LIMBS <= 4;
  const int rg = warp & 3, cg0 = (warp >> 2) * kTiles;
  const int g = lane >> 2, t2 = 2 * (lane & 3);
  uint8_t* const bufs[2] = {S.a, kTwo ? SM::a2() : S.a};
  uint32_t acc[2 * LIMBS - 1][4];
  uint64_t lv[kN][4];
  // Past the pivots H is zero: any of U's rows will do.
  const auto row = [pb](int k) { return k < pb ? k : 0; };
  // Strips of kCols column tiles whose right operands fill region b: the left
  // operand's load and the barriers are shared by them.
  constexpr int kCols = LIMBS == 8 || !kTwo ? 1 : LIMBS == 4 ? 2 : 4;
  bool nz = false;
  for (int ct = cb; ct < n && rb < n; ct += kP * kCols) {
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
          uv[w][u] = col < n ? m[(int64_t)perm[r0 + row(4 * ((tid >> 6) + kRows4 * w) + u)] * n + col] : 0;
#pragma unroll
      for (int w = 0; w < kN; ++w)
        mml::put_planes4<LIMBS>(S.b + s * LIMBS * kPlane + (tid & 63) * kStride + 4 * ((tid >> 6) + kRows4 * w),
                                kPlane, uv[w]);
    }
    if (kEarly) load_rows<kT>(m, n, perm, c0, rb, lv);
    for (int rt = rb, k = 0; rt < n; rt += stride, k ^= 1) {
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
      if (!kEarly) load_rows<kT>(m, n, perm, c0, rt, lv);
      if (!kTwo && rt > rb) __syncthreads();
      put_rows<LIMBS, kT>(bufs[k], lv);
      __syncthreads();
      if (kEarly && rt + stride < n) load_rows<kT>(m, n, perm, c0, rt + stride, lv);
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
  return nz;
}

// How often a block step is tried with other rows at `rows` remaining ones. A
// failed attempt costs an inverse (10 to 30 us), so it has to be bad luck: a
// uniform 64 x 64 block fails with probability 4 / p, whereas dependent columns
// fail for all rows, and do so in every panel of some matrices (150 of side 500
// mod 2 with a dependent column in each panel: 14.6 ms with three tries and the
// update on the integer pipes, 7.9 now). Where failure is chance, all three pay:
// 300 of side 384 mod 5 3.5 ms with three, 4.2 with two, 4.7 with one; mod 3, on
// long matrices only, 5.3 with three and 6.7 without.
__device__ __forceinline__ int block_tries(uint64_t p, int rows) {
  if (p < 5) return p == 3 && rows >= 320 ? 3 : 0;  // 0.7 and 10 % succeed mod 2 and 3
  return p < 256 ? 3 : 1;
}

// The panel's arithmetic: residues below 2^32 in 32 bits, and for 16-bit primes
// 32-bit products reduced by the rounded-down reciprocal (at most 2 p too many).
template <class F, int LIMBS>
struct PanelField {
  using V = uint64_t;
  const F f;
  __device__ explicit PanelField(const F& g) : f(g) {}
  __device__ __forceinline__ V mul(V a, V b) const { return f.mul(a, b); }
  __device__ __forceinline__ V sub(V a, V b) const { return f.sub(a, b); }
};
template <int LIMBS>
struct PanelField<FpSmall, LIMBS> {
  using V = uint32_t;
  const FpSmall f;
  const uint32_t p, mu;
  __device__ explicit PanelField(const FpSmall& g) : f(g), p((uint32_t)g.modulus()), mu(0xffffffffu / p) {}
  __device__ __forceinline__ V mul(V a, V b) const {
    if constexpr (LIMBS > 2) {
      return (V)f.mul(a, b);
    } else {
      const uint32_t x = a * b;
      uint32_t r = x - __umulhi(x, mu) * p;  // < 3 p
      r = min(r, r - p);
      return min(r, r - p);
    }
  }
  __device__ __forceinline__ V sub(V a, V b) const { return a >= b ? a - b : a + p - b; }
};

// ---------------------------------------------------------------------------
// The panel path: W columns from c0 without a block step, as the reference's
// (src/fp.rs:146-200).
// eliminate_panel: in-panel elimination of the rows from r0 on, the first nonzero
// row as pivot. The pivots come first in the row order, the multipliers stay in
// the pivots' columns (S.pcol). Returns the number of pivots. 296 matrices of
// side 63 mod 65521 take 200 us (273 with four barriers, 64-bit arithmetic and up
// to three products a row and column), over 2^61 - 1 368 (382). Bound by
// instruction issue and the chain of a column, with two barriers: warp 0 fetches
// the pivot row, inverts the pivot and scales the row by it, then all warps
// update their rows and look for the next column's pivot on the way.
// ---------------------------------------------------------------------------
template <class F, int LIMBS, class SM>
__device__ __noinline__ int eliminate_panel(const F& fr, uint64_t* __restrict__ m, const int n, int r0, int c0, int W) {
  using V = typename PanelField<F, LIMBS>::V;
  BatchSmem& S = SM::smem();
  int* const perm = SM::perm();
  const PanelField<F, LIMBS> f(fr);
  constexpr int kT = SM::kT, kWarps = kT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Whether rows r on hold something nonzero in the panel's columns from k on,
  // and into S.red, per warp, the first of them with an entry in column k.
  const auto scan = [&](int r, int k) {
    int first = INT_MAX;
    V any = 0;
    for (int base = r + warp; base < n; base += kWarps * kG) {
      V x0[kG], x1[kG];
#pragma unroll
      for (int g = 0; g < kG; ++g) {
        const int i = base + g * kWarps;
        const uint64_t* R = i < n ? m + (int64_t)perm[i] * n + c0 : nullptr;
        x0[g] = R && lane >= k && lane < W ? (V)R[lane] : 0;
        x1[g] = R && lane + 32 >= k && lane + 32 < W ? (V)R[lane + 32] : 0;
      }
#pragma unroll
      for (int g = 0; g < kG; ++g) {
        any |= x0[g] | x1[g];
        if ((k < 32 ? x0[g] : x1[g]) != 0) first = min(first, base + g * kWarps);
      }
    }
    first = __shfl_sync(0xffffffffu, first, k & 31);
    if (lane == 0) S.red[warp] = first;
    return __syncthreads_or(any != 0) != 0;
  };
  int pb = 0;
  if (!scan(r0, 0)) return 0;
  for (int kk = 0; kk < W && r0 + pb < n; ++kk) {
    const int r = r0 + pb;
    if (warp == 0) {
      const int b = __reduce_min_sync(0xffffffffu, lane < kWarps ? S.red[lane] : INT_MAX);
      if (b != INT_MAX) {
        const int row = perm[b], other = perm[r];
        const uint64_t* P = m + (int64_t)row * n + c0;
        const V x0 = lane < W ? (V)P[lane] : 0, x1 = lane + 32 < W ? (V)P[lane + 32] : 0;
        const uint64_t e = __shfl_sync(0xffffffffu, kk < 32 ? x0 : x1, kk & 31);
        const V inv = (V)(std::is_same<F, FpM61>::value ? fp_inv_m61(e) : fp_inv_binary(e, fr.modulus()));
        S.prow[lane] = lane > kk ? f.mul(x0, inv) : lane == kk ? inv : 0;
        S.prow[lane + 32] = lane + 32 > kk ? f.mul(x1, inv) : lane + 32 == kk ? inv : 0;
        if (lane == 0) {
          perm[b] = other;
          perm[r] = row;
          S.pcol[pb] = c0 + kk;
        }
      }
      if (lane == 0) S.found = b != INT_MAX;
    }
    __syncthreads();
    const int kn = kk + 1;
    if (!S.found) {
      if (kn < W && !scan(r, kn)) break;  // nothing is left in the panel
      continue;
    }
    // Up to kG rows per warp at a time, without branches between them, so that
    // their loads and chains overlap: lane l holds panel entries l and l + 32 of
    // each row. A row's multiplier is its entry times the inverse, its other
    // entries lose the entry times the scaled pivot row: one product per half
    // of the row.
    const V pv0 = (V)S.prow[lane], pv1 = (V)S.prow[lane + 32];
    const bool h0 = kk < 32, h1 = W > 32;  // the halves that change
    const bool put0 = lane >= kk && lane < W, put1 = lane + 32 >= kk && lane + 32 < W;
    int next = INT_MAX;  // in lane kn: the first row with an entry in column kn
    const auto rows = [&](auto count, int base) {
      constexpr int N = decltype(count)::value;
      uint64_t* R[N];
      V x0[N], x1[N], e[N];
#pragma unroll
      for (int g = 0; g < N; ++g) {
        const int i = base + g * kWarps;
        R[g] = i < n ? m + (int64_t)perm[i] * n + c0 : nullptr;
        x0[g] = R[g] && h0 && lane < W ? (V)R[g][lane] : 0;
        x1[g] = R[g] && lane + 32 < W ? (V)R[g][lane + 32] : 0;
      }
#pragma unroll
      for (int g = 0; g < N; ++g) e[g] = __shfl_sync(0xffffffffu, h0 ? x0[g] : x1[g], kk & 31);
      V some = 0;
#pragma unroll
      for (int g = 0; g < N; ++g) some |= e[g];
      if (some) {  // the same in all lanes
        if (h0) {
#pragma unroll
          for (int g = 0; g < N; ++g) {
            const V t = f.mul(e[g], pv0);
            x0[g] = lane == kk ? t : f.sub(x0[g], t);
          }
        }
        if (h1) {
#pragma unroll
          for (int g = 0; g < N; ++g) {
            const V t = f.mul(e[g], pv1);
            x1[g] = lane + 32 == kk ? t : f.sub(x1[g], t);
          }
        }
#pragma unroll
        for (int g = 0; g < N; ++g) {
          if (R[g] && put0) R[g][lane] = x0[g];
          if (R[g] && put1) R[g][lane + 32] = x1[g];
        }
      }
      int first = INT_MAX;
#pragma unroll
      for (int g = N - 1; g >= 0; --g)
        if ((kn < 32 ? x0[g] : x1[g]) != 0) first = base + g * kWarps;
      next = min(next, first);
    };
    constexpr int kMost = std::is_same<F, FpBarrett>::value ? kG / 2 : kG;  // 8 rows of its chains spill
    for (int base = r + 1 + warp; base < n; base += kWarps * kMost) {
      if (base + kWarps * (kMost / 2) < n)
        rows(std::integral_constant<int, kMost>(), base);
      else if (base + kWarps * (kMost / 4) < n)
        rows(std::integral_constant<int, kMost / 2>(), base);
      else
        rows(std::integral_constant<int, kMost / 4>(), base);
    }
    next = __shfl_sync(0xffffffffu, next, kn & 31);
    if (lane == 0) S.red[warp] = next;
    __syncthreads();
    ++pb;
  }
  return pb;
}

// panel_rows: the pivot rows' U in place, by forward substitution per 64-column
// tile (src/fp.rs:181-200), and H for update_rest: the other rows' multipliers,
// negated, in the panel's first pb columns, zeros behind them (W is 64 here).
template <class F, class SM>
__device__ __noinline__ void panel_rows(const F& fr, uint64_t* __restrict__ m, const int n, int r0, int pb, int c0) {
  BatchSmem& S = SM::smem();
  const int* const perm = SM::perm();
  const F f = fr;
  constexpr int kT = SM::kT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  using A = Acc<F>;
  using AT = typename A::T;
  const uint64_t p = f.modulus();
  const uint64_t sb = A::batch(f);
  uint64_t(*LF)[kP + 1] = reinterpret_cast<uint64_t(*)[kP + 1]>(S.a);  // the pivot rows' multipliers F[k][k2]
  uint64_t(*Us)[kP] = reinterpret_cast<uint64_t(*)[kP]>(S.b);          // U block of one 64-column tile
  for (int idx = tid; idx < pb * pb; idx += kT) {
    const int k = idx / pb, k2 = idx - k * pb;
    LF[k][k2] = k2 < k ? m[(int64_t)perm[r0 + k] * n + S.pcol[k2]] : 0;
  }
  for (int ct = c0 + kP; ct < n; ct += kP) {
    for (int idx = tid; idx < pb * kP; idx += kT) {
      const int k = idx >> 6, ci = idx & 63;
      const int cc = ct + ci;
      Us[k][ci] = cc < n ? m[(int64_t)perm[r0 + k] * n + cc] : 0;
    }
    __syncthreads();
    {
      // U_k -= sum_{k2<k} F[k][k2] U_k2, kQ threads per column.
      constexpr int kQ = kT / kP;
      const int ci = tid / kQ, q = tid % kQ;
      for (int k = 1; k < pb; ++k) {
        AT acc = 0;
        uint64_t tot = 0, cnt = 0;
        for (int k2 = q; k2 < k; k2 += kQ) {
          acc += A::prod(f, LF[k][k2], Us[k2][ci]);
          if (++cnt >= sb) {
            tot = f.add(tot, A::reduce(f, acc));
            acc = 0;
            cnt = 0;
          }
        }
        uint64_t part = f.add(tot, A::reduce(f, acc));
#pragma unroll
        for (int o = 1; o < kQ; o <<= 1) part = f.add(part, __shfl_xor_sync(0xffffffffu, part, o));
        if (q == 0) Us[k][ci] = f.sub(Us[k][ci], part);
        __syncwarp();
      }
    }
    __syncthreads();
    for (int idx = tid; idx < pb * kP; idx += kT) {
      const int k = idx >> 6, cc = ct + (idx & 63);
      if (cc < n) m[(int64_t)perm[r0 + k] * n + cc] = Us[k][idx & 63];
    }
    __syncthreads();
  }
  for (int i = r0 + pb + warp; i < n; i += kT / 32) {  // a warp per row
    uint64_t* R = m + (int64_t)perm[i] * n;
    const uint64_t h0 = lane < pb ? R[S.pcol[lane]] : 0, h1 = lane + 32 < pb ? R[S.pcol[lane + 32]] : 0;
    __syncwarp();
    R[c0 + lane] = h0 ? p - h0 : 0;
    R[c0 + lane + 32] = h1 ? p - h1 : 0;
  }
}

}  // namespace

}  // namespace modlin
