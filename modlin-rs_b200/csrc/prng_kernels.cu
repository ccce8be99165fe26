// Device fill of the generators under test.
//
// MIXMAX (src/prng.rs:133-270, ROOT's MixMaxEngine) is linear over
// F_p, p = 2^61 - 1: one iteration maps the state (sumtot, v[1..N-1]) by a
// fixed N x N matrix, so the state any number of iterations ahead is a matrix
// power times the starting state (the host builds the matrix; powers come
// from m61_gemm). Each warp then runs one segment of the stream from its
// jump-ahead state. Within an iteration the two running sums of ROOT's loop
// (tp = v[1] + ... + v[i], tv = sumtot + tp_1 + ... + tp_i, plus the
// rotated-tp term when SPECIALMUL != 0) are two prefix scans over the state,
// 8 entries per lane and five shuffle steps across the warp.
//
// Bit parity with ROOT's arithmetic: ROOT folds each sum once
// (MOD_MERSENNE), which is exact mod p but can leave 2^61 - 1 where the
// canonical residue is 0, and that representation reaches the outputs
// (raw << 3). Every folded sum is below 3 * 2^61, so its result is at most
// 2^61 - 1 and equals it only when the sum is = 0 (mod p). Hence if no
// intermediate of an iteration (tp_i, tv_i, the special term, the corrected
// v[2]) is = 0 and no input entry is 2^61 - 1, ROOT's values are the
// canonical residues the scans compute; sumtot is ROOT's own formula on the
// exact 128-bit sum. Any other iteration is run by lane 0 exactly as ROOT
// runs it. A segment that ends on an entry 2^61 - 1 flags the next one, whose
// canonical jump-ahead start may then differ from ROOT's state in
// representation; the host reruns it from the flagged segment's exact end.
//
// xoroshiro128++ (src/prng.rs:48-83): the state transition T is linear over
// GF(2), and the matrices T^(2^k) are kept on the device; one thread per
// segment of 2^m outputs, each block of threads jumps to its segments itself,
// and outputs are staged 16 per thread in shared memory and written in rows.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "field.cuh"
#include "launch.cuh"
#include "mma_limbs.cuh"
#include "prng_kernels.cuh"

namespace modlin {

namespace {

constexpr uint64_t kP = kM61;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint64_t padd(uint64_t a, uint64_t b) {
  const uint64_t s = a + b;
  return s >= kP ? s - kP : s;
}
__device__ __forceinline__ uint64_t fold61(uint64_t k) { return (k & kP) + (k >> 61); }
__device__ __forceinline__ uint64_t rot61(uint64_t x, int s) { return ((x << s) & kP) | (x >> (61 - s)); }

// ---- reductions of outputs to the field ------------------------------------
struct RedRaw {
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const { return x; }
};
struct RedM61 {
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const {
    const uint64_t y = fold61(x);
    return y >= kP ? y - kP : y;
  }
};
struct RedBarrett {
  FpBarrett f;
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const { return f.reduce((u128)x); }
};
struct RedSmall {
  FpSmall f;
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const { return f.reduce64(x); }
};

// ---- C = A * B mod 2^61 - 1 ------------------------------------------------
// 64 x 32 output tiles, K in chunks of 64 as 8-bit limb products on the tensor
// cores (mma_limbs.cuh), each chunk's diagonals folded into one 64-bit sum. A
// state doubling of MIXMAX-256 (2048 x 256 x 256) takes 35 us (330 with
// 128-bit sums on the integer pipes).
constexpr int kGM = 64, kGN = 32, kGK = 64, kGStride = 80;
constexpr int kGemmSmem = 8 * (kGM + kGN) * kGStride;

__global__ void __launch_bounds__(256) m61_gemm_kernel(const uint64_t* __restrict__ A, const uint64_t* __restrict__ B,
                                                       uint64_t* __restrict__ C, int M, int K, int N) {
  extern __shared__ __align__(16) uint8_t gsm[];
  uint8_t *pa = gsm, *pb = gsm + 8 * kGM * kGStride;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.y * kGM, c0 = blockIdx.x * kGN;
  const int rg = warp & 3, cg0 = 2 * (warp >> 2);  // this warp's 16 rows and two groups of 8 columns
  uint64_t sum[2][4] = {};
  for (int k0 = 0; k0 < K; k0 += kGK) {
    uint64_t va[4][4], vb[2][4];
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + (tid >> 4) + 16 * w, k = k0 + 4 * (tid & 15) + u;
        va[w][u] = r < M && k < K ? A[(int64_t)r * K + k] : 0;
      }
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = c0 + lane, k = k0 + 4 * (warp + 8 * w) + u;
        vb[w][u] = c < N && k < K ? B[(int64_t)k * N + c] : 0;
      }
    __syncthreads();  // the previous chunk's planes have been read
#pragma unroll
    for (int w = 0; w < 4; ++w)
      mml::put_planes4<8>(pa + ((tid >> 4) + 16 * w) * kGStride + 4 * (tid & 15), kGM * kGStride, va[w]);
#pragma unroll
    for (int w = 0; w < 2; ++w)
      mml::put_planes4<8>(pb + lane * kGStride + 4 * (warp + 8 * w), kGN * kGStride, vb[w]);
    __syncthreads();
    if (r0 + 16 * rg < M) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t acc[15][4];
        mml::tile_k32<8, 2, kGStride>(acc, mml::saddr(pa) + 16 * rg * kGStride, kGM * kGStride,
                                      mml::saddr(pb) + 8 * (cg0 + q) * kGStride, kGN * kGStride);
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[q][e] = fold61(sum[q][e] + m61_fold15(acc, e));  // < 2^61 + 8
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = r0 + 16 * rg + (lane >> 2) + 8 * (e >> 1), c = c0 + 8 * (cg0 + q) + 2 * (lane & 3) + (e & 1);
      const uint64_t v = fold61(sum[q][e]);
      if (r < M && c < N) C[(int64_t)r * N + c] = v >= kP ? v - kP : v;
    }
}

// ---- MIXMAX ---------------------------------------------------------------------
template <int N>
struct MixTraits;
template <>
struct MixTraits<17> {  // TRandomMixMax17: SPECIALMUL 36, no special term, no skip
  static constexpr int E = 1, SM = 36, SKIP = 0, SK = 0;
};
template <>
struct MixTraits<240> {  // TRandomMixMax: SPECIALMUL 51, special * v[1], no skip
  static constexpr int E = 8, SM = 51, SKIP = 0, SK = 2;
};
template <>
struct MixTraits<256> {  // TRandomMixMax256: no SPECIALMUL, special -1, skip 2
  static constexpr int E = 8, SM = 0, SKIP = 2, SK = 1;
};

constexpr int kMixWarps = 4;

// Inclusive prefix sum mod p across the warp, returned exclusive.
__device__ __forceinline__ uint64_t warp_excl_scan(uint64_t v, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t y = __shfl_up_sync(kFull, v, off);
    if (lane >= off) v = padd(v, y);
  }
  const uint64_t ex = __shfl_up_sync(kFull, v, 1);
  return lane ? ex : 0;
}

// ROOT's iteration, run by one thread on the state s[0] = sumtot,
// s[1..N-1] = v[1..N-1] (src/prng.rs:191-222).
struct MixLinear {
  __device__ __forceinline__ int operator()(int e) const { return e; }
};
template <int N, class At = MixLinear>
__device__ void mix_iterate_exact(uint64_t* st, uint64_t special, At at = At()) {
  using T = MixTraits<N>;
  struct Ref {
    uint64_t* st;
    At at;
    __device__ uint64_t& operator[](int e) const { return st[at(e)]; }
  } s{st, at};
  const uint64_t temp2 = s[1];
  uint64_t tv = s[0], acc = tv, ovf = 0, tp = 0;
  for (int i = 1; i < N; ++i) {
    if (T::SM) {
      const uint64_t tpo = ((tp << T::SM) & kP) | (tp >> (61 - T::SM));
      tp = fold61(tp + s[i]);
      tv = fold61(tv + tp + tpo);
    } else {
      tp = fold61(tp + s[i]);
      tv = fold61(tv + tp);
    }
    s[i] = tv;
    const uint64_t t = acc + tv;
    ovf += t < acc;
    acc = t;
  }
  if (T::SK) {
    uint64_t t2;
    if (T::SK == 1) {
      t2 = kP - temp2;
    } else {
      const u128 m = (u128)special * temp2;
      const uint64_t lo = (uint64_t)m, hi = (uint64_t)(m >> 64);
      t2 = fold61((lo & kP) + hi * 8 + (lo >> 61));
    }
    s[2] = fold61(s[2] + t2);
    const uint64_t t = acc + t2;
    ovf += t < acc;
    acc = t;
  }
  s[0] = fold61(fold61(acc) + (ovf << 3));
}

// One iteration of the warp's state x (entry idx = lane * E + k).
template <int N>
__device__ __forceinline__ void mix_iterate(uint64_t (&x)[MixTraits<N>::E], uint64_t& v0, uint64_t* s, int lane,
                                            uint64_t special) {
  using T = MixTraits<N>;
  constexpr int E = T::E;
  bool bad = false;
#pragma unroll
  for (int k = 0; k < E; ++k) bad |= x[k] == kP;
  const uint64_t sum_old = __shfl_sync(kFull, x[0], 0);
  const uint64_t temp2 = __shfl_sync(kFull, x[1 % E], 1 / E);
  // tp_i = v[1] + ... + v[i]
  uint64_t tp[E];
  uint64_t run = 0;
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int idx = lane * E + k;
    run = padd(run, (idx >= 1 && idx < N) ? x[k] : 0);
    tp[k] = run;
  }
  const uint64_t ex1 = warp_excl_scan(run, lane);
  // u_0 = sumtot, u_i = tp_i (+ 2^SM tp_{i-1}); tv_i = u_0 + ... + u_i
  uint64_t tv[E];
  uint64_t prev = ex1;
  run = 0;
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int idx = lane * E + k;
    const uint64_t t = padd(tp[k], ex1);
    uint64_t u = 0;
    if (idx == 0) {
      u = sum_old;
    } else if (idx < N) {
      bad |= t == 0;
      u = T::SM ? padd(t, rot61(prev, T::SM)) : t;
    }
    prev = t;
    run = padd(run, u);
    tv[k] = run;
  }
  const uint64_t ex2 = warp_excl_scan(run, lane);
  uint64_t t2 = 0;
  if (T::SK == 1) {
    t2 = temp2 ? kP - temp2 : 0;
    bad |= temp2 == 0;
  } else if (T::SK == 2) {
    t2 = FpM61().mul(special, temp2);
    bad |= t2 == 0;
  }
  uint64_t lo = 0, hi = 0;
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int idx = lane * E + k;
    tv[k] = padd(tv[k], ex2);
    if (idx < N) {
      if (idx >= 1) bad |= tv[k] == 0;
      lo += tv[k];
      hi += lo < tv[k];
    }
  }
  if (lane == 0) {
    lo += t2;
    hi += lo < t2;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t olo = __shfl_xor_sync(kFull, lo, off), ohi = __shfl_xor_sync(kFull, hi, off);
    const uint64_t l2 = lo + olo;
    hi += ohi + (l2 < lo);
    lo = l2;
  }
  if (T::SK) {
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (lane * E + k == 2) {
        tv[k] = padd(tv[k], t2);
        bad |= tv[k] == 0;
      }
  }
  if (!__any_sync(kFull, bad)) {
    const uint64_t sumtot = fold61(fold61(lo) + (hi << 3));
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int idx = lane * E + k;
      x[k] = idx == 0 ? sumtot : (idx < N ? tv[k] : 0);
    }
  } else {
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (lane * E + k < N) s[lane * E + k] = x[k];
    __syncwarp();
    if (lane == 0) mix_iterate_exact<N>(s, special);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < E; ++k) x[k] = lane * E + k < N ? s[lane * E + k] : 0;
    __syncwarp();
  }
  v0 = sum_old;
}

// ---- MIXMAX-256: a block of three iterations in lazily reduced sums ---------
// No special multiplier here, so an iteration is two running sums and the
// correction of v[2] and sumtot. In 64 bits there is room for sums of four
// residues, and a third word takes the rest, so entries are reduced once per
// iteration and running sums not at all. Only the third iteration's entries
// are output: what ROOT leaves for a residue other than 0 does not depend on
// the representation of its inputs (a folded sum lies in [0, p]), so the only
// blocks to be run as ROOT runs them are those with an output entry, or a
// sumtot, that is 0 mod p. Integer ALU bound: 2^28 outputs in 1715 us (3017
// with every sum reduced and checked), 82 % of the ALU pipe.
struct U96 {  // w2 2^64 + w1 2^32 + w0
  uint32_t w0, w1, w2;
  __device__ __forceinline__ void add(uint64_t v) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
        : "+r"(w0), "+r"(w1), "+r"(w2)
        : "r"((uint32_t)v), "r"((uint32_t)(v >> 32)));
  }
  __device__ __forceinline__ void add(const U96& v) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(w0), "+r"(w1), "+r"(w2)
        : "r"(v.w0), "r"(v.w1), "r"(v.w2));
  }
  // Congruent mod p and below 2^61 + 8 (w2 + 1).
  __device__ __forceinline__ uint64_t fold() const {
    return ((uint64_t)(w1 & 0x1fffffffu) << 32 | w0) + __funnelshift_l(w1, w2, 3);
  }
};
__device__ __forceinline__ U96 u96(uint64_t v) { return U96{(uint32_t)v, (uint32_t)(v >> 32), 0}; }
// y < 2^62: the canonical residue.
__device__ __forceinline__ uint64_t canon(uint64_t y) { return (y + ((y + 1) >> 61)) & kP; }

// Exclusive sum across the warp of values below 2^61 + 2^8, congruent mod p
// and below 2^61 + 8.
__device__ __forceinline__ uint64_t lazy_excl_scan(uint64_t v, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t y = __shfl_up_sync(kFull, v, off);
    if (lane >= off) v += y;
    if (off == 2 || off == 8) v = fold61(v);  // sums of four so far, below 2^63 + 2^10
  }
  const uint64_t ex = __shfl_up_sync(kFull, v, 1);
  return lane ? fold61(ex) : 0;
}

// One iteration on x (entry lane * 8 + k, below 2^61 + 2^8); kLast: canonical
// results. zero: an entry or sumtot may be 0 mod p (sumtot in every iteration).
template <bool kLast>
__device__ __forceinline__ void mix256_iterate(uint64_t (&x)[8], uint64_t& v0, int lane, bool& zero) {
  const uint64_t sum_old = __shfl_sync(kFull, x[0], 0);
  const uint64_t temp2 = __shfl_sync(kFull, x[1], 0);
  if (lane == 0) x[0] = 0;  // entry 0 is sumtot, not part of tp
  // Lane totals: tp of the last entry, and the sum of the tp.
  U96 tp = u96(x[0]), T = tp;
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    tp.add(x[k]);
    T.add(tp);
  }
  const uint64_t ex1 = lazy_excl_scan(tp.fold(), lane);
  if (lane == 0) T.add(sum_old);
  T.add(ex1 << 2);  // 8 ex1 in two parts below 2^64
  T.add(ex1 << 2);
  const uint64_t ex2 = lazy_excl_scan(T.fold(), lane);
  // tv: running sum of ex1 + tp from ex2.
  U96 t = u96(ex1), r = u96(ex2);
  uint64_t sum = 0;
  U96 wide = u96(0);
  uint32_t low = 0xffffffffu;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    t.add(x[k]);
    r.add(t);
    if (k == 0 && lane == 0) r.add(sum_old);
    uint64_t y = r.fold();
    if (k == 2 && lane == 0) y = fold61(y + 4 * kP - temp2);  // special = -1: v[2] -= the old v[1]
    if (kLast) {
      y = canon(y);
      if (k > 0 || lane > 0) low = min(low, (uint32_t)y);
      sum += y;  // 8 (p - 1) < 2^64
    } else {
      wide.add(y);
    }
    x[k] = y;
  }
  uint64_t tot = kLast ? fold61(sum) : wide.fold();
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    tot += __shfl_xor_sync(kFull, tot, off);
    if (off == 2 || off == 8) tot = fold61(tot);
  }
  tot = canon(fold61(tot));
  zero |= tot == 0 || (kLast && low == 0);  // low words: 2^-32 a false alarm
  if (lane == 0) x[0] = tot;
  v0 = sum_old;
}

// Entry e of a warp's state in shared memory: the 8 entries of a lane rotate
// with it, so that lanes writing their k-th entries meet in few banks.
struct MixSwizzle {
  __device__ __forceinline__ int operator()(int e) const { return (e & ~7) | ((e ^ (e >> 3)) & 7); }
};

// The segment loop. kFast (MIXMAX-256): blocks by mix256_iterate, s holding
// the state at the block's start for the exact run.
template <int N, class R>
__global__ void __launch_bounds__(kMixWarps * 32) mixmax_fill_kernel(MixFill a, R red) {
  using T = MixTraits<N>;
  constexpr int E = T::E;
  constexpr bool kFast = N == 256;
  static_assert(!kFast || (T::SM == 0 && T::SK == 1 && E == 8), "mix256_iterate");
  using At = typename std::conditional<kFast, MixSwizzle, MixLinear>::type;
  const At at;
  __shared__ uint64_t sh[kMixWarps][N];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t seg = a.seg_begin + (int64_t)blockIdx.x * kMixWarps + w;
  if (seg >= a.seg_end) return;
  uint64_t* s = sh[w];
  uint64_t x[E];
  const uint64_t* st = a.starts + seg * N;
  const auto put = [&]() {
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (lane * E + k < N) s[at(lane * E + k)] = x[k];
    __syncwarp();
  };
#pragma unroll
  for (int k = 0; k < E; ++k) x[k] = lane * E + k < N ? st[lane * E + k] : 0;
  uint64_t v0 = 0;
  if (kFast || (seg == 0 && a.h0 > 0)) put();
  if (seg == 0 && a.h0 > 0) {  // the rest of the starting block
    for (int64_t j = lane; j < a.h0; j += 32) a.out[j] = red(s[at((int)(a.c0 + j))] << 3);
    __syncwarp();
  }
  const int64_t b0 = seg * a.G + 1, b1 = (seg + 1) * a.G < a.nbk ? (seg + 1) * a.G : a.nbk;
  for (int64_t b = b0; b <= b1; ++b) {
    if constexpr (kFast) {
      bool zero = false;
#pragma unroll 1
      for (int it = 0; it < T::SKIP; ++it) mix256_iterate<false>(x, v0, lane, zero);
      mix256_iterate<true>(x, v0, lane, zero);
      if (__any_sync(kFull, zero)) {
        uint64_t v = 0;
        if (lane == 0)
          for (int it = 0; it <= T::SKIP; ++it) {
            v = s[at(0)];
            mix_iterate_exact<N>(s, a.special, at);
          }
        v0 = __shfl_sync(kFull, v, 0);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < E; ++k) x[k] = s[at(lane * E + k)];
        __syncwarp();
      }
    } else {
#pragma unroll 1
      for (int it = 0; it <= T::SKIP; ++it) mix_iterate<N>(x, v0, s, lane, a.special);
    }
    put();
    const int64_t base = a.h0 + (b - 1) * (N - 1) - 1;  // output index of v[e] is base + e
    if (base + N <= a.count) {
#pragma unroll
      for (int e0 = 0; e0 < N; e0 += 32) {
        const int e = e0 + lane;
        if (e >= 1 && e < N) a.out[base + e] = red(s[at(e)] << 3);
      }
    } else {
      for (int e = lane; e < N; e += 32)
        if (e >= 1 && base + e < a.count) a.out[base + e] = red(s[at(e)] << 3);
    }
    __syncwarp();
  }
  uint64_t* en = a.ends + seg * (N + 1);
  bool kmp = false;
#pragma unroll
  for (int k = 0; k < E; ++k)
    if (lane * E + k < N) {
      en[lane * E + k] = x[k];
      kmp |= x[k] == kP;
    }
  if (lane == 0) en[N] = v0;
  if (__any_sync(kFull, kmp) && lane == 0 && seg + 1 < a.S) {
    a.flags[seg + 1] = 1;
    atomicAdd(a.any, 1);
  }
}

template <int N, class R>
cudaError_t launch_mix(const MixFill& a, R red, cudaStream_t st) {
  const int64_t segs = a.seg_end - a.seg_begin;
  if (segs <= 0) return cudaSuccess;
  const int64_t blocks = (segs + kMixWarps - 1) / kMixWarps;
  mixmax_fill_kernel<N, R><<<(unsigned)blocks, kMixWarps * 32, 0, st>>>(a, red);
  return cudaGetLastError();
}

template <int N>
cudaError_t mix_dispatch(const MixFill& a, uint64_t p, const FieldParams& fp, cudaStream_t st) {
  if (p == 0) return launch_mix<N>(a, RedRaw{}, st);
  if (p == kM61) return launch_mix<N>(a, RedM61{}, st);
  if (p < (1ULL << 32)) return launch_mix<N>(a, RedSmall{FpSmall(fp)}, st);
  return launch_mix<N>(a, RedBarrett{FpBarrett(fp)}, st);
}

// ---- xoroshiro128++ ----------------------------------------------------------------
constexpr int kXoroThreads = 128;
constexpr int kXoroRow = 16;              // outputs staged per thread: 128-byte rows
constexpr int kXoroStride = kXoroRow + 2;  // 16-byte aligned rows, conflict-free 16-byte accesses

__device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }

// acc ^= column j of a GF(2) matrix for every set bit j of the 32-bit word w.
__device__ __forceinline__ void gf2_word(uint4& acc, uint32_t w, const uint4* col) {
#pragma unroll 8
  for (int j = 0; j < 32; ++j) {
    const uint32_t m = 0u - ((w >> j) & 1u);
    const uint4 c = col[j];
    acc.x ^= c.x & m;
    acc.y ^= c.y & m;
    acc.z ^= c.z & m;
    acc.w ^= c.w & m;
  }
}

// Thread t runs segment t. Its state is T^(2^m t) times the starting state:
// warp 0 applies the matrices of the bits of the block's first segment (a
// lane holds 4 of the 128 columns), then 7 doublings fill the block's 128
// states (about 4 % of the work of 2^11-output segments). The fill itself is
// bound by instruction issue, about 30 an output: 2^28 outputs mod 2^61 - 1
// take 490 us (the segments' states came from the host before: 19400).
template <class R>
__global__ void __launch_bounds__(kXoroThreads) xoro_fill_kernel(XoroFill a, R red) {
  __shared__ __align__(16) uint64_t sh[kXoroThreads / 32][32 * kXoroStride];
  __shared__ uint4 mat[128];
  __shared__ uint4 state[kXoroThreads];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t first = (int64_t)blockIdx.x * kXoroThreads, t = first + tid, t0 = t - lane;
  const uint4* mats = reinterpret_cast<const uint4*>(a.mats);  // T^(2^k) at 128 k, by columns
  if (w == 0) {
    uint4 v = make_uint4((uint32_t)a.s0, (uint32_t)(a.s0 >> 32), (uint32_t)a.s1, (uint32_t)(a.s1 >> 32));
    for (int k = 7; first >> k; ++k) {
      if (!((first >> k) & 1)) continue;
      const uint4* col = mats + 128 * (a.m + k) + 4 * lane;
      const uint32_t word = lane < 8 ? v.x : lane < 16 ? v.y : lane < 24 ? v.z : v.w;
      uint4 acc = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t mk = 0u - ((word >> (4 * (lane & 7) + j)) & 1u);
        const uint4 c = col[j];
        acc.x ^= c.x & mk;
        acc.y ^= c.y & mk;
        acc.z ^= c.z & mk;
        acc.w ^= c.w & mk;
      }
      v = make_uint4(__reduce_xor_sync(kFull, acc.x), __reduce_xor_sync(kFull, acc.y),
                     __reduce_xor_sync(kFull, acc.z), __reduce_xor_sync(kFull, acc.w));
    }
    if (lane == 0) state[0] = v;
  }
  const int64_t segs = a.S - first;  // of this block (at least one)
  for (int have = 1, k = 0; have < kXoroThreads && have < segs; have *= 2, ++k) {
    __syncthreads();
    mat[tid] = mats[128 * (a.m + k) + tid];
    __syncthreads();
    if (tid < have) {
      const uint4 v = state[tid];
      uint4 acc = make_uint4(0, 0, 0, 0);
      gf2_word(acc, v.x, mat);
      gf2_word(acc, v.y, mat + 32);
      gf2_word(acc, v.z, mat + 64);
      gf2_word(acc, v.w, mat + 96);
      state[have + tid] = acc;
    }
  }
  __syncthreads();
  if (t0 >= a.S) return;
  const bool act = t < a.S;
  const uint4 v = state[tid];  // of a segment past the last: unused
  uint64_t s0 = (uint64_t)v.y << 32 | v.x, s1 = (uint64_t)v.w << 32 | v.z;
  const int64_t L = (int64_t)1 << a.m;
  const int64_t beg = t << a.m, cnt = act ? ((a.count - beg) < L ? (a.count - beg) : L) : 0;
  uint64_t* row = sh[w] + lane * kXoroStride;
  const auto next = [&]() {  // src/prng.rs:75-83
    const uint64_t r = rotl64(s0 + s1, 17) + s0;
    const uint64_t b = s1 ^ s0;
    s0 = rotl64(s0, 49) ^ b ^ (b << 21);
    s1 = rotl64(b, 28);
    return red(r);
  };
  // The warp's rows are all full when its last segment is.
  const bool full = t0 + 31 < a.S && ((t0 + 32) << a.m) <= a.count && ((uintptr_t)a.out & 15) == 0;
  for (int64_t c = 0; c < L; c += kXoroRow) {
    if (full) {
#pragma unroll
      for (int i = 0; i < kXoroRow; i += 2) {
        const uint64_t r0 = next(), r1 = next();
        *reinterpret_cast<ulonglong2*>(row + i) = make_ulonglong2(r0, r1);
      }
      __syncwarp();
      // 8 lanes write a row's 128 bytes.
      uint64_t* dst = a.out + ((t0 + (lane >> 3)) << a.m) + c + 2 * (lane & 7);
      const uint64_t* src = sh[w] + (lane >> 3) * kXoroStride + 2 * (lane & 7);
#pragma unroll
      for (int r = 0; r < 32; r += 4)
        *reinterpret_cast<ulonglong2*>(dst + ((int64_t)r << a.m)) =
            *reinterpret_cast<const ulonglong2*>(src + r * kXoroStride);
      __syncwarp();
    } else {
      for (int i = 0; i < kXoroRow; ++i)
        if (c + i < cnt) row[i] = next();
      __syncwarp();
      for (int r = lane >> 4; r < 32; r += 2) {
        const int64_t rb = ((t0 + r) << a.m) + c + (lane & 15);
        if (t0 + r < a.S && rb < a.count) a.out[rb] = sh[w][r * kXoroStride + (lane & 15)];
      }
      __syncwarp();
    }
  }
  if (t == a.S - 1) {
    a.ends[0] = s0;
    a.ends[1] = s1;
  }
}

template <class R>
cudaError_t launch_xoro(const XoroFill& a, R red, cudaStream_t st) {
  if (a.S <= 0) return cudaSuccess;
  xoro_fill_kernel<R><<<(unsigned)((a.S + kXoroThreads - 1) / kXoroThreads), kXoroThreads, 0, st>>>(a, red);
  return cudaGetLastError();
}

}  // namespace

cudaError_t m61_gemm(const uint64_t* A, const uint64_t* B, uint64_t* C, int M, int K, int N, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  static PerDevice once;
  const cudaError_t attr = allow_smem(once, m61_gemm_kernel, kGemmSmem);
  if (attr != cudaSuccess) return attr;
  const dim3 grid((N + kGN - 1) / kGN, (M + kGM - 1) / kGM);
  m61_gemm_kernel<<<grid, 256, kGemmSmem, st>>>(A, B, C, M, K, N);
  return cudaGetLastError();
}

cudaError_t mixmax_fill(const MixFill& a, uint64_t p, const FieldParams& fp, cudaStream_t st) {
  switch (a.N) {
    case 17: return mix_dispatch<17>(a, p, fp, st);
    case 240: return mix_dispatch<240>(a, p, fp, st);
    case 256: return mix_dispatch<256>(a, p, fp, st);
    default: return cudaErrorInvalidValue;
  }
}

int mixmax_resident_warps(int N, int num_sms) {
  int per_sm = 0;
  cudaError_t e = cudaErrorInvalidValue;
  if (N == 17) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mixmax_fill_kernel<17, RedM61>, kMixWarps * 32, 0);
  if (N == 240) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mixmax_fill_kernel<240, RedM61>, kMixWarps * 32, 0);
  if (N == 256) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mixmax_fill_kernel<256, RedM61>, kMixWarps * 32, 0);
  if (e != cudaSuccess || per_sm < 1) per_sm = 1;
  return per_sm * kMixWarps * num_sms;
}

cudaError_t xoro_fill(const XoroFill& a, uint64_t p, const FieldParams& fp, cudaStream_t st) {
  if (p == 0) return launch_xoro(a, RedRaw{}, st);
  if (p == kM61) return launch_xoro(a, RedM61{}, st);
  if (p < (1ULL << 32)) return launch_xoro(a, RedSmall{FpSmall(fp)}, st);
  return launch_xoro(a, RedBarrett{FpBarrett(fp)}, st);
}

}  // namespace modlin

// ---------------------------------------------------------------------------
// Host side: jump-ahead states, launches, the boundary repair, write-back.
// ---------------------------------------------------------------------------
#include <algorithm>
#include <vector>

#include "../host/prng.h"

namespace modlin {

namespace {

constexpr int kPowMax = 64;

uint64_t hmul(uint64_t a, uint64_t b) { return (uint64_t)(((u128)a * b) % kM61); }
uint64_t hadd(uint64_t a, uint64_t b) { return (a + b) % kM61; }

// One MIXMAX iteration as the linear map it is over F_p (canonical
// residues): the state x = [sumtot, v[1..N-1]] (src/prng.rs:191-222).
void mix_linear_step(const modlin_prng_impl::MixMax& m, const uint64_t* x, uint64_t* y) {
  const int N = m.N;
  const uint64_t sum_old = x[0], temp2 = x[1];
  const uint64_t two_sm = m.specialmul ? (1ULL << m.specialmul) % kM61 : 0;
  uint64_t tp = 0, tv = sum_old, tot = sum_old;
  for (int i = 1; i < N; ++i) {
    const uint64_t tpo = m.specialmul ? hmul(tp, two_sm) : 0;
    tp = hadd(tp, x[i]);
    tv = hadd(hadd(tv, tp), tpo);
    y[i] = tv;
    tot = hadd(tot, tv);
  }
  if (m.special) {
    const uint64_t t2 = m.special == UINT64_MAX ? (kM61 - temp2) % kM61 : hmul(m.special % kM61, temp2);
    y[2] = hadd(y[2], t2);
    tot = hadd(tot, t2);
  }
  y[0] = tot;
}

int kind_slot(int N) { return N == 17 ? 0 : N == 240 ? 1 : 2; }

#define PCK(x)                                                        \
  do {                                                                \
    cudaError_t e_ = (x);                                             \
    if (e_ != cudaSuccess) {                                          \
      cudaGetLastError();                                             \
      return e_ == cudaErrorMemoryAllocation ? MODLIN_ENOMEM : MODLIN_ECUDA; \
    }                                                                 \
  } while (0)

int ensure_ws(PrngCache& c, size_t bytes) {
  if (bytes <= c.ws_bytes) return MODLIN_OK;
  if (c.ws) cudaFree(c.ws);
  c.ws = nullptr;
  c.ws_bytes = 0;
  PCK(cudaMalloc(&c.ws, bytes));
  c.ws_bytes = bytes;
  return MODLIN_OK;
}

// B^(2^k) for k <= kmax in the cache (B built on the host, squared here).
int ensure_pows(PrngCache& c, const modlin_prng_impl::MixMax& m, int kmax, cudaStream_t st, uint64_t* launches) {
  const int slot = kind_slot(m.N), N = m.N;
  const size_t mat = (size_t)N * N;
  if (!c.pow[slot]) {
    PCK(cudaMalloc(&c.pow[slot], mat * kPowMax * sizeof(uint64_t)));
    std::vector<uint64_t> Q(mat), x(N), y(N);
    for (int j = 0; j < N; ++j) {  // row j = B e_j
      std::fill(x.begin(), x.end(), 0);
      x[j] = 1;
      for (int it = 0; it <= m.skip; ++it) {
        mix_linear_step(m, x.data(), y.data());
        x.swap(y);
      }
      std::copy(x.begin(), x.end(), Q.begin() + (size_t)j * N);
    }
    PCK(cudaMemcpyAsync(c.pow[slot], Q.data(), mat * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    PCK(cudaStreamSynchronize(st));
    c.have[slot] = 1;
  }
  for (int k = c.have[slot]; k <= kmax; ++k) {
    const uint64_t* P = c.pow[slot] + (size_t)(k - 1) * mat;
    PCK(m61_gemm(P, P, c.pow[slot] + (size_t)k * mat, N, N, N, st));
    ++*launches;
    c.have[slot] = k + 1;
  }
  return MODLIN_OK;
}

int mix_fill(PrngCache& c, int num_sms, modlin_prng_impl::MixMax& m, uint64_t p, const FieldParams& fp,
             uint64_t* d_out, uint64_t count, cudaStream_t st, uint64_t* launches) {
  const int N = m.N;
  const size_t mat = (size_t)N * N;
  const int64_t c0 = m.counter;
  const int64_t h0 = c0 < N ? std::min<int64_t>(N - c0, (int64_t)count) : 0;
  const int64_t rest = (int64_t)count - h0;
  const int64_t nbk = rest > 0 ? (rest + N - 2) / (N - 1) : 0;
  int64_t S = 1, G = 1;
  int bits = 0;
  if (nbk > 0) {
    // Segments of 2^bits blocks, so that every jump between them is a cached
    // power: the longest that leave three quarters of the resident warps busy
    // (the kernel is bound by the ALUs, not by the warps in flight).
    const int64_t R = mixmax_resident_warps(N, num_sms);
    while (bits < 40 && ((nbk + ((int64_t)2 << bits) - 1) >> (bits + 1)) >= R * 3 / 4) ++bits;
    G = (int64_t)1 << bits;
    S = (nbk + G - 1) / G;
  }
  // workspace: starts S x N | ends S x (N+1) | flags S + 1 ints
  const size_t o_ends = (size_t)S * N, o_flags = o_ends + (size_t)S * (N + 1);
  int rc = ensure_ws(c, (o_flags + 1) * sizeof(uint64_t) + (size_t)(S + 1) * sizeof(int));
  if (rc) return rc;
  uint64_t* ws = static_cast<uint64_t*>(c.ws);
  uint64_t *starts = ws, *ends = ws + o_ends;
  int* flags = reinterpret_cast<int*>(ws + o_flags);
  int* any = flags + S;

  // The exact host state; its canonical form seeds the jump-ahead.
  std::vector<uint64_t> x0(N);
  x0[0] = m.sumtot;
  for (int i = 1; i < N; ++i) x0[i] = m.v[i];
  if (S > 1) {
    int top = bits;
    while (((int64_t)1 << (top - bits + 1)) < S) ++top;  // B^(2^bits) .. B^(2^top)
    rc = ensure_pows(c, m, top, st, launches);
    if (rc) return rc;
    std::vector<uint64_t> xc(x0);
    for (auto& v : xc) v %= kM61;
    PCK(cudaMemcpyAsync(starts, xc.data(), N * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    // Doubling: states [have, 2 have) = states [0, have) * B^(G have).
    int k = bits;
    for (int64_t have = 1; have < S; ++k) {
      const int64_t w = std::min(have, S - have);
      PCK(m61_gemm(starts, c.pow[kind_slot(N)] + (size_t)k * mat, starts + (size_t)have * N, (int)w, N, N, st));
      ++*launches;
      have += w;
    }
  }
  PCK(cudaMemcpyAsync(starts, x0.data(), N * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
  PCK(cudaMemsetAsync(flags, 0, (size_t)(S + 1) * sizeof(int), st));
  MixFill a{};
  a.N = N;
  a.special = m.special == UINT64_MAX ? 0 : m.special;
  a.starts = starts;
  a.ends = ends;
  a.flags = flags;
  a.any = any;
  a.out = d_out;
  a.count = (int64_t)count;
  a.h0 = h0;
  a.nbk = nbk;
  a.G = G;
  a.S = S;
  a.c0 = (int)c0;
  a.seg_begin = 0;
  a.seg_end = S;
  PCK(mixmax_fill(a, p, fp, st));
  ++*launches;
  int h_any = 0;
  PCK(cudaMemcpyAsync(&h_any, any, sizeof(int), cudaMemcpyDeviceToHost, st));
  PCK(cudaStreamSynchronize(st));
  if (h_any) {
    // A segment ended on an entry 2^61 - 1: rerun the next one from that
    // exact end (its canonical start differs in representation), in order.
    std::vector<int> hf(S);
    PCK(cudaMemcpyAsync(hf.data(), flags, S * sizeof(int), cudaMemcpyDeviceToHost, st));
    PCK(cudaStreamSynchronize(st));
    for (int64_t s = 1; s < S; ++s) {
      if (!hf[s]) continue;
      PCK(cudaMemcpyAsync(starts + (size_t)s * N, ends + (size_t)(s - 1) * (N + 1), N * sizeof(uint64_t),
                          cudaMemcpyDeviceToDevice, st));
      if (s + 1 < S) PCK(cudaMemsetAsync(flags + s + 1, 0, sizeof(int), st));
      a.seg_begin = s;
      a.seg_end = s + 1;
      PCK(mixmax_fill(a, p, fp, st));
      ++*launches;
      if (s + 1 < S) {
        PCK(cudaMemcpyAsync(&hf[s + 1], flags + s + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        PCK(cudaStreamSynchronize(st));
      }
    }
  }
  if (nbk == 0) {
    PCK(cudaStreamSynchronize(st));
    m.counter = (int)(c0 + (int64_t)count);
    return MODLIN_OK;
  }
  std::vector<uint64_t> e(N + 1);
  PCK(cudaMemcpyAsync(e.data(), ends + (size_t)(S - 1) * (N + 1), (N + 1) * sizeof(uint64_t),
                      cudaMemcpyDeviceToHost, st));
  PCK(cudaStreamSynchronize(st));
  m.sumtot = e[0];
  for (int i = 1; i < N; ++i) m.v[i] = e[i];
  m.v[0] = e[N];
  m.counter = (int)((rest - 1) % (N - 1) + 2);  // one past the last element output
  return MODLIN_OK;
}

// GF(2) 128 x 128 matrices over the xoroshiro state (s0 = bits 0..63,
// s1 = bits 64..127), stored by columns.
struct V128 {
  uint64_t lo, hi;
};
struct M128 {
  V128 col[128];
};

V128 gf2_apply(const M128& A, V128 v) {
  V128 r{0, 0};
  for (int j = 0; j < 64; ++j)
    if ((v.lo >> j) & 1) {
      r.lo ^= A.col[j].lo;
      r.hi ^= A.col[j].hi;
    }
  for (int j = 0; j < 64; ++j)
    if ((v.hi >> j) & 1) {
      r.lo ^= A.col[64 + j].lo;
      r.hi ^= A.col[64 + j].hi;
    }
  return r;
}
void gf2_mul(const M128& A, const M128& B, M128* C) {  // C = A B
  for (int j = 0; j < 128; ++j) C->col[j] = gf2_apply(A, B.col[j]);
}

// The matrices T^(2^k), k < kXoroPows, on the device (built once per device).
constexpr int kXoroPows = 48;

int ensure_xoro_pows(PrngCache& c, cudaStream_t st) {
  if (c.xoro) return MODLIN_OK;
  std::vector<M128> P(kXoroPows);
  for (int j = 0; j < 128; ++j) {
    modlin_prng_impl::Xoroshiro u;
    u.s0 = j < 64 ? 1ULL << j : 0;
    u.s1 = j < 64 ? 0 : 1ULL << (j - 64);
    u.step();
    P[0].col[j] = V128{u.s0, u.s1};
  }
  for (int k = 1; k < kXoroPows; ++k) gf2_mul(P[k - 1], P[k - 1], &P[k]);
  uint64_t* d = nullptr;
  PCK(cudaMalloc(&d, kXoroPows * sizeof(M128)));
  cudaError_t e = cudaMemcpyAsync(d, P.data(), kXoroPows * sizeof(M128), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(d);
    cudaGetLastError();
    return MODLIN_ECUDA;
  }
  c.xoro = d;
  return MODLIN_OK;
}

int xoro_fill_host(PrngCache& c, int num_sms, modlin_prng_impl::Xoroshiro& x, uint64_t p, const FieldParams& fp,
                   uint64_t* d_out, uint64_t count, cudaStream_t st, uint64_t* launches) {
  // Segments of a power of two of outputs (their jumps are single cached
  // matrices): the longest that leave 512 threads an SM, at least 64.
  int m = 6;
  while (m < 30 && ((int64_t)count >> (m + 1)) >= (int64_t)num_sms * 512) ++m;
  const int64_t S = ((int64_t)count + ((int64_t)1 << m) - 1) >> m;
  if (m + 1 + (64 - __builtin_clzll((uint64_t)S)) > kXoroPows) return MODLIN_EINVAL_N;  // 2^47 outputs
  int rc = ensure_xoro_pows(c, st);
  if (rc) return rc;
  rc = ensure_ws(c, 2 * sizeof(uint64_t));
  if (rc) return rc;
  uint64_t* ends = static_cast<uint64_t*>(c.ws);
  const XoroFill a{c.xoro, ends, d_out, (int64_t)count, S, x.s0, x.s1, m};
  PCK(xoro_fill(a, p, fp, st));
  ++*launches;
  uint64_t e[2];
  PCK(cudaMemcpyAsync(e, ends, sizeof(e), cudaMemcpyDeviceToHost, st));
  PCK(cudaStreamSynchronize(st));
  x.s0 = e[0];
  x.s1 = e[1];
  return MODLIN_OK;
}

}  // namespace

int prng_fill_device(PrngCache& c, int num_sms, modlin_prng* g, uint64_t p, const FieldParams& fp, uint64_t* d_out,
                     uint64_t count, cudaStream_t st, uint64_t* launches) {
  if (!count) return MODLIN_OK;
  if (g->xo) return xoro_fill_host(c, num_sms, *g->xo, p, fp, d_out, count, st, launches);
  if (g->mm) return mix_fill(c, num_sms, *g->mm, p, fp, d_out, count, st, launches);
  return MODLIN_EINVAL_ARG;
}

}  // namespace modlin
