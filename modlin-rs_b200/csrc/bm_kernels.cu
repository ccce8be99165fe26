// Linear complexity over F_p on the GPU (the value of src/fp.rs:257-308).
//
// The reference runs Berlekamp-Massey: at step i the discrepancy of the
// connection polynomial c, d = s[i] + sum_j c[j] s[i-j], is the coefficient of
// x^i in c(x) s(x), and c is updated by c -= (d/bb) x^m b
// (src/fp.rs:272-306). Only the complexity l leaves the function, and l
// depends on the discrepancies alone, so the kernels keep the two products
// A = x^-i c s and B = x^-i x^m b s instead of c and b: the residual form of
// the same recurrence (the extended Euclidean algorithm on s). With d = A[0]
// and bb = B[0], a step is
//     d == 0:              A <- A >> 1
//     d != 0:              A <- (bb A - d B) >> 1,
//     and if 2 l <= i:     B <- the old A, bb <- d, l <- i + 1 - l.
// Every A is a nonzero multiple of the reference's product, so d vanishes at
// the same steps and l evolves identically. There is no dot product and hence
// no reduction across threads in a step, no inverse, and once A is all zero
// no later step can change l: a recurrence of order L ends after 2 L steps.
//
// Steps are taken kBmK = 32 at a time. Which updates happen in 32 steps
// depends on the first 32 entries of A and B only, so one warp runs them on
// that window (bm_base), collecting the 2 x 2 polynomial matrix
//     A' = P A + Q B,  B' = U A + V B   (degree <= 32, about 16 as a rule)
// which the other threads then apply to the rest of A and B (bm_tile): 2 x 2
// products per entry and coefficient, about 2 per entry and step, summed
// without reduction and reduced once per 32 steps.
//
// Kernels:
//  * bm_block_kernel / bm_batch_kernel — one CTA per sequence, A and B in its
//    shared memory: warp 0 computes the next window first and runs the next 32
//    steps while the other warps apply the previous matrix. The batch form
//    pulls sequences (longest first) from a device counter.
//  * bm_long_kernel — one sequence on many CTAs: CTA 0 runs the steps on the
//    front of A and B and publishes the matrices; the others keep slices of A
//    and B in shared memory and apply them.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "bm_kernels.cuh"
#include "field.cuh"

namespace modlin {

namespace {

constexpr int kBmK = 32;          // steps per block, window entries
constexpr int kCoefRows = kBmK + 1;  // offsets 0 .. 32
constexpr int kBmPad = 2 * kBmK;  // entries past the end that a window may read
constexpr unsigned kAll = 0xffffffffu;

// ---------------------------------------------------------------------------
// Field policies. R: a canonical residue. S: what the arrays and matrices
// hold; pack(R). W: what bm_base works on; load(S), store(W) -> S.
// comb = (bb a + nd b) / r mod p on W, nd = neg(d). Dot: a sum of up to
// 2 * kCoefRows = 66 products of S, reduced once by value(), / r^2. r = 1, or
// the Montgomery radix 2^32 or 2^64: a common factor of all of A (or of all of
// B) changes no zero and so no complexity, and Montgomery's reduction is a
// third of Barrett's dependent chain. A Dot that can overflow is folded every
// kFold offsets (two products each), and after kFoldHigh of those again.
// ---------------------------------------------------------------------------

// p = 2^61 - 1. S and W are two 31-bit halves (M61Halves); S is balanced (|lo|
// <= 2^30, |hi| <= 2^29 + 1), so that a Dot takes more products.
struct BmM61 : M61Halves {
  using S = uint64_t;
  using R = uint64_t;
  __device__ explicit BmM61(const FieldParams&) {}
  __device__ __forceinline__ S pack(R x) const {
    const int64_t y = (int64_t)x - (x >= (1ULL << 60) ? (int64_t)kM61 : 0);  // in [-2^60, 2^60]
    const int32_t l = (int32_t)((uint32_t)y << 1) >> 1;
    return words(l, (int32_t)((y - l) >> 31));
  }
  __device__ __forceinline__ W load(S x) const {
    int64_t v = ((int64_t)hi(x) << 31) + lo(x);
    if (v < 0) v += (int64_t)kM61;
    return split((uint64_t)v);
  }
  __device__ __forceinline__ S store(W x) const { return pack(M61Halves::value(x)); }
  __device__ __forceinline__ R add(R a, R b) const {
    const uint64_t s = a + b;
    return s >= kM61 ? s - kM61 : s;
  }
  // Three offsets: |ll| <= 6 * 2^60, |mid| <= 12 * 2^59 (1 + 2^-28), then fold
  // moves ll's high part into mid and mid's into hh. Nine offsets: |hh| <=
  // 18 * 2^58 + 2^61, then fold_high takes it mod p below 2^61 + 4.
  struct Dot {
    int64_t ll = 0, mid = 0, hh = 0;
    __device__ __forceinline__ void mac(S a, S b) {
      ll = mad(lo(a), lo(b), ll);
      mid = mad(lo(a), hi(b), mid);
      hh = mad(hi(a), hi(b), hh);
      mid = mad(hi(a), lo(b), mid);
    }
  };
  static constexpr int kFold = 3, kFoldHigh = 3;
  __device__ __forceinline__ void fold_high(Dot& d) const { d.hh = (d.hh & (int64_t)kM61) + (d.hh >> 61); }
  __device__ __forceinline__ void fold(Dot& d) const {
    d.mid += d.ll >> 31;
    d.ll &= 0x7fffffff;
    d.hh += d.mid >> 31;
    d.mid &= 0x7fffffff;
  }
  __device__ __forceinline__ R value(const Dot& d) const {
    // As in comb; ll and mid are below 2^63 in absolute value, hh may use all
    // 64 bits: 2 hh = 2 (hh mod 2^60) + (hh >> 60) mod p.
    const uint64_t t0 = ((uint64_t)d.ll & kM61) + 8 + (uint64_t)(d.ll >> 61);
    const uint64_t t1 = ((uint64_t)((uint32_t)d.mid & 0x3fffffffu) << 31) + (1ULL << 34) + (uint64_t)(d.mid >> 30);
    const uint64_t t2 = (((uint64_t)d.hh & ((1ULL << 60) - 1)) << 1) + 16 + (uint64_t)(d.hh >> 60);
    uint64_t x = t0 + t1 + t2;  // each below 2^61 + 2^35; too large by c
    constexpr uint64_t c = 8 + (1ULL << 34) + 16;
    x = (x & kM61) + (x >> 61) + (kM61 - c);
    x = (x & kM61) + (x >> 61);
    return x >= kM61 ? x - kM61 : x;
  }
};

// Even p (p = 2): Barrett reduction.
struct BmBarrett {
  using S = uint64_t;
  using W = S;
  using R = S;
  FpBarrett f;
  uint64_t r128;  // 2^128 mod p
  __device__ explicit BmBarrett(const FieldParams& p) : f(p) {
    const uint64_t m = f.reduce(~(u128)0);
    r128 = m + 1 == f.p ? 0 : m + 1;
  }
  __device__ __forceinline__ S pack(S x) const { return x; }
  __device__ __forceinline__ S load(S x) const { return x; }
  __device__ __forceinline__ S store(S x) const { return x; }
  __device__ __forceinline__ S neg(S d) const { return f.p - d; }
  __device__ __forceinline__ bool zero(S d) const { return d == 0; }
  __device__ __forceinline__ S comb(S bb, S a, S nd, S b) const { return f.reduce((u128)bb * a + (u128)nd * b); }
  __device__ __forceinline__ S add(S a, S b) const { return f.add(a, b); }
  struct Dot {
    u128 v = 0;
    uint32_t c = 0;
    __device__ __forceinline__ void mac(S a, S b) {
      const u128 t = (u128)a * b;
      v += t;
      c += v < t;
    }
  };
  static constexpr int kFold = kCoefRows, kFoldHigh = 0;
  __device__ __forceinline__ void fold_high(Dot&) const {}
  __device__ __forceinline__ void fold(Dot&) const {}
  __device__ __forceinline__ S value(const Dot& d) const { return f.add(f.reduce(d.v), f.mul(r128, d.c % f.p)); }
};

// Odd p < 2^63, R = 2^64: t < 2 p^2 reduces to (t + m p) / R < 2 p < 2^64.
struct BmMont64 {
  using S = uint64_t;
  using W = S;
  using R = S;
  uint64_t p, np;  // np = -1/p mod 2^64
  __device__ explicit BmMont64(const FieldParams& f) : p(f.p) {
    uint64_t x = p;  // p x = 1 mod 8, doubled in precision each time
#pragma unroll
    for (int i = 0; i < 5; ++i) x *= 2 - p * x;
    np = 0 - x;
  }
  // (t + m p) / 2^64 for t = hi 2^64 + lo: the low words cancel, with a carry
  // unless lo is 0.
  __device__ __forceinline__ u128 redc(uint64_t lo, u128 hi) const {
    return hi + __umul64hi(lo * np, p) + (lo != 0);
  }
  __device__ __forceinline__ S last(uint64_t u) const { return u >= p ? u - p : u; }
  __device__ __forceinline__ S pack(S x) const { return x; }
  __device__ __forceinline__ S load(S x) const { return x; }
  __device__ __forceinline__ S store(S x) const { return x; }
  __device__ __forceinline__ S neg(S d) const { return p - d; }
  __device__ __forceinline__ bool zero(S d) const { return d == 0; }
  __device__ __forceinline__ S comb(S bb, S a, S nd, S b) const {
    const u128 t = (u128)bb * a + (u128)nd * b;
    return last((uint64_t)(t >> 64) + __umul64hi((uint64_t)t * np, p) + ((uint64_t)t != 0));
  }
  __device__ __forceinline__ S add(S a, S b) const { return a >= p - b ? a - (p - b) : a + b; }
  struct Dot {
    u128 v = 0;
    uint32_t c = 0;
    __device__ __forceinline__ void mac(S a, S b) {
      const u128 t = (u128)a * b;
      v += t;
      c += v < t;
    }
  };
  static constexpr int kFold = kCoefRows, kFoldHigh = 0;
  __device__ __forceinline__ void fold_high(Dot&) const {}
  __device__ __forceinline__ void fold(Dot&) const {}
  __device__ __forceinline__ S value(const Dot& d) const {  // t < 66 p^2: 34 p after one step, 2 p after two
    const u128 u = redc((uint64_t)d.v, (u128)(uint64_t)(d.v >> 64) + ((u128)d.c << 64));
    return last((uint64_t)redc((uint64_t)u, (u128)(uint64_t)(u >> 64)));
  }
};

// Odd p < 2^31, residues stored in 32 bits, radix 2^32: t < 2 p^2 < 2^63
// reduces to (t + m p) / 2^32 < 2 p < 2^32. kWide (p >= 2^28, where 66
// products may pass 2^63): S is balanced, |x| <= 2^30, so that three offsets
// fit in 63 bits, and the high words are moved aside after them.
template <bool kWide>
struct BmMont32 {
  using S = int32_t;
  using W = uint32_t;
  using R = uint32_t;
  uint32_t p, np;  // np = -1/p mod 2^32
  __device__ explicit BmMont32(const FieldParams& f) : p((uint32_t)f.p) {
    uint32_t x = p;
#pragma unroll
    for (int i = 0; i < 4; ++i) x *= 2 - p * x;
    np = 0 - x;
  }
  __device__ __forceinline__ uint32_t last(uint32_t u) const { return min(u, u - p); }  // u < 2 p
  __device__ __forceinline__ S pack(R x) const { return kWide && x > p / 2 ? (S)(x - p) : (S)x; }
  __device__ __forceinline__ W load(S x) const { return kWide && x < 0 ? (W)x + p : (W)x; }
  __device__ __forceinline__ S store(W x) const { return pack(x); }
  __device__ __forceinline__ W neg(W d) const { return p - d; }
  __device__ __forceinline__ bool zero(W d) const { return d == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const {
    const uint64_t t = (uint64_t)bb * a + (uint64_t)nd * b;
    return last((uint32_t)((t + (uint64_t)((uint32_t)t * np) * p) >> 32));
  }
  __device__ __forceinline__ R add(R a, R b) const { return last(a + b); }
  struct Dot {
    int64_t v = 0;
    int64_t h = 0;  // high words of earlier offsets
    __device__ __forceinline__ void mac(S a, S b) { v += (int64_t)a * b; }
  };
  static constexpr int kFold = kWide ? 3 : kCoefRows, kFoldHigh = 0;
  __device__ __forceinline__ void fold_high(Dot&) const {}
  __device__ __forceinline__ void fold(Dot& d) const {
    if (!kWide) return;
    d.h += d.v >> 32;
    d.v = (uint32_t)d.v;
  }
  __device__ __forceinline__ R value(const Dot& d) const {
    // t = 2^32 h + v: one step leaves the high part, |u| < 2^36, plus m p /
    // 2^32 and a carry unless the low word is 0; 2^37 / p multiples of p make
    // it positive; the second step leaves less than p + 2^7.
    const uint32_t lo = (uint32_t)d.v;
    int64_t u = (d.v >> 32) + __umulhi(lo * np, p) + (lo != 0);
    if (kWide) u += d.h + ((int64_t)p << 9);
    return last((uint32_t)(((uint64_t)u + (uint64_t)((uint32_t)u * np) * p) >> 32));
  }
};

// The matrix of one block by offset: A'[j] = sum_o P[o] A[j+o] + Q[o] B[j+o],
// B'[j] = sum_o U[o] A[j+o] + V[o] B[j+o], o = omin .. 32.
template <class S>
struct alignas(4 * sizeof(S)) Coef {
  S c[4];  // P, Q, U, V
};

template <class S>
struct BmMatrix {
  Coef<S> row[kCoefRows];
  int omin;
};

// ---------------------------------------------------------------------------
// bm_base — one warp runs steps i .. min(i + 32, n) on the windows a, b (lane
// j: A[j], B[j]) and writes their matrix. In the frame of the block's start,
// after k steps, A_k = P A + Q B is divisible by x^k and B_k = x^sb (U A + V B)
// with deg P, Q < max(k, 1) and sb + deg U, V <= k; so window entry j and
// coefficient j never need the same lane at once, and x holds P in lanes
// below k and A_k's entries from lane k on, y holds U and the unshifted B_k's
// entries likewise (entry k - sb, the pivot, is kept in bb).
// Latency-bound chain of 32 x (shuffle, two products, reduction).
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void bm_base(const F& f, typename F::S a, typename F::S b, int64_t i, int64_t n,
                                        int64_t& l_io, BmMatrix<typename F::S>* M) {
  using W = typename F::W;
  const int lane = threadIdx.x & 31;
  W x = f.load(a), y = lane == 0 ? 0 : f.load(b), Q = 0, V = lane == 0;
  W bb = __shfl_sync(kAll, f.load(b), 0);
  int sb = 0, da = 0, db = 0;
  int64_t l = l_io;
  const int steps = n - i < kBmK ? (int)(n - i) : kBmK;
  int slack = (int)(i - 2 * l);  // 2 l <= i + k exactly when slack + k >= 0
  int dl = 0;                    // change of l
#pragma unroll 4
  for (int k = 0; k < steps; ++k) {
    const W d = __shfl_sync(kAll, x, k);
    W ys = __shfl_sync(kAll, y, lane - sb), vs = __shfl_sync(kAll, V, lane - sb);
    if (lane < sb) ys = vs = 0;
    if (lane == k) x = k == 0;
    // d == 0 takes the same update: A <- bb A, a nonzero multiple.
    const W nd = f.neg(d);
    const W nx = f.comb(bb, x, nd, ys), nq = f.comb(bb, Q, nd, vs);
    const bool nzd = !f.zero(d);
    const bool grow = nzd && slack + k >= 0;  // 2 l <= i + k
    const int dn = nzd && sb + db > da ? sb + db : da;
    if (grow) {
      const int g = slack + k + 1;  // l <- i + k + 1 - l
      dl += g;
      slack -= 2 * g;
      db = da;
    }
    y = grow ? x : y;
    V = grow ? Q : V;
    bb = grow ? d : bb;
    sb = grow ? 1 : sb + 1;
    da = dn;
    x = nx;
    Q = nq;
  }
  l_io = l + dl;
  // Offsets: coefficient k of the A row sits at 32 - k, of the B row at
  // 32 - sb - k.
  if (steps < kBmK) return;  // the sequence ends here: nothing is applied
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    M->row[lane].c[q] = 0;
    if (lane == 0) M->row[kBmK].c[q] = 0;
  }
  __syncwarp();
  M->row[kBmK - lane].c[0] = f.store(x);
  M->row[kBmK - lane].c[1] = f.store(Q);
  if (lane <= db) {
    M->row[kBmK - sb - lane].c[2] = f.store(y);
    M->row[kBmK - sb - lane].c[3] = f.store(V);
  }
  if (lane == 0) M->omin = kBmK - (da > sb + db ? da : sb + db);
  __syncwarp();
}

// ---------------------------------------------------------------------------
// bm_front — kFront warps compute the next window, outputs 0 .. 31: warp w
// sums every (kFront / 4)-th offset of coefficient w & 3 (P, Q, U, V); warp 0
// adds the parts and returns the window. Barrier 3 joins the warps. On the
// critical path of the steps, so spread thin: latency of ~5 dependent
// products at 8 warps.
// ---------------------------------------------------------------------------
template <int kFront, class F>
__device__ __forceinline__ void bm_front(const F& f, const typename F::S* A, const typename F::S* B,
                                         const BmMatrix<typename F::S>& M, typename F::R (*fr)[32], int w,
                                         typename F::S& a, typename F::S& b) {
  using S = typename F::S;
  using R = typename F::R;
  constexpr int kStep = kFront / 4;
  const int lane = threadIdx.x & 31;
  const S* X = ((w & 1) ? B : A) + lane;
  const S* c = &M.row[0].c[w & 3];
  typename F::Dot acc[2];
  int o = M.omin + (w >> 2);
#pragma unroll 1
  for (; o + 3 * kStep < kCoefRows; o += 4 * kStep) {
    S xv[4], cv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      xv[u] = X[o + u * kStep];
      cv[u] = c[4 * (o + u * kStep)];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u & 1].mac(cv[u], xv[u]);
    f.fold(acc[0]);
    f.fold(acc[1]);
  }
#pragma unroll
  for (int u = 0; u < 3; ++u)
    if (o + u * kStep < kCoefRows) acc[u & 1].mac(c[4 * (o + u * kStep)], X[o + u * kStep]);
  const R v = f.add(f.value(acc[0]), f.value(acc[1]));
  if (w != 0) {
    fr[w][lane] = v;
    asm volatile("bar.arrive 3, %0;" ::"n"(32 * kFront) : "memory");
    return;
  }
  asm volatile("bar.sync 3, %0;" ::"n"(32 * kFront) : "memory");
  R ra = f.add(v, fr[1][lane]), rb = f.add(fr[2][lane], fr[3][lane]);
#pragma unroll
  for (int q = 4; q < kFront; q += 4) {
    ra = f.add(ra, f.add(fr[q][lane], fr[q + 1][lane]));
    rb = f.add(rb, f.add(fr[q + 2][lane], fr[q + 3][lane]));
  }
  a = f.pack(ra);
  b = f.pack(rb);
}

// ---------------------------------------------------------------------------
// bm_dots — entries j[q] (q < N) of A' and B' by one thread. Bound by the
// integer multiply pipe: four products per entry pair and offset.
// ---------------------------------------------------------------------------
template <int N, class F>
__device__ __forceinline__ void bm_dots(const F& f, const typename F::S* A, const typename F::S* B,
                                        const BmMatrix<typename F::S>& M, int j0, int T, int lim,
                                        typename F::R (&va)[4], typename F::R (&vb)[4]) {
  using S = typename F::S;
  typename F::Dot da[N], db[N];
  const S *pa[N], *pb[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int j = min(j0 + q * T, lim - 1);
    pa[q] = A + j;
    pb[q] = B + j;
  }
  const auto at = [&](int o) {
    const Coef<S> c = M.row[o];
    S av[N], bv[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      av[q] = pa[q][o];
      bv[q] = pb[q][o];
    }
#pragma unroll
    for (int q = 0; q < N; ++q) da[q].mac(c.c[0], av[q]);
#pragma unroll
    for (int q = 0; q < N; ++q) db[q].mac(c.c[2], av[q]);
#pragma unroll
    for (int q = 0; q < N; ++q) da[q].mac(c.c[1], bv[q]);
#pragma unroll
    for (int q = 0; q < N; ++q) db[q].mac(c.c[3], bv[q]);
  };
  constexpr int kU = F::kFold < 4 ? F::kFold : 4;
  int o = M.omin, high = 0;
#pragma unroll 1
  for (; o + kU <= kCoefRows; o += kU) {
#pragma unroll
    for (int u = 0; u < kU; ++u) at(o + u);
    if (F::kFold < kCoefRows) {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        f.fold(da[q]);
        f.fold(db[q]);
      }
    }
    if (F::kFoldHigh && ++high == F::kFoldHigh) {
      high = 0;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        f.fold_high(da[q]);
        f.fold_high(db[q]);
      }
    }
  }
#pragma unroll 1
  for (; o < kCoefRows; ++o) at(o);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    va[q] = f.value(da[q]);
    vb[q] = f.value(db[q]);
  }
}

// ---------------------------------------------------------------------------
// bm_apply — entries t0 .. lim of A' and B' in place by a group of T threads
// (t: this thread's number), up to four entries per thread and tile. Output j
// is stored at j and reads reach from j to j + 32, so bar(k), the barrier of
// tile k, separates the group's reads from its writes. A warp computes only as
// many entries as it has (a tile's last entries leave the other warps free).
// ---------------------------------------------------------------------------
template <class F, class Bar>
__device__ __forceinline__ void bm_apply(const F& f, typename F::S* A, typename F::S* B,
                                         const BmMatrix<typename F::S>& M, int t0, int T, int t, int lim, bool& nz,
                                         Bar&& bar) {
  for (int k = 0; t0 < lim; ++k, t0 += 4 * T) {
    typename F::R va[4], vb[4];
    const int left = lim - t0 - (t & ~31);  // from this warp's first entry
    const int mine = left <= 0 ? 0 : (left + T - 1) / T;
    if (mine >= 3)
      bm_dots<4>(f, A, B, M, t0 + t, T, lim, va, vb);
    else if (mine == 2)
      bm_dots<2>(f, A, B, M, t0 + t, T, lim, va, vb);
    else if (mine == 1)
      bm_dots<1>(f, A, B, M, t0 + t, T, lim, va, vb);
    bar(k);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = t0 + q * T + t;
      if (q < mine && j < lim) {
        A[j] = f.pack(va[q]);
        B[j] = f.pack(vb[q]);
        nz |= va[q] != 0;
      }
    }
  }
}

// Entries of A and B of the start: c = b = 1, bb = 1 (src/fp.rs:262-268), so
// A = s and B = 1 + x s.
__device__ __forceinline__ uint64_t bm_b0(const uint64_t* s, int64_t j) { return j ? s[j - 1] : 1; }

struct BmShared {
  BmMatrix<uint64_t> M[2];
  alignas(16) uint64_t fr[8][32];
  int64_t l;
  long long job;
  int flag;
};

// ---------------------------------------------------------------------------
// One sequence with the whole CTA (blockDim a multiple of 32, at least 128).
// A, B: n + kBmPad entries each, owned by this CTA. Per block of 32 steps one
// barrier of the whole CTA, and one among the applying warps per tile.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ int64_t bm_run(const F& f, const uint64_t* __restrict__ s, int64_t n64, typename F::S* A,
                                          typename F::S* B, BmShared& sh) {
  using S = typename F::S;
  using R = typename F::R;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int n = (int)n64;
  BmMatrix<S>* M = reinterpret_cast<BmMatrix<S>*>(sh.M);
  typename F::R(*fr)[32] = reinterpret_cast<typename F::R(*)[32]>(sh.fr);
  bool nz = false;
  for (int j = tid; j < n + kBmPad; j += T) {
    const S v = j < n ? f.pack((R)s[j]) : 0;
    A[j] = v;
    B[j] = j < n ? f.pack((R)bm_b0(s, j)) : 0;
    nz |= v != 0;
  }
  int64_t l = 0;
  __syncthreads();
  S a = 0, b = 0;
  if (warp == 0) {
    a = A[lane];
    b = B[lane];
    bm_base(f, a, b, 0, n, l, &M[0]);
  }
  for (int i = 0;; i += kBmK) {
    // Every thread's part of A (steps i on) has been written and tested, and
    // the block's matrix is there.
    const bool any = __syncthreads_or(nz);
    if (!any || i + kBmK >= n) break;
    nz = false;
    const BmMatrix<S>& m = M[(i / kBmK) & 1];
    const int lim = n - i - kBmK;  // outputs
    if (T >= 512) {
      if (warp < 8) bm_front<8>(f, A, B, m, fr, warp, a, b);
    } else if (warp < 4) {
      bm_front<4>(f, A, B, m, fr, warp, a, b);
    }
    if (warp == 0) {
      // The first tile's writes wait until the front has read its inputs.
      if (lim > kBmK) asm volatile("bar.arrive 1, %0;" ::"r"(T) : "memory");
      if (lane >= lim) a = b = 0;
      nz = a != 0;
      A[lane] = a;  // read by no thread until the next barrier of the CTA
      B[lane] = b;
      bm_base(f, a, b, i + kBmK, n, l, &M[((i / kBmK) & 1) ^ 1]);
    } else {
      bm_apply(f, A, B, m, kBmK, T - 32, tid - 32, lim, nz, [&](int k) {
        if (k == 0)
          asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
        else
          asm volatile("bar.sync 2, %0;" ::"r"(T - 32) : "memory");
      });
    }
  }
  if (tid == 0) sh.l = l;
  __syncthreads();
  return sh.l;
}

template <class F>
__device__ __forceinline__ int64_t bm_any(const BmJob& job, const FieldParams& fp, uint64_t* smem, uint64_t* gws,
                                          int64_t smem_words, BmShared& sh) {
  using S = typename F::S;
  const F f(fp);
  const int64_t m = job.n + kBmPad;
  if (bm_words<S>(job.n) <= smem_words) {
    S* A = reinterpret_cast<S*>(smem);
    return bm_run(f, job.s, job.n, A, A + m, sh);
  }
  S* A = reinterpret_cast<S*>(gws);
  return bm_run(f, job.s, job.n, A, A + m, sh);
}

__device__ __forceinline__ int64_t bm_dispatch(const BmJob& job, uint64_t* smem, uint64_t* gws, int64_t smem_words,
                                               BmShared& sh) {
  if (job.n <= 0) return 0;
  const FieldParams fp{job.p, job.mu_lo, job.mu_hi, job.safe_batch};
  if (job.p == kM61) return bm_any<BmM61>(job, fp, smem, gws, smem_words, sh);
  if (!(job.p & 1)) return bm_any<BmBarrett>(job, fp, smem, gws, smem_words, sh);
  if (job.p < (1ULL << 28)) return bm_any<BmMont32<false>>(job, fp, smem, gws, smem_words, sh);
  if (job.p < (1ULL << 31)) return bm_any<BmMont32<true>>(job, fp, smem, gws, smem_words, sh);
  return bm_any<BmMont64>(job, fp, smem, gws, smem_words, sh);
}

// Plain form: one CTA runs one sequence, A and B in dynamic shared memory when
// they fit, else in the global workspace.
__global__ void __launch_bounds__(512) bm_block_kernel(BmJob job, uint64_t* gws, int64_t smem_words, int64_t* out) {
  extern __shared__ __align__(16) uint64_t bm_smem[];
  __shared__ BmShared sh;
  const int64_t l = bm_dispatch(job, bm_smem, gws, smem_words, sh);
  if (threadIdx.x == 0) *out = l;
}

// Batched form: persistent CTAs take jobs from a device counter; the host
// orders jobs longest first (LPT). Each CTA has smem_words of dynamic shared
// memory and a private global slice of gws_words for jobs that do not fit.
__global__ void __launch_bounds__(512)
    bm_batch_kernel(const BmJob* __restrict__ jobs, int64_t count, unsigned long long* next, uint64_t* gws,
                    int64_t gws_words, int64_t smem_words, int64_t* out) {
  extern __shared__ __align__(16) uint64_t bm_smem[];
  __shared__ BmShared sh;
  for (;;) {
    if (threadIdx.x == 0) sh.job = (long long)atomicAdd(next, 1ULL);
    __syncthreads();
    const long long q = sh.job;
    __syncthreads();
    if (q >= count) break;
    const BmJob job = jobs[q];
    const int64_t l = bm_dispatch(job, bm_smem, gws + (int64_t)blockIdx.x * gws_words, smem_words, sh);
    if (threadIdx.x == 0) out[job.slot] = l;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// bm_long_kernel — one sequence on G co-resident CTAs.
//
// Steps run in superblocks of kBmT = 512 (16 blocks). CTA 0 holds the first
// 512 entries of A and B, runs the superblock's blocks on them and publishes
// every matrix in a ring in global memory. The other CTAs take chunks of the
// outputs (the superblock's A and B, 512 steps on): a chunk's inputs and the
// 512 entries after it are loaded into shared memory, the 16 matrices are
// applied in place as they arrive (the valid part shrinks by 32 each time),
// and the outputs go to the other of two global buffers. The first 512
// outputs, which CTA 0 needs next, are chunks of their own of 128 outputs;
// CTA 0 starts the next superblock when they are there, while the rest of
// the outputs are still being computed. A chunk of the next superblock starts
// when all chunks of this one are done.
//
// Waits (all bounded; on expiry the error word is set, every CTA leaves, and
// the host reports it): CTA 0 on `front`, chunks on `done` and on `pub`. The
// CTAs are co-resident (cooperative launch, or one cluster).
// skip_cta >= 0 is a failure-detection test: that CTA does not signal (CTA 0
// its first matrix, another its first chunk), so the waits expire.
// ---------------------------------------------------------------------------
constexpr int kBmH = 16;
constexpr int kBmT = kBmH * kBmK;
constexpr int kBmFront = 128;   // outputs of a front chunk
constexpr int kLongThreads = 512;
constexpr int64_t kLongSmem = 200 * 1024;

struct LongSync {
  unsigned int pub, front, done;  // matrices published, front chunks and chunks finished
  int stop, err;
};

struct LongArgs {
  const uint64_t* s;
  int64_t n;
  void* buf;        // [2][2][n + kBmPad] entries: parity, A or B
  void* ring;       // [2 kBmH] matrices
  unsigned int* nz;  // per superblock: some output is nonzero
  LongSync* gs;
  int64_t* out;
  long long spin;
  int skip_cta, cap;  // cap: largest chunk
};

// The chunks of superblock s: nf of front outputs in `front` chunks, the rest
// in chunks of `size`.
struct LongPlan {
  int64_t nout, nf, size;
  int front, chunks;
  __device__ LongPlan(int64_t n, int64_t s, int G, int cap) {
    nout = n - (s + 1) * kBmT;
    if (nout < 0) nout = 0;
    nf = nout < kBmT ? nout : kBmT;
    front = (int)((nf + kBmFront - 1) / kBmFront);
    const int64_t rest = nout - nf;
    const int64_t w = G - 1 - front > 0 ? G - 1 - front : 1;
    size = ((rest + w - 1) / w + 31) / 32 * 32;
    if (size < kBmFront) size = kBmFront;
    if (size > cap) size = cap;
    chunks = front + (int)((rest + size - 1) / size);
  }
  __device__ void range(int c, int64_t& lo, int64_t& hi) const {
    lo = c < front ? (int64_t)c * kBmFront : nf + (c - front) * size;
    hi = c < front ? (lo + kBmFront < nf ? lo + kBmFront : nf) : (lo + size < nout ? lo + size : nout);
  }
};

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// One thread waits until *p >= want (as a running count); false on stop,
// error or expiry.
__device__ __forceinline__ bool long_wait(const unsigned int* p, unsigned int want, LongSync* gs, long long spin) {
  const long long t0 = clock64();
  while ((int)(ld_acquire(p) - want) < 0) {
    if (ld_acquire(reinterpret_cast<unsigned int*>(&gs->stop))) return false;
    if (*(volatile int*)&gs->err) return false;
    if (clock64() - t0 > spin) {
      atomicExch(&gs->err, 1);
      return false;
    }
  }
  return true;
}

template <class F>
__global__ void __launch_bounds__(kLongThreads, 1) bm_long_kernel(FieldParams fp, LongArgs g) {
  using S = typename F::S;
  extern __shared__ __align__(16) uint64_t bm_smem[];
  __shared__ BmShared sh;
  const F f(fp);
  const int tid = threadIdx.x, T = kLongThreads, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x;
  const int64_t n = g.n, pitch = n + kBmPad;
  S* buf = static_cast<S*>(g.buf);
  BmMatrix<S>* ring = static_cast<BmMatrix<S>*>(g.ring);
  BmMatrix<S>* M = reinterpret_cast<BmMatrix<S>*>(sh.M);
  S* A = reinterpret_cast<S*>(bm_smem);
  // Entry j of A (which = 0) or B (1) at the start of superblock s.
  const auto entry = [&](int64_t s, int which, int64_t j) -> S {
    if (j >= n - s * kBmT) return 0;
    if (s == 0) return f.pack((typename F::R)(which ? bm_b0(g.s, j) : g.s[j]));
    return __ldcg(buf + ((s & 1) * 2 + which) * pitch + j);
  };

  if (blockIdx.x == 0) {
    // ---------------- the steps -------------------------------------------
    S* B = A + kBmT + kBmPad;
    typename F::R(*fr)[32] = reinterpret_cast<typename F::R(*)[32]>(sh.fr);
    int64_t l = 0;
    unsigned int want_front = 0, want_done = 0;
    bool ok = true;
    for (int64_t s = 0; s * kBmT < n; ++s) {
      if (s > 0) {
        const LongPlan prev(n, s - 1, G, g.cap);
        want_front += prev.front;
        want_done += prev.chunks;
        if (tid == 0) sh.flag = long_wait(&g.gs->front, want_front, g.gs, g.spin);
        __syncthreads();
        ok = sh.flag;
        if (!ok) break;
      }
      bool nz = false;
      for (int j = tid; j < kBmT + kBmPad; j += T) {
        const S v = j < kBmT ? entry(s, 0, j) : 0;
        A[j] = v;
        B[j] = j < kBmT ? entry(s, 1, j) : 0;
        nz |= v != 0;
      }
      const bool any = __syncthreads_or(nz);
      if (s > 0 && !any) {
        // The window is zero: if all of A is, the sequence is done.
        if (tid == 0) {
          sh.flag = long_wait(&g.gs->done, want_done, g.gs, g.spin);
          if (sh.flag && __ldcg(g.nz + s) == 0) sh.flag = 2;
        }
        __syncthreads();
        if (sh.flag != 1) {
          ok = sh.flag == 2;
          break;
        }
      }
      S a = 0, b = 0;
      const int64_t i0 = s * kBmT;
      const bool feeds = n - i0 > kBmT;  // later steps need the matrices
      if (warp == 0) {
        a = A[lane];
        b = B[lane];
        bm_base(f, a, b, i0, n, l, &M[0]);
      }
      for (int h = 0; h < kBmH && i0 + h * kBmK < n; ++h) {
        __syncthreads();
        const BmMatrix<S>& m = M[h & 1];
        const int lim = kBmT - (h + 1) * kBmK;  // outputs inside the window
        const bool more = lim > 0 && i0 + (h + 1) * kBmK < n;
        if (more && warp < 8) bm_front<8>(f, A, B, m, fr, warp, a, b);
        if (warp == 0) {
          if (more) {
            if (lim > kBmK) asm volatile("bar.arrive 1, %0;" ::"r"(T - 32) : "memory");
            A[lane] = a;
            B[lane] = b;
            bm_base(f, a, b, i0 + (h + 1) * kBmK, n, l, &M[(h & 1) ^ 1]);
          }
        } else if (warp == T / 32 - 1) {
          if (feeds) {
            // The last warp publishes: 16-byte words of the matrix, then the count.
            const int64_t q = s * kBmH + h;
            const uint4* src = reinterpret_cast<const uint4*>(&m);
            uint4* dst = reinterpret_cast<uint4*>(ring + q % (2 * kBmH));
            for (int w = lane; w < (int)(sizeof(BmMatrix<S>) / 16); w += 32) __stcg(dst + w, src[w]);
            __threadfence();
            __syncwarp();
            if (lane == 0 && !(q == 0 && g.skip_cta == 0)) atomicAdd(&g.gs->pub, 1u);
          }
        } else if (more) {
          bool unused = false;
          bm_apply(f, A, B, m, kBmK, T - 64, tid - 32, lim, unused, [&](int k) {
            if (k == 0)
              asm volatile("bar.sync 1, %0;" ::"r"(T - 32) : "memory");
            else
              asm volatile("bar.sync 2, %0;" ::"r"(T - 64) : "memory");
          });
        }
      }
      __syncthreads();
    }
    if (tid == 0) {
      __threadfence();
      atomicExch(&g.gs->stop, 1);
      if (ok) *g.out = l;
    }
    return;
  }

  // ---------------- the chunks ----------------------------------------------
  const int wk = blockIdx.x - 1;
  S* B = A + g.cap + kBmT + kBmPad;
  unsigned int want_done = 0;
  for (int64_t s = 0;; ++s) {
    const LongPlan P(n, s, G, g.cap);
    if (P.nout == 0) return;
    for (int c = wk; c < P.chunks; c += G - 1) {
      if (tid == 0) sh.flag = long_wait(&g.gs->done, want_done, g.gs, g.spin);
      __syncthreads();
      if (!sh.flag) return;
      int64_t lo, hi;
      P.range(c, lo, hi);
      const int len = (int)(hi - lo);
      for (int j = tid; j < len + kBmT; j += T) {
        A[j] = entry(s, 0, lo + j);
        B[j] = entry(s, 1, lo + j);
      }
      bool nz = false;
      for (int h = 0; h < kBmH; ++h) {
        const int64_t q = s * kBmH + h;
        if (tid == 0) sh.flag = long_wait(&g.gs->pub, (unsigned)(q + 1), g.gs, g.spin);
        __syncthreads();  // also: the previous matrix has been applied
        if (!sh.flag) return;
        const uint4* src = reinterpret_cast<const uint4*>(ring + q % (2 * kBmH));
        uint4* dst = reinterpret_cast<uint4*>(&M[0]);
        for (int w = tid; w < (int)(sizeof(BmMatrix<S>) / 16); w += T) dst[w] = __ldcg(src + w);
        __syncthreads();
        nz = false;
        bm_apply(f, A, B, M[0], 0, T, tid, len + kBmT - (h + 1) * kBmK, nz, [](int) { __syncthreads(); });
      }
      __syncthreads();
      S* oa = buf + ((s + 1) & 1) * 2 * pitch + lo;
      for (int j = tid; j < len; j += T) {
        __stcg(oa + j, A[j]);
        __stcg(oa + pitch + j, B[j]);
      }
      __threadfence();
      const bool any = __syncthreads_or(nz);
      if (tid == 0 && !(s == 0 && (int)blockIdx.x == g.skip_cta)) {
        if (any) atomicOr(g.nz + s + 1, 1u);
        __threadfence();
        if (c < P.front) atomicAdd(&g.gs->front, 1u);
        atomicAdd(&g.gs->done, 1u);
      }
    }
    want_done += P.chunks;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host launchers.
// ---------------------------------------------------------------------------
int64_t bm_smem_words(uint64_t p, int64_t n) { return (p & 1) && p < (1ULL << 31) ? bm_words<uint32_t>(n) : bm_words<uint64_t>(n); }
int64_t bm_workspace_words(int64_t n) { return bm_words<uint64_t>(n); }

cudaError_t launch_bm_block(const BmJob& job, uint64_t* gws, int64_t smem_words, int threads, int64_t* d_out,
                            cudaStream_t st) {
  const int64_t need = bm_smem_words(job.p, job.n);
  const size_t smem = need <= smem_words ? (size_t)need * 8 : 0;
  if (smem > 0)  // dynamic + static shared memory may pass 48 KiB even when smem alone does not
    cudaFuncSetAttribute(bm_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  bm_block_kernel<<<1, threads, smem, st>>>(job, gws, smem_words, d_out);
  return cudaGetLastError();
}

cudaError_t bm_block_prepare() {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, bm_block_kernel);
}

// The batch kernel's dynamic shared memory cap is set once to the largest
// size any batch asks for (200 KiB), so launches of any batch, graph-captured
// ones included, need no attribute call.
static cudaError_t bm_batch_attr() {
  static cudaError_t e =
      cudaFuncSetAttribute(bm_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  return e;
}

cudaError_t launch_bm_batch(const BmJob* d_jobs, int64_t count, unsigned long long* d_next, uint64_t* gws,
                            int64_t gws_words, int64_t smem_words, int blocks, int threads, int64_t* d_out,
                            cudaStream_t st) {
  const size_t smem = (size_t)smem_words * 8;
  cudaError_t e = bm_batch_attr();
  if (e != cudaSuccess) return e;
  bm_batch_kernel<<<blocks, threads, smem, st>>>(d_jobs, count, d_next, gws, gws_words, smem_words, d_out);
  return cudaGetLastError();
}

int bm_batch_max_blocks_per_sm(int threads, int64_t smem_words) {
  const size_t smem = (size_t)smem_words * 8;
  if (bm_batch_attr() != cudaSuccess) return 0;
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, bm_batch_kernel, threads, smem);
  return nb;
}

// Layout of the long kernel's workspace: sync words, nonzero flags per
// superblock, the ring, the two buffers.
static size_t long_flags(int64_t n) { return ((size_t)(n / kBmT + 3) * sizeof(unsigned int) + 255) / 256 * 256; }
static size_t long_ring() { return (2 * kBmH * sizeof(BmMatrix<uint64_t>) + 255) / 256 * 256; }

size_t bm_long_bytes(int64_t n) {
  return 256 + long_flags(n) + long_ring() + (size_t)4 * (n + kBmPad) * sizeof(uint64_t);
}
int bm_long_err_offset() { return (int)offsetof(LongSync, err); }

template <class F>
static cudaError_t launch_long_t(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, bool cluster,
                                 void* ws, long long spin, int skip_cta, int64_t* d_out, cudaStream_t st) {
  using S = typename F::S;
  char* w = static_cast<char*>(ws);
  LongArgs a{};
  a.s = s;
  a.n = n;
  a.gs = reinterpret_cast<LongSync*>(w);
  a.nz = reinterpret_cast<unsigned int*>(w + 256);
  a.ring = w + 256 + long_flags(n);
  a.buf = w + 256 + long_flags(n) + long_ring();
  a.out = d_out;
  a.spin = spin;
  a.skip_cta = skip_cta;
  // The largest chunk: the first superblock's share, within the shared memory.
  const int64_t front = std::min<int64_t>(std::max<int64_t>(n - kBmT, 0), kBmT);
  const int64_t fchunks = (front + kBmFront - 1) / kBmFront;
  const int64_t rest = std::max<int64_t>(n - 2 * kBmT, 0);
  const int64_t share = std::max<int64_t>(ctas - 1 - fchunks, 1);
  const int64_t room = kLongSmem / (2 * (int64_t)sizeof(S)) - kBmT - kBmPad;
  int64_t cap = ((rest + share - 1) / share + 31) / 32 * 32;
  cap = std::max<int64_t>(std::min(cap, room / 32 * 32), kBmFront);
  a.cap = (int)cap;
  const size_t smem = (size_t)2 * (cap + kBmT + kBmPad) * sizeof(S);
  cudaError_t e = cudaFuncSetAttribute(bm_long_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(ws, 0, 256 + long_flags(n), st);
  if (e != cudaSuccess) return e;
  if (!cluster) {
    FieldParams f = fp;
    void* args[] = {&f, &a};
    return cudaLaunchCooperativeKernel((void*)bm_long_kernel<F>, dim3(ctas), dim3(kLongThreads), args, smem, st);
  }
  if (ctas > 8) {
    e = cudaFuncSetAttribute(bm_long_kernel<F>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kLongThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  e = cudaOccupancyMaxActiveClusters(&nclusters, bm_long_kernel<F>, &cfg);
  if (e != cudaSuccess) return e;
  if (nclusters < 1) return cudaErrorInvalidConfiguration;
  return cudaLaunchKernelEx(&cfg, bm_long_kernel<F>, fp, a);
}

static cudaError_t launch_long(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, bool cluster, void* ws,
                               long long spin, int skip_cta, int64_t* d_out, cudaStream_t st) {
  if (fp.p == kM61) return launch_long_t<BmM61>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st);
  if (!(fp.p & 1)) return launch_long_t<BmBarrett>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st);
  if (fp.p < (1ULL << 28))
    return launch_long_t<BmMont32<false>>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st);
  if (fp.p < (1ULL << 31))
    return launch_long_t<BmMont32<true>>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st);
  return launch_long_t<BmMont64>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st);
}

cudaError_t launch_bm_long(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, int num_sms, void* ws,
                           long long spin, int skip_cta, int64_t* d_out, cudaStream_t st) {
  // One CTA per SM; no more than have a chunk in the first superblock.
  const int64_t useful = 1 + (std::max<int64_t>(n - kBmT, 0) + kBmFront - 1) / kBmFront;
  const int G = (int)std::max<int64_t>(2, std::min<int64_t>({(int64_t)ctas, (int64_t)num_sms, useful}));
  return launch_long(fp, s, n, G, false, ws, spin, skip_cta, d_out, st);
}

cudaError_t launch_bm_cluster(const FieldParams& fp, const uint64_t* s, int64_t n, void* ws, long long spin,
                              int64_t* d_out, cudaStream_t st) {
  cudaError_t e = launch_long(fp, s, n, 16, true, ws, spin, -1, d_out, st);
  if (e != cudaSuccess) {  // a device without 16-CTA clusters
    cudaGetLastError();
    e = launch_long(fp, s, n, 8, true, ws, spin, -1, d_out, st);
  }
  return e;
}

}  // namespace modlin
