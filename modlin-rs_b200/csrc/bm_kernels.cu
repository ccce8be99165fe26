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
// which the other warps then apply to the rest of A and B (bm_apply): 2 x 2
// products per entry and coefficient, about 2 per entry and step, as 8-bit limb
// products on the tensor cores, reduced once per 32 steps.
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
#include "launch.cuh"
#include "mma_limbs.cuh"

namespace modlin {

namespace {

constexpr int kBmK = 32;             // steps per block, window entries
constexpr int kCoefRows = kBmK + 1;  // offsets 0 .. 32
constexpr unsigned kAll = 0xffffffffu;

// ---------------------------------------------------------------------------
// Field policies. W: what bm_base works on; load and store convert canonical
// residues. comb = (bb a + nd b) / r mod p, nd = neg(d), with r = 1 or the
// Montgomery radix 2^32 or 2^64: a common factor of all of A (or of all of B)
// changes no zero and so no complexity, and Montgomery's reduction is a third
// of Barrett's dependent chain. Red, L: the reductions of limb products
// (limb_sums.cuh) and the limbs of a residue.
// ---------------------------------------------------------------------------
// Values up to p + 6 on W: bb a + nd b < 2^122.1 + 2^123.1.
struct BmM61 {
  using F = FpM61;
  using W = uint64_t;
  static constexpr int L = 8;
  __device__ explicit BmM61(const FieldParams&) {}
  __device__ __forceinline__ W load(uint64_t x) const { return x; }
  __device__ __forceinline__ uint64_t store(W x) const { return x >= kM61 ? x - kM61 : x; }
  __device__ __forceinline__ W neg(W d) const { return 2 * kM61 - d; }
  __device__ __forceinline__ bool zero(W d) const { return d == 0 || d == kM61; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const {
    const u128 t = (u128)bb * a + (u128)nd * b;
    const uint64_t lo = (uint64_t)t, hi = (uint64_t)(t >> 64);  // hi < 2^60
    return FpM61::fold((lo & kM61) + ((hi << 3) | (lo >> 61)));
  }
};

// Even p (p = 2): Barrett reduction.
template <class G, int LIMBS>
struct BmBarrett {
  using F = G;
  using W = uint64_t;
  static constexpr int L = LIMBS;
  F f;
  __device__ explicit BmBarrett(const FieldParams& p) : f(p) {}
  __device__ __forceinline__ W load(uint64_t x) const { return x; }
  __device__ __forceinline__ uint64_t store(W x) const { return x; }
  __device__ __forceinline__ W neg(W d) const { return f.modulus() - d; }
  __device__ __forceinline__ bool zero(W d) const { return d == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const { return f.reduce2(f.prod(bb, a) + f.prod(nd, b)); }
};

// Odd p < 2^63, r = 2^64: t < 2 p^2 reduces to (t + m p) / r < 2 p < 2^64.
struct BmMont64 {
  using F = FpBarrett;
  using W = uint64_t;
  static constexpr int L = 8;
  uint64_t p, np;  // np = -1/p mod 2^64
  __device__ explicit BmMont64(const FieldParams& f) : p(f.p) {
    uint64_t x = p;  // p x = 1 mod 8, doubled in precision each time
#pragma unroll
    for (int i = 0; i < 5; ++i) x *= 2 - p * x;
    np = 0 - x;
  }
  __device__ __forceinline__ W load(uint64_t x) const { return x; }
  __device__ __forceinline__ uint64_t store(W x) const { return x; }
  __device__ __forceinline__ W neg(W d) const { return p - d; }
  __device__ __forceinline__ bool zero(W d) const { return d == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const {
    const u128 t = (u128)bb * a + (u128)nd * b;
    // The low words cancel, with a carry unless they are 0.
    const uint64_t u = (uint64_t)(t >> 64) + __umul64hi((uint64_t)t * np, p) + ((uint64_t)t != 0);
    return u >= p ? u - p : u;
  }
};

// Odd p < 2^31, r = 2^32: t < 2 p^2 < 2^63 reduces to (t + m p) / r < 2 p < 2^32.
template <int LIMBS>
struct BmMont32 {
  using F = FpSmall;
  using W = uint32_t;
  static constexpr int L = LIMBS;
  uint32_t p, np;  // np = -1/p mod 2^32
  __device__ explicit BmMont32(const FieldParams& f) : p((uint32_t)f.p) {
    uint32_t x = p;
#pragma unroll
    for (int i = 0; i < 4; ++i) x *= 2 - p * x;
    np = 0 - x;
  }
  __device__ __forceinline__ W load(uint64_t x) const { return (W)x; }
  __device__ __forceinline__ uint64_t store(W x) const { return x; }
  __device__ __forceinline__ W neg(W d) const { return p - d; }
  __device__ __forceinline__ bool zero(W d) const { return d == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const {
    const uint64_t t = (uint64_t)bb * a + (uint64_t)nd * b;
    const uint32_t u = (uint32_t)((t + (uint64_t)((uint32_t)t * np) * p) >> 32);
    return min(u, u - p);
  }
};

// The matrix of one block by offset: A'[j] = sum_o c[0][o] A[j+o] + c[1][o]
// B[j+o], B'[j] = sum_o c[2][o] A[j+o] + c[3][o] B[j+o], o = omin .. 32 (P, Q, U,
// V; canonical residues).
struct alignas(16) BmMatrix {
  uint64_t c[4][kCoefRows];
  int omin;
};
static_assert(sizeof(BmMatrix) % 16 == 0, "published as 16-byte words");

// ---------------------------------------------------------------------------
// bm_base — one warp runs steps i .. min(i + 32, n) on the windows a, b (lane
// j: A[j], B[j], canonical) and writes their matrix. In the frame of the
// block's start, after k steps, A_k = P A + Q B is divisible by x^k and B_k =
// x^sb (U A + V B) with deg P, Q < max(k, 1) and sb + deg U, V <= k; so window
// entry j and coefficient j never need the same lane at once, and x holds P in
// lanes below k and A_k's entries from lane k on, y holds U and the unshifted
// B_k's entries likewise (entry k - sb, the pivot, is kept in bb).
// A dependent chain of 32 x (shuffle, two products, reduction): 190 cycles a
// step over 2^61 - 1, 90 with 32-bit Montgomery. (A second warp for Q and V
// measured 203 and 120: the chain, not the issue, is the bound.)
// ---------------------------------------------------------------------------
template <class P>
__device__ __forceinline__ void bm_base(const P& f, uint64_t a, uint64_t b, int64_t i, int64_t n, int64_t& l_io,
                                        BmMatrix* M) {
  using W = typename P::W;
  const int lane = threadIdx.x & 31;
  W x = f.load(a), y = lane == 0 ? 0 : f.load(b), Q = 0, V = lane == 0 ? f.load(1) : 0;
  W bb = __shfl_sync(kAll, f.load(b), 0);
  int sb = 0, da = 0, db = 0;
  const int64_t l = l_io;
  const int steps = n - i < kBmK ? (int)(n - i) : kBmK;
  int slack = (int)(i - 2 * l);  // 2 l <= i + k exactly when slack + k >= 0
  int dl = 0;                    // change of l
#pragma unroll 4
  for (int k = 0; k < steps; ++k) {
    const W d = __shfl_sync(kAll, x, k);
    W ys = __shfl_sync(kAll, y, lane - sb), vs = __shfl_sync(kAll, V, lane - sb);
    if (lane < sb) ys = vs = 0;
    if (lane == k) x = k == 0 ? f.load(1) : 0;
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
    M->c[q][lane] = 0;
    if (lane == 0) M->c[q][kBmK] = 0;
  }
  __syncwarp();
  M->c[0][kBmK - lane] = f.store(x);
  M->c[1][kBmK - lane] = f.store(Q);
  if (lane <= db) {
    M->c[2][kBmK - sb - lane] = f.store(y);
    M->c[3][kBmK - sb - lane] = f.store(V);
  }
  if (lane == 0) M->omin = kBmK - (da > sb + db ? da : sb + db);
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Applying a matrix: limb products on the tensor cores (mma_limbs.cuh). A and
// B are kept as L byte planes each (plane q at q * pitch; A's, then B's). A tile
// is 64 consecutive outputs j = base + 4 m + r (m < 16, r < 4) of both A' and
// B': the left operand of the m16n8k32 product has row m = plane bytes from
// base + wb + 4 m on (32 window positions, read as words from shared memory),
// the right one column 2 r + type with the coefficients shifted by r. With the
// usual 17 offsets (16 .. 32) one window of 32 positions covers all; below
// offset 4 it takes two. 2 L^2 instructions per tile: 128 over 2^61 - 1, i.e. 256
// cycles of an SM per 64 outputs, against 1150 on the integer pipes (18 x 4
// multiply-adds at 4 cycles a warp for each of four half products).
// ---------------------------------------------------------------------------
template <int L>
struct BmFrag {
  uint32_t b[2][L][2];  // [source A or B][limb][k half]
};

template <int L>
__device__ __forceinline__ void bm_frag(BmFrag<L>& fr, const BmMatrix& M, int wb) {
  const int lane = threadIdx.x & 31, n = lane >> 2, t = lane & 3;
#pragma unroll
  for (int src = 0; src < 2; ++src)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint64_t* c = M.c[(n & 1) * 2 + src];
      const int o = wb + 4 * t + 16 * h - (n >> 1);
      uint64_t v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = (unsigned)(o + q) < (unsigned)kCoefRows ? c[o + q] : 0;
      uint32_t w[L];
      mml::limb_words<L>(w, v);
#pragma unroll
      for (int i = 0; i < L; ++i) fr.b[src][i][h] = w[i];
    }
}

// Adds the products of the tile at `base` (a multiple of 4) to acc.
template <int L, class I>
__device__ __forceinline__ void bm_tile(uint32_t (&acc)[2 * L - 1][4], const BmFrag<L>& fr, const uint8_t* planes,
                                        I pitch, I pos) {
  const int lane = threadIdx.x & 31;
  const uint8_t* p0 = planes + pos + 4 * ((lane >> 2) + (lane & 3));
#pragma unroll
  for (int src = 0; src < 2; ++src)
#pragma unroll
    for (int i = 0; i < L; ++i) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(p0 + (src * L + i) * pitch);
      const uint32_t a[4] = {w[0], w[8], w[4], w[12]};
#pragma unroll
      for (int j = 0; j < L; ++j) mml::mma_k32(acc[i + j], a, fr.b[src][j][0], fr.b[src][j][1]);
    }
}

// The fragments of a matrix as a warp keeps them, and one tile's residues: v =
// A'(j0), B'(j0), A'(j0 + 32), B'(j0 + 32) with j0 = base + lane.
template <class P>
struct BmApply {
  static constexpr int L = P::L;
  const LimbRed<typename P::F, L>& red;
  const BmMatrix& M;
  BmFrag<L> fr;
  int wb;
  bool two;
  __device__ __forceinline__ BmApply(const LimbRed<typename P::F, L>& r, const BmMatrix& m) : red(r), M(m) {
    wb = M.omin & ~3;
    two = wb == 0;
    bm_frag(fr, M, wb);
  }
  template <class I>
  __device__ __forceinline__ void tile(const uint8_t* planes, I pitch, I base, uint64_t (&v)[4]) {
    uint32_t acc[2 * L - 1][4];
#pragma unroll
    for (int d = 0; d < 2 * L - 1; ++d)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[d][q] = 0;
    bm_tile<L, I>(acc, fr, planes, pitch, base + wb);
    if (two) {
      bm_frag(fr, M, 32);
      bm_tile<L, I>(acc, fr, planes, pitch, base + 32);
      bm_frag(fr, M, 0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = red.residue(acc, q);
  }
};

template <int L, class I>
__device__ __forceinline__ void bm_put(uint8_t* planes, I pitch, I j, uint64_t a, uint64_t b) {
  mml::put_planes1<L>(planes + j, pitch, a);
  mml::put_planes1<L>(planes + L * pitch + j, pitch, b);
}

// Outputs t0 .. lim in place by the `warps` warps of a group (this one: w),
// two tiles per warp and pass: output j is stored at j and reads reach past it
// only, so bar(k), the barrier of pass k, separates the reads from the writes.
template <class P, class I, class Bar>
__device__ __forceinline__ void bm_apply(const LimbRed<typename P::F, P::L>& red, uint8_t* planes, I pitch,
                                         const BmMatrix& M, I t0, int warps, int w, I lim, bool& nz, Bar&& bar) {
  constexpr int kPer = 2;
  const int lane = threadIdx.x & 31;
  if (t0 >= lim) return;
  BmApply<P> ap(red, M);
  for (int k = 0; t0 < lim; ++k, t0 += 64 * kPer * warps) {
    uint64_t v[kPer][4];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const I base = t0 + 64 * (q * warps + w);
      if (base < lim) ap.tile(planes, pitch, base, v[q]);
    }
    bar(k);
#pragma unroll
    for (int q = 0; q < kPer; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const I j = t0 + 64 * (q * warps + w) + 32 * h + lane;
        if (j < lim) {
          bm_put<P::L, I>(planes, pitch, j, v[q][2 * h], v[q][2 * h + 1]);
          nz |= v[q][2 * h] != 0;
        }
      }
  }
}

// ---------------------------------------------------------------------------
// bm_front — the next window (outputs 0 .. 31 as v[0], v[1] of warp 0), on the
// chain of the steps: kParts warps take a source each, with 8 limbs also half
// of its limbs each, and warp 0 adds the parts (barrier 3). Cycles in one warp
// and as it is: 1830 and 980 (8 limbs), 1070 and 805 (4 limbs); with fewer
// limbs one warp is enough.
// ---------------------------------------------------------------------------
template <int L>
constexpr int bm_front_parts() {
  return L == 8 ? 4 : L == 4 ? 2 : 1;
}
template <class P, class I>
__device__ __forceinline__ void bm_front(const LimbRed<typename P::F, P::L>& red, const uint8_t* planes, I pitch,
                                         const BmMatrix& M, uint64_t (*fr)[2][32], int w, uint64_t (&v)[2]) {
  constexpr int L = P::L, kParts = bm_front_parts<L>();
  constexpr int H = kParts == 4 ? L / 2 : L, kSrc = kParts == 1 ? 2 : 1;  // limbs and sources of a warp
  const int lane = threadIdx.x & 31, n = lane >> 2, t = lane & 3;
  const int src0 = w & 1, hi = w >> 1;
  const typename P::F& f = red.field();
  uint32_t acc[2 * L - 1][4];
#pragma unroll
  for (int d = 0; d < 2 * L - 1; ++d)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[d][q] = 0;
  for (int wb = M.omin & ~3; wb <= kBmK; wb += 32) {
#pragma unroll
    for (int k = 0; k < kSrc; ++k) {
      const int src = src0 + k;
      const uint64_t* c = M.c[(n & 1) * 2 + src];
      uint32_t b[2][L];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = wb + 4 * t + 16 * h - (n >> 1);
        uint64_t x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = (unsigned)(o + q) < (unsigned)kCoefRows ? c[o + q] : 0;
        mml::limb_words<L>(b[h], x);
      }
      const uint8_t* p0 = planes + (src * L + hi * H) * pitch + wb + 4 * (n + t);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const uint32_t* x = reinterpret_cast<const uint32_t*>(p0 + i * pitch);
        const uint32_t a[4] = {x[0], x[8], x[4], x[12]};
#pragma unroll
        for (int j = 0; j < L; ++j) mml::mma_k32(acc[i + j], a, b[0][j], b[1][j]);
      }
    }
    if (wb >= 4) break;  // this window covers all offsets
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint64_t x = red.residue(acc, q);
    if (kParts == 4 && hi) x = red.template shifted<8 * (L / 2)>(x);
    v[q] = x;
  }
  if constexpr (kParts == 1) {
    __syncwarp();
  } else {
    if (w != 0) {
      fr[w - 1][0][lane] = v[0];
      fr[w - 1][1][lane] = v[1];
      asm volatile("bar.arrive 3, %0;" ::"n"(32 * kParts) : "memory");
      return;
    }
    asm volatile("bar.sync 3, %0;" ::"n"(32 * kParts) : "memory");
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if constexpr (kParts == 4)
        v[q] = f.add(f.add(v[q], fr[0][q][lane]), f.add(fr[1][q][lane], fr[2][q][lane]));
      else
        v[q] = f.add(v[q], fr[0][q][lane]);
    }
  }
}

// Entry j from its byte planes.
template <int L, class I>
__device__ __forceinline__ uint64_t bm_get(const uint8_t* planes, I pitch, int j) {
  uint64_t v = 0;
#pragma unroll
  for (int i = 0; i < L; ++i) v |= (uint64_t)planes[i * pitch + j] << (8 * i);
  return v;
}

// Entries of A and B of the start: c = b = 1, bb = 1 (src/fp.rs:262-268), so
// A = s and B = 1 + x s.
__device__ __forceinline__ uint64_t bm_b0(const uint64_t* s, int64_t j) { return j ? s[j - 1] : 1; }

// Byte planes of a sequence's residuals: pitch bytes each, past the end as much
// as a tile may read.
constexpr int kBmPad = 160;
__host__ __device__ constexpr int64_t bm_pitch(int64_t n) { return (n + kBmPad + 15) / 16 * 16; }

struct BmShared {
  BmMatrix M[2];
  uint64_t fr[3][2][32];  // parts of the next window
  int64_t l;
  long long job;
  int flag;
};

// Entries [0, n) of the start and zeros behind them, n rounded up to a word.
template <int L, class I>
__device__ __forceinline__ bool bm_start(const uint64_t* __restrict__ s, I n, uint8_t* planes, I pitch) {
  bool nz = false;
  for (I j = 4 * threadIdx.x; j < pitch; j += 4 * blockDim.x) {
    uint64_t a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = j + q < n ? s[j + q] : 0;
      b[q] = j + q < n ? bm_b0(s, j + q) : 0;
      nz |= a[q] != 0;
    }
    mml::put_planes4<L>(planes + j, pitch, a);
    mml::put_planes4<L>(planes + L * pitch + j, pitch, b);
  }
  return nz;
}

// ---------------------------------------------------------------------------
// One sequence with the whole CTA (blockDim a multiple of 32, at least 128):
// the first warps compute the next window, then warp 0 runs the next 32 steps
// while the others apply the matrix. Per block of 32 steps one barrier of the
// whole CTA, and one among the applying warps per pass. planes: 2 L of
// bm_pitch(n) bytes, owned by this CTA. I: int for planes in shared memory,
// int64_t for the workspace, where 8 planes of a sequence of 2^28 pass 2^31.
// ---------------------------------------------------------------------------
template <class I, class P>
__device__ __forceinline__ int64_t bm_run(const P& f, const LimbRed<typename P::F, P::L>& red,
                                          const uint64_t* __restrict__ s, int64_t n64, uint8_t* planes,
                                          BmShared& sh) {
  constexpr int L = P::L;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const I n = (I)n64, pitch = (I)bm_pitch(n64);
  bool nz = bm_start<L>(s, n, planes, pitch);
  int64_t l = 0;
  __syncthreads();
  if (warp == 0)
    bm_base(f, bm_get<L, I>(planes, pitch, lane), bm_get<L, I>(planes + L * pitch, pitch, lane), 0, n, l, &sh.M[0]);
  for (I i = 0;; i += kBmK) {
    // Every thread's part of A (steps i on) has been written and tested, and
    // the block's matrix is there.
    const bool any = __syncthreads_or(nz);
    if (!any || i + kBmK >= n) break;
    nz = false;
    const int par = (int)(i / kBmK) & 1;
    const BmMatrix& m = sh.M[par];
    const I lim = n - i - kBmK;  // outputs
    uint64_t v[2];
    if (warp < bm_front_parts<L>()) bm_front<P, I>(red, planes, pitch, m, sh.fr, warp, v);
    if (warp == 0) {
      // The first pass's writes wait until the front has read its inputs.
      if (lim > kBmK) asm volatile("bar.arrive 1, %0;" ::"r"(T) : "memory");
      if (lane >= lim) v[0] = v[1] = 0;
      nz |= v[0] != 0;
      bm_put<L, I>(planes, pitch, lane, v[0], v[1]);  // read by no other warp before the barrier
      bm_base(f, v[0], v[1], i + kBmK, n, l, &sh.M[par ^ 1]);
    } else {
      bm_apply<P, I>(red, planes, pitch, m, kBmK, T / 32 - 1, warp - 1, lim, nz, [&](int k) {
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

template <class P>
__device__ __noinline__ int64_t bm_any(const BmJob& job, uint64_t* gws, int64_t smem_words, BmShared& sh) {
  extern __shared__ __align__(16) uint64_t bm_smem[];
  const FieldParams fp{job.p, job.mu_lo, job.mu_hi, job.safe_batch};
  const P f(fp);
  const LimbRed<typename P::F, P::L> red{typename P::F(fp)};
  const bool fits = bm_words(P::L, job.n) <= smem_words;
  if (fits) return bm_run<int>(f, red, job.s, job.n, reinterpret_cast<uint8_t*>(bm_smem), sh);
  return bm_run<int64_t>(f, red, job.s, job.n, reinterpret_cast<uint8_t*>(gws), sh);
}

__device__ __forceinline__ int64_t bm_dispatch(const BmJob& job, uint64_t* gws, int64_t smem_words, BmShared& sh) {
  if (job.n <= 0) return 0;
  const uint64_t p = job.p;
  if (p == kM61) return bm_any<BmM61>(job, gws, smem_words, sh);
  if (!(p & 1) || (p >> 31 == 1))
    return p < (1ULL << 32) ? bm_any<BmBarrett<FpSmall, 4>>(job, gws, smem_words, sh)
                            : bm_any<BmBarrett<FpBarrett, 8>>(job, gws, smem_words, sh);
  if (p < (1ULL << 8)) return bm_any<BmMont32<1>>(job, gws, smem_words, sh);
  if (p < (1ULL << 16)) return bm_any<BmMont32<2>>(job, gws, smem_words, sh);
  if (p < (1ULL << 31)) return bm_any<BmMont32<4>>(job, gws, smem_words, sh);
  return bm_any<BmMont64>(job, gws, smem_words, sh);
}

// Plain form: one CTA runs one sequence, A and B in dynamic shared memory when
// they fit, else in the global workspace.
__global__ void __launch_bounds__(512) bm_block_kernel(BmJob job, uint64_t* gws, int64_t smem_words, int64_t* out) {
  __shared__ BmShared sh;
  const int64_t l = bm_dispatch(job, gws, smem_words, sh);
  if (threadIdx.x == 0) *out = l;
}

// Batched form: persistent CTAs take jobs from a device counter; the host
// orders jobs longest first (LPT). Each CTA has smem_words of dynamic shared
// memory and a private global slice of gws_words for jobs that do not fit.
__global__ void __launch_bounds__(512)
    bm_batch_kernel(const BmJob* __restrict__ jobs, int64_t count, unsigned long long* next, uint64_t* gws,
                    int64_t gws_words, int64_t smem_words, int64_t* out) {
  __shared__ BmShared sh;
  for (;;) {
    if (threadIdx.x == 0) sh.job = (long long)atomicAdd(next, 1ULL);
    __syncthreads();
    const long long q = sh.job;
    __syncthreads();
    if (q >= count) break;
    const BmJob job = jobs[q];
    const int64_t l = bm_dispatch(job, gws + (int64_t)blockIdx.x * gws_words, smem_words, sh);
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
  uint8_t* buf;     // [2][2 L][bm_pitch(n)] bytes: parity, A's and B's limb planes
  BmMatrix* ring;   // [2 kBmH]
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

template <class P>
__global__ void __launch_bounds__(kLongThreads, 1) bm_long_kernel(FieldParams fp, LongArgs g) {
  constexpr int L = P::L;
  extern __shared__ __align__(16) uint64_t bm_smem[];
  __shared__ BmShared sh;
  const P f(fp);
  const LimbRed<typename P::F, L> red{typename P::F(fp)};
  const int tid = threadIdx.x, T = kLongThreads, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x;
  const int64_t n = g.n, gpitch = bm_pitch(n);
  uint8_t* planes = reinterpret_cast<uint8_t*>(bm_smem);
  // Entries lo .. lo + len (len a multiple of 4, as is lo) of A and B at the
  // start of superblock s into the planes; whether an A entry is nonzero.
  const auto load = [&](int64_t s, int64_t lo, int len, int pitch) {
    const int64_t left = n - s * kBmT - lo;  // valid entries
    bool nz = false;
    if (s == 0) {
      for (int j = 4 * tid; j < len; j += 4 * T) {
        uint64_t a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[q] = j + q < left ? g.s[lo + j + q] : 0;
          b[q] = j + q < left ? bm_b0(g.s, lo + j + q) : 0;
          nz |= a[q] != 0;
        }
        mml::put_planes4<L>(planes + j, pitch, a);
        mml::put_planes4<L>(planes + L * pitch + j, pitch, b);
      }
    } else {
      const uint8_t* src = g.buf + (s & 1) * 2 * L * gpitch + lo;
      for (int j = 4 * tid; j < len; j += 4 * T) {
        // Bytes past the valid entries are zeroed (the buffer holds older ones).
        const uint32_t mask = j + 4 <= left ? 0xffffffffu : j >= left ? 0u : (1u << (8 * (int)(left - j))) - 1;
#pragma unroll
        for (int q = 0; q < 2 * L; ++q) {
          const uint32_t v = mask ? __ldcg(reinterpret_cast<const unsigned int*>(src + q * gpitch + j)) & mask : 0;
          *reinterpret_cast<uint32_t*>(planes + q * pitch + j) = v;
          if (q < L) nz |= v != 0;
        }
      }
    }
    return nz;
  };

  if (blockIdx.x == 0) {
    // ---------------- the steps -------------------------------------------
    const int pitch = (int)bm_pitch(kBmT);
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
      const bool any = __syncthreads_or(load(s, 0, kBmT, pitch));
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
      const int64_t i0 = s * kBmT;
      const bool feeds = n - i0 > kBmT;  // later steps need the matrices
      if (warp == 0)
        bm_base(f, bm_get<L, int>(planes, pitch, lane), bm_get<L, int>(planes + L * pitch, pitch, lane), i0, n, l, &sh.M[0]);
      for (int h = 0; h < kBmH && i0 + h * kBmK < n; ++h) {
        __syncthreads();
        const BmMatrix& m = sh.M[h & 1];
        const int lim = kBmT - (h + 1) * kBmK;  // outputs inside the window
        const bool more = lim > 0 && i0 + (h + 1) * kBmK < n;
        uint64_t v[2];
        if (more && warp < bm_front_parts<L>()) bm_front<P, int>(red, planes, pitch, m, sh.fr, warp, v);
        if (warp == 0) {
          if (more) {
            if (lim > kBmK) asm volatile("bar.arrive 1, %0;" ::"r"(T - 32) : "memory");
            bm_put<L, int>(planes, pitch, lane, v[0], v[1]);
            bm_base(f, v[0], v[1], i0 + (h + 1) * kBmK, n, l, &sh.M[(h & 1) ^ 1]);
          }
        } else if (warp == T / 32 - 1) {
          if (feeds) {
            // The last warp publishes: 16-byte words of the matrix, then the count.
            const int64_t q = s * kBmH + h;
            const uint4* src = reinterpret_cast<const uint4*>(&m);
            uint4* dst = reinterpret_cast<uint4*>(g.ring + q % (2 * kBmH));
            for (int w = lane; w < (int)(sizeof(BmMatrix) / 16); w += 32) __stcg(dst + w, src[w]);
            __threadfence();
            __syncwarp();
            if (lane == 0 && !(q == 0 && g.skip_cta == 0)) atomicAdd(&g.gs->pub, 1u);
          }
        } else if (more) {
          bool unused = false;
          bm_apply<P, int>(red, planes, pitch, m, kBmK, T / 32 - 2, warp - 1, lim, unused, [&](int k) {
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
  const int pitch = (int)bm_pitch(g.cap + kBmT);
  unsigned int want_done = 0;
  for (int64_t s = 0;; ++s) {
    const LongPlan plan(n, s, G, g.cap);
    if (plan.nout == 0) return;
    for (int c = wk; c < plan.chunks; c += G - 1) {
      if (tid == 0) sh.flag = long_wait(&g.gs->done, want_done, g.gs, g.spin);
      __syncthreads();
      if (!sh.flag) return;
      int64_t lo, hi;
      plan.range(c, lo, hi);
      const int len = (int)(hi - lo);
      load(s, lo, (len + kBmT + 3) / 4 * 4, pitch);
      bool nz = false;
      for (int h = 0; h < kBmH; ++h) {
        const int64_t q = s * kBmH + h;
        if (tid == 0) sh.flag = long_wait(&g.gs->pub, (unsigned)(q + 1), g.gs, g.spin);
        __syncthreads();  // also: the previous matrix has been applied
        if (!sh.flag) return;
        const uint4* src = reinterpret_cast<const uint4*>(g.ring + q % (2 * kBmH));
        uint4* dst = reinterpret_cast<uint4*>(&sh.M[0]);
        for (int w = tid; w < (int)(sizeof(BmMatrix) / 16); w += T) dst[w] = __ldcg(src + w);
        __syncthreads();
        nz = false;
        bm_apply<P, int>(red, planes, pitch, sh.M[0], 0, T / 32, warp, len + kBmT - (h + 1) * kBmK, nz,
                    [](int) { __syncthreads(); });
      }
      __syncthreads();
      uint8_t* dst = g.buf + ((s + 1) & 1) * 2 * L * gpitch + lo;
      for (int j = 4 * tid; j < len; j += 4 * T)
#pragma unroll
        for (int q = 0; q < 2 * L; ++q) {
          // A chunk's last word may reach into the next chunk's.
          const uint8_t* w = planes + q * pitch + j;
          uint8_t* d = dst + q * gpitch + j;
          if (j + 4 <= len)
            __stcg(reinterpret_cast<unsigned int*>(d), *reinterpret_cast<const unsigned int*>(w));
          else
            for (int e = 0; j + e < len; ++e) d[e] = w[e];
        }
      __threadfence();
      const bool any = __syncthreads_or(nz);
      if (tid == 0 && !(s == 0 && (int)blockIdx.x == g.skip_cta)) {
        if (any) atomicOr(g.nz + s + 1, 1u);
        __threadfence();
        if (c < plan.front) atomicAdd(&g.gs->front, 1u);
        atomicAdd(&g.gs->done, 1u);
      }
    }
    want_done += plan.chunks;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host launchers.
// ---------------------------------------------------------------------------
static int bm_limbs(uint64_t p) {
  if (p >= (1ULL << 32)) return 8;
  if (!(p & 1) || p >= (1ULL << 16)) return 4;
  return p < (1ULL << 8) ? 1 : 2;
}
int64_t bm_smem_words(uint64_t p, int64_t n) { return bm_words(bm_limbs(p), n); }
int64_t bm_workspace_words(int64_t n) { return bm_words(8, n); }

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

// The batch kernel's dynamic shared memory cap is set once per device to the largest
// size any batch asks for (200 KiB), so launches of any batch, graph-captured
// ones included, need no attribute call.
static cudaError_t bm_batch_attr() {
  static PerDevice once;
  return allow_smem(once, bm_batch_kernel, 200 * 1024);
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
static size_t long_ring() { return (2 * kBmH * sizeof(BmMatrix) + 255) / 256 * 256; }

size_t bm_long_bytes(uint64_t p, int64_t n) {
  return 256 + long_flags(n) + long_ring() + (size_t)4 * bm_limbs(p) * bm_pitch(n);
}
int bm_long_err_offset() { return (int)offsetof(LongSync, err); }

// Cycles that a wait may take beyond its base limit, per output of a working
// CTA: a wait can span one sweep of all outputs, measured at 330 cycles an
// output and CTA over 2^63 - 25 (180 over 2^61 - 1, 36 mod 65521), twice that
// where a matrix takes two windows.
constexpr long long kSweepCycles = 3000;

template <class P>
static cudaError_t launch_long_t(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, bool cluster,
                                 void* ws, long long spin, int skip_cta, int64_t* d_out, cudaStream_t st) {
  char* w = static_cast<char*>(ws);
  LongArgs a{};
  a.s = s;
  a.n = n;
  a.gs = reinterpret_cast<LongSync*>(w);
  a.nz = reinterpret_cast<unsigned int*>(w + 256);
  a.ring = reinterpret_cast<BmMatrix*>(w + 256 + long_flags(n));
  a.buf = reinterpret_cast<uint8_t*>(w + 256 + long_flags(n) + long_ring());
  a.out = d_out;
  a.spin = skip_cta >= 0 ? spin : spin + kSweepCycles * (n / (ctas - 1));
  a.skip_cta = skip_cta;
  // The largest chunk: the first superblock's share, within the shared memory.
  const int64_t front = std::min<int64_t>(std::max<int64_t>(n - kBmT, 0), kBmT);
  const int64_t fchunks = (front + kBmFront - 1) / kBmFront;
  const int64_t rest = std::max<int64_t>(n - 2 * kBmT, 0);
  const int64_t share = std::max<int64_t>(ctas - 1 - fchunks, 1);
  const int64_t room = kLongSmem / (2 * P::L) - kBmT - kBmPad - 16;
  int64_t cap = ((rest + share - 1) / share + 31) / 32 * 32;
  cap = std::max<int64_t>(std::min(cap, room / 32 * 32), kBmFront);
  a.cap = (int)cap;
  const size_t smem = (size_t)2 * P::L * bm_pitch(cap + kBmT);
  cudaError_t e = cudaFuncSetAttribute(bm_long_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(ws, 0, 256 + long_flags(n), st);
  if (e != cudaSuccess) return e;
  if (!cluster) {
    FieldParams f = fp;
    void* args[] = {&f, &a};
    return cudaLaunchCooperativeKernel((void*)bm_long_kernel<P>, dim3(ctas), dim3(kLongThreads), args, smem, st);
  }
  if (ctas > 8) {
    e = cudaFuncSetAttribute(bm_long_kernel<P>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
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
  e = cudaOccupancyMaxActiveClusters(&nclusters, bm_long_kernel<P>, &cfg);
  if (e != cudaSuccess) return e;
  if (nclusters < 1) return cudaErrorInvalidConfiguration;
  return cudaLaunchKernelEx(&cfg, bm_long_kernel<P>, fp, a);
}

static cudaError_t launch_long(const FieldParams& fp, const uint64_t* s, int64_t n, int ctas, bool cluster, void* ws,
                               long long spin, int skip_cta, int64_t* d_out, cudaStream_t st) {
  const uint64_t p = fp.p;
#define MODLIN_LONG(P) launch_long_t<P>(fp, s, n, ctas, cluster, ws, spin, skip_cta, d_out, st)
  using Even32 = BmBarrett<FpSmall, 4>;
  using Even64 = BmBarrett<FpBarrett, 8>;
  if (p == kM61) return MODLIN_LONG(BmM61);
  if (!(p & 1) || (p >> 31 == 1)) return p < (1ULL << 32) ? MODLIN_LONG(Even32) : MODLIN_LONG(Even64);
  if (p < (1ULL << 8)) return MODLIN_LONG(BmMont32<1>);
  if (p < (1ULL << 16)) return MODLIN_LONG(BmMont32<2>);
  if (p < (1ULL << 31)) return MODLIN_LONG(BmMont32<4>);
  return MODLIN_LONG(BmMont64);
#undef MODLIN_LONG
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
