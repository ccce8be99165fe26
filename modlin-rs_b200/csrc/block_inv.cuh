// Inverse of a 64 x 64 block of residues by one CTA.
//
// In-place Gauss-Jordan by 16-column blocks, fraction-free. Before block step
// k the rows from 16 k on are s times those of the unscaled elimination (s the
// product of the earlier d); the step inverts their diagonal block as
// numerators N and one scalar d (A_kk^-1 = N / d) and sets
//   rows k:      A_k* <- T = N A_k*,              A_kk <- s N,
//   other rows:  A_i* <- d A_i* - A_ik T,         A_ik <- -A_ik (s N),
// which scales every other row by d. In the end row block k is P^-1's times
// the product of d_k and the later d: the caller multiplies it by fac[k],
// (d_0 .. d_(k-1)) / (d_0 .. d_3). The one modular inverse runs beside the last
// update. The products (K = 16) are limb products on the tensor cores
// (mma_limbs.cuh); the diagonal blocks are eliminated the same way entry by
// entry (one thread an entry, one barrier a column: the dependent chain of the
// whole inverse), swapping rows inside the 16 when a pivot is zero. A block
// whose 16 rows have no pivot is left to the caller (P singular, or for about
// 4 / p of the invertible ones).
#pragma once
#include <cstdint>
#include <type_traits>

#include "field.cuh"
#include "mma_limbs.cuh"

namespace modlin {

// comb = bb a + nd b mod p on the elimination's working form.
template <class F>
struct ElimField {
  using W = uint64_t;
  F f;
  __device__ explicit ElimField(const F& g) : f(g) {}
  __device__ __forceinline__ W in(uint64_t x) const { return x; }
  __device__ __forceinline__ uint64_t out(W x) const { return x; }
  __device__ __forceinline__ W neg(W x) const { return f.modulus() - x; }
  __device__ __forceinline__ bool zero(W x) const { return x == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const { return f.reduce2(f.prod(bb, a) + f.prod(nd, b)); }
};
// Two products of 32-bit residues in 64 bits and a carry.
template <>
struct ElimField<FpSmall> {
  using W = uint64_t;
  FpSmall f;
  uint64_t r64;  // 2^64 mod p
  __device__ explicit ElimField(const FpSmall& g) : f(g) {
    const uint64_t r = 0 - g.wide.mu_hi * g.wide.p;  // 2^64 - floor((2^64 - 1) / p) p, in [1, p]
    r64 = r == g.wide.p ? 0 : r;
  }
  __device__ __forceinline__ W in(uint64_t x) const { return x; }
  __device__ __forceinline__ uint64_t out(W x) const { return x; }
  __device__ __forceinline__ W neg(W x) const { return f.wide.p - x; }
  __device__ __forceinline__ bool zero(W x) const { return x == 0; }
  __device__ __forceinline__ W comb(W bb, W a, W nd, W b) const {
    const uint64_t u = (uint64_t)(uint32_t)bb * (uint32_t)a, s = u + (uint64_t)(uint32_t)nd * (uint32_t)b;
    const uint64_t v = f.reduce64(s);
    return s < u ? f.add(v, r64) : v;
  }
};
template <>
struct ElimField<FpM61> : M61Halves {
  __device__ explicit ElimField(const FpM61&) {}
  __device__ __forceinline__ W in(uint64_t x) const { return split(x); }
  __device__ __forceinline__ uint64_t out(W x) const { return value(x); }
};

constexpr int kInvLd = 66;  // words per row of the block (even: 16-byte aligned rows)

template <int LIMBS>
struct InvScratch {
  alignas(16) uint8_t a[LIMBS][48][16];   // A_ik: other rows x block columns
  alignas(16) uint8_t r[LIMBS][48][16];   // A_k*: other columns x block rows
  alignas(16) uint8_t b[LIMBS][64][16];   // T and N: columns x block rows
  alignas(16) uint8_t nn[LIMBS][16][16];  // N
  uint64_t w[2][16][17];
  uint64_t pre[17];  // products of the first pivots of the diagonal block
  uint64_t d[4], fac[4], scale;
  uint8_t order[64];  // slot c of the eliminated block holds its row order[c]
  int ok;
};

// M (64 rows of kInvLd words in shared memory) -> numerators of row block k to
// be multiplied by S.fac[k]. The inverse is of the block with rows in S.order.
// Returns false (the same in every thread) when a pivot block has no
// pivot; M is then spoilt. NT: threads (a multiple of 32, at least 256), all
// calling; M is complete before the call (a barrier of the caller's).
template <class F, int LIMBS, int NT>
__device__ bool inv64(const F& f, const LimbRed<F, LIMBS>& red, uint64_t* M, InvScratch<LIMBS>& S) {
  using E = ElimField<F>;
  using W = typename E::W;
  const E ef(f);
  const uint64_t p = f.modulus();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = NT / 32;
  constexpr int kPl48 = 48 * 16, kPl64 = 64 * 16, kPl16 = 16 * 16;
  for (int c = tid; c < 64; c += NT) S.order[c] = (uint8_t)c;
  if (tid == 0) S.ok = 1;
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    const int kb = 16 * k;
    const auto other = [kb](int n) { return n < kb ? n : n + 16; };  // the 48 rows or columns outside the block
    // Planes of A_ik, and the diagonal block.
    for (int t = tid; t < 192; t += NT) {
      const int i = t >> 2, k4 = 4 * (t & 3);
      const uint64_t* src = M + other(i) * kInvLd + kb + k4;
      const uint64_t v[4] = {src[0], src[1], src[2], src[3]};
      mml::put_planes4<LIMBS>(&S.a[0][i][k4], kPl48, v);
    }
    const int j = (tid >> 4) & 15, i = tid & 15;
    if (tid < 256) {
      if (tid == 0) S.pre[0] = ef.in(1);
      S.w[0][j][i] = ef.in(M[(kb + j) * kInvLd + kb + i]);
      bool ok = true;
#pragma unroll 1
      for (int c = 0; c < 16; ++c) {
        asm volatile("bar.sync 1, 256;" ::: "memory");
        W(*cur)[17] = S.w[c & 1];
        W e = cur[c][c], h = cur[j][c], x = cur[j][i], m = cur[c][i];
        const W sc = S.pre[c];
        if (ef.zero(e)) {  // the same in all 256 threads
          int pv = -1;
          for (int q = 15; q > c; --q)
            if (!ef.zero(cur[q][c])) pv = q;
          if (pv < 0) {
            ok = false;
            break;
          }
          const W y = cur[j == c ? pv : j == pv ? c : j][i];
          asm volatile("bar.sync 1, 256;" ::: "memory");
          cur[j][i] = y;
          if (tid == 0) {
            const uint8_t o = S.order[kb + c];
            S.order[kb + c] = S.order[kb + pv];
            S.order[kb + pv] = o;
          }
          asm volatile("bar.sync 1, 256;" ::: "memory");
          e = cur[c][c];
          h = cur[j][c];
          x = y;
          m = cur[c][i];
        }
        // Entry (j, i) <- e x - h m; in column c -h s, in row c as it was, s
        // at the pivot (s: the product of the earlier pivots), whose thread
        // takes the next product e s instead.
        const bool in_c = i == c;
        const W v = ef.comb(in_c && j != c ? (W)0 : e, in_c ? sc : x, j == c ? (W)0 : ef.neg(h), in_c ? sc : m);
        S.w[(c & 1) ^ 1][j][i] = j != c ? v : in_c ? sc : x;
        if (j == c && in_c) S.pre[c + 1] = v;
      }
      if (!ok) {
        if (tid == 0) S.ok = 0;
      } else {
        // Row j is A_kk^-1's times the product of its pivot and the later ones.
        const uint64_t v = f.mul(ef.out(S.w[0][j][i]), ef.out(S.pre[j]));  // step 15 wrote buffer 0
        const uint64_t sv = k ? f.mul(v, S.scale) : v;
        M[(kb + j) * kInvLd + kb + i] = sv;
        mml::put_planes1<LIMBS>(&S.nn[0][j][i], kPl16, v);
        mml::put_planes1<LIMBS>(&S.b[0][48 + i][j], kPl64, sv);
      }
    }
    __syncthreads();
    if (!S.ok) return false;
    // Planes of A_k* in the rows' order; d.
    for (int t = tid; t < 192; t += NT) {
      const int n = t >> 2, k4 = 4 * (t & 3);
      const uint64_t* src = M + other(n);
      uint64_t v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = src[S.order[kb + k4 + q] * kInvLd];
      mml::put_planes4<LIMBS>(&S.r[0][n][k4], kPl48, v);
    }
    if (tid == NT - 1) S.d[k] = ef.out(S.pre[16]);
    __syncthreads();
    uint32_t acc[2 * LIMBS - 1][4];
    const int g = lane >> 2, t2 = 2 * (lane & 3);
    for (int q = warp; q < 6; q += NW) {  // T = N A_k*
      mml::tile_k16<LIMBS>(acc, mml::saddr(S.nn), kPl16, mml::saddr(&S.r[0][8 * q][0]), kPl48);
      uint64_t v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = red.residue(acc, e);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = g + 8 * (e >> 1), n = 8 * q + t2 + (e & 1);
        M[(kb + row) * kInvLd + other(n)] = v[e];
        mml::put_planes1<LIMBS>(&S.b[0][n][row], kPl64, v[e]);
      }
    }
    __syncthreads();
    const uint64_t d = S.d[k];
    // The last update leaves one warp to the inverse of the common factor.
    const int nw = k == 3 ? NW - 1 : NW;
    if (warp < nw) {
      for (int q = warp; q < 24; q += nw) {
        const int rg = q >> 3, ng = q & 7;
        // Columns 2 t and 2 t + 1 are neighbours in M, 16-byte aligned.
        const int n = 8 * ng + t2, col = ng < 6 ? other(n) : kb + n - 48;
        ulonglong2* m0 = reinterpret_cast<ulonglong2*>(M + other(16 * rg + g) * kInvLd + col);
        ulonglong2* m1 = reinterpret_cast<ulonglong2*>(M + other(16 * rg + g + 8) * kInvLd + col);
        const ulonglong2 x0 = *m0, x1 = *m1;
        const uint64_t dd = ng < 6 ? d : 0;
        mml::tile_k16<LIMBS>(acc, mml::saddr(&S.a[0][16 * rg][0]), kPl48, mml::saddr(&S.b[0][8 * ng][0]), kPl64);
        *m0 = make_ulonglong2(red.mul_sub(dd, x0.x, acc, 0), red.mul_sub(dd, x0.y, acc, 1));
        *m1 = make_ulonglong2(red.mul_sub(dd, x1.x, acc, 2), red.mul_sub(dd, x1.y, acc, 3));
      }
    } else if (lane == 0) {
      const uint64_t d01 = f.mul(S.d[0], S.d[1]), d012 = S.scale, all = f.mul(d012, d);
      const uint64_t inv = std::is_same<F, FpM61>::value ? fp_inv_m61(all) : fp_inv_binary(all, p);
      S.fac[0] = inv;
      S.fac[1] = f.mul(inv, S.d[0]);
      S.fac[2] = f.mul(inv, d01);
      S.fac[3] = f.mul(inv, d012);
    }
    __syncthreads();
    if (tid == 0) S.scale = k ? f.mul(S.scale, d) : d;  // read after the next barrier of all threads
  }
  return true;
}

}  // namespace modlin
