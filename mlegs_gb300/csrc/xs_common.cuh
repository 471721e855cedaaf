// xs_common.cuh — arithmetic of the exact-slice (Ozaki) tensor-core contractions shared by
// xs_radial.cu and xs_vec2tp.cu.
//
// A value x with |x| < 2^E becomes the integer X = round(x 2^(nb - E)) of nb = w NS bits (|X| <= 2^nb),
// and X is cut into NS two's-complement digits of w bits, most significant first:
//   X = d_0 2^(w (NS-1)) + sum_{s>0} d_s 2^(w (NS-1-s)),  d_0 = X >> w (NS-1) in [-2^w, 2^w],
//   d_s in [0, 2^w) for s > 0.
// Every digit is an exact BF16 and every digit product an exact FP32 integer of magnitude <= 2^(2w), so
// a K-term sum of the products of one digit order stays exact while K (pairs of the order) 2^(2w) < 2^24.
// Balanced digits (nb = 63): the digits after the first lie in [-2^(w-1), 2^(w-1)) and the first, of
// eight bits, in [-128, 128), so a digit product is at most 2^(2w-2) (2^(w+6) with one first digit, 2^14 with two) and
// the order sums stay exact for 8 digits of 8 bits up to K = 128 and for 9 of 7 bits up to K = 372, half of that where an
// order holds two products (xs_order_bound; unsigned digits need 9 of 7 bits up to K = 113 and 10 of 6, 60 bits, beyond).
// The first digit needs |X| < 2^63 - 2^56, so that the carry of the digits below it does not leave its eight bits: the
// scale E of a row or column whose largest magnitude has its upper six fraction bits set is one larger
// (xs_ebound_bal).
// All conversions run on the integer and FP32 pipes: GB300 issues FP64 at about 2 operations per clock
// per SM.
#pragma once
#include "common.cuh"
#include <cmath>
#include <cstdint>
#include <type_traits>

namespace mlg {

// exponent bound of a magnitude bit pattern: |v| < 2^E for E = exponent field - 1022
__device__ __forceinline__ int xs_ebound(unsigned long long absbits) { return (int)(absbits >> 52) - 1022; }

// x 2^(nb - E) rounded to the nearest integer (halves away from zero) for |x| < 2^E (nb <= 63), from
// the FP64 bit pattern; zero, subnormal and non-finite inputs and E <= -2000 (an all-zero row or
// column) give 0.  Rounding, not truncation: a truncated fixed-point operand carries a one-signed bias
// of half a unit, and a K-term contraction against a table of one sign sums it coherently (K units
// instead of sqrt(K)), which the inverse Laplacian of the projection's chi then magnified.
__device__ __forceinline__ long long xs_fix(double x, int E, int nb) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7FF);
  if (e == 0 || e == 0x7FF || E <= -2000) return 0;
  const unsigned long long M = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = e - 1075 + nb - E;     // |x| 2^(nb - E) = M 2^sh, and M 2^sh < 2^nb
  unsigned long long X;
  if (sh >= 0) X = (sh <= 10) ? (M << sh) : 0ull;  // sh < nb - 52 <= 11 when |x| < 2^E
  else X = (sh > -63) ? ((M + (1ull << (-sh - 1))) >> (-sh)) : 0ull;
  return (b >> 63) ? -(long long)X : (long long)X;
}

// What FP32 accumulates exactly, and the largest magnitude that an order of ns balanced digits of w bits can reach with `products`
// products per digit pair over K terms: order d has d + 1 pairs, two of them (one, for d = 0) with a first digit
constexpr double XS_EXACT = 16777216.0;
__host__ __device__ constexpr double xs_order_bound(int ns, int w, int products, int K) {
  const double first = 128.0, other = (double)(1 << (w - 1));
  double most = first * first;
  for (int d = 1; d < ns; ++d) {
    const double v = 2.0 * first * other + (d - 1) * other * other;
    most = v > most ? v : most;
  }
  return most * products * K;
}

// exponent bound for balanced digits from a magnitude's high word: |v| < 2^E (1 - 2^-7)
__device__ __forceinline__ int xs_ebound_bal(unsigned abshi) { return (int)((abshi + 0x4000u) >> 20) - 1022; }

// the scale of a plain-form column that holds a non-finite sample: every value of it gives 0 (xs_fix_base), and its outputs come
// from elsewhere
constexpr int XS_NONFIN = 4096;
__device__ __forceinline__ bool xs_nonfin(unsigned abshi) { return abshi >= 0x7FF00000u; }   // a largest magnitude's high word

// the shift base of xs_fixs for a scale E; `ok` false (no column, or an all-zero one): every value gives 0
__device__ __forceinline__ int xs_fix_base(int E, int nb, bool ok) { return ok && E > -2000 ? 1085 - nb + E : (1 << 20); }
// xs_fix with the shift base worked out once per column.  The significand starts at bit 63 and is shifted right only
// (by base - exponent >= 0, clamped to 64 by the instruction) with one bit to spare, which the rounding consumes:
// halves go away from zero, as in xs_fix.
__device__ __forceinline__ long long xs_fixs(double x, int base) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7FFu);
  int r = base - e;
  if ((unsigned)(e - 1) >= 0x7FEu) r = 64;   // zero, subnormal, non-finite
  const unsigned mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, ml = lo << 11;
  unsigned long long M = ((unsigned long long)mh << 32) | ml, X;
  asm("shr.u64 %0, %1, %2;" : "=l"(X) : "l"(M), "r"(r));
  X = (X + 1) >> 1;
  const long long sg = (long long)((int)hi >> 31);
  return (long long)(X ^ (unsigned long long)sg) - sg;
}

// the offset that makes every balanced digit non-negative: 2^(w-1) in the place of each digit, 128 in the first one's
template <int NS, int W> __host__ __device__ constexpr unsigned long long xs_bias() {
  unsigned long long b = 128ull << (W * (NS - 1));
  for (int s = 0; s < NS - 1; ++s) b += (1ull << (W - 1)) << (W * s);
  return b;
}
// a.x - c, a.y - c for the two FP32 bit patterns a0, a1, in one instruction; returned as a packed BF16 pair (the
// results are small integers, so their BF16 patterns are their upper halves)
__device__ __forceinline__ uint32_t xs_sub2_pack(uint32_t a0, uint32_t a1, float c) {
  unsigned long long v, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a0), "r"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(-c), "f"(-c));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(v), "l"(d));
  return __byte_perm((uint32_t)v, (uint32_t)(v >> 32), 0x7632);
}
// digit S of the values X0, X1 (balanced: X + xs_bias) as a packed BF16 pair (X0 low): the digit's bits are put into
// the fraction of 2^23, and one packed FP32 subtraction takes 2^23 (and the balanced digit's offset) away again
template <int NS, int W, bool BAL, int S> __device__ __forceinline__ uint32_t xs_digit2(unsigned long long X0, unsigned long long X1) {
  constexpr int SH = W * (NS - 1 - S);
  static_assert(!BAL || W * (NS - 1) == 56, "the first balanced digit is the upper byte");
  if constexpr (BAL && (W == 8 || S == 0)) {   // digits that are bytes
    constexpr unsigned sel = 0x7440u + (SH & 31) / 8;
    const unsigned a = SH >= 32 ? (unsigned)(X0 >> 32) : (unsigned)X0, b = SH >= 32 ? (unsigned)(X1 >> 32) : (unsigned)X1;
    return xs_sub2_pack(__byte_perm(a, 0x4B000000u, sel), __byte_perm(b, 0x4B000000u, sel), 8388608.0f + 128.0f);
  } else if constexpr (BAL || S > 0) {
    constexpr unsigned mask = (1u << W) - 1u;
    return xs_sub2_pack(((unsigned)(X0 >> SH) & mask) | 0x4B000000u, ((unsigned)(X1 >> SH) & mask) | 0x4B000000u,
                        8388608.0f + (BAL ? (float)(1 << (W - 1)) : 0.0f));
  } else {   // the signed first digit
    return xs_sub2_pack(0x4B400000u + (unsigned)(int)((long long)X0 >> SH), 0x4B400000u + (unsigned)(int)((long long)X1 >> SH),
                        12582912.0f);
  }
}

// |X0| and |X1| (|X| < 2^63) in units of 2^32 as a packed BF16 pair: the operands of a contraction's magnitude sum
__device__ __forceinline__ uint32_t xs_mag2(long long X0, long long X1) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"((float)(int)(X1 >> 32)), "f"((float)(int)(X0 >> 32)));
  return r & 0x7FFF7FFFu;
}
// Where the digits of a plain contraction of K terms are too few.  Their error, the dropped orders and the rounding of the
// operands, is 2^-61.9 sqrt(K / 96) of 2^(row scale + column scale) in the root mean square (measured over K = 96..372); an FP64
// sum rounds K times by up to 2^-53 of S = sum |terms|.  The magnitude sum S is contracted beside the digits as one more digit
// product (xs_mag2), and outputs whose S is so small that the digits' error would pass one such rounding, 2^-53 S, are summed
// again in FP64 (k_xs_again, k_xv_again).  The least S in units of 2^-62 2^(row scale + column scale), those of the products of
// xs_mag2.
constexpr int XS_AGAIN = 4861, XS_AGAIN_T = 256;   // their warps (about 32 an SM) and threads per CTA
inline float xs_least_sum(int K) { return (float)(std::exp2(62.0 - 8.9) * std::sqrt(K / 96.0)); }

// the exact integer value of an FP32 accumulator entry (integral, |x| < 2^24)
__device__ __forceinline__ int xs_f2i(float x) { return __float2int_rn(x); }

// f(std::integral_constant<int, 0>()), ..., f(std::integral_constant<int, N-1>())
template <int I, int N, class F> __device__ __forceinline__ void xs_static_for_(F& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>());
    xs_static_for_<I + 1, N>(f);
  }
}
template <int N, class F> __device__ __forceinline__ void xs_static_for(F f) { xs_static_for_<0, N>(f); }

// x 2^s for s >= 0, floor(x 2^s) for s < 0
__device__ __forceinline__ long long xs_shl(long long x, int s) { return s >= 0 ? (x << s) : (x >> (-s)); }

// T 2^e2 rounded once to FP64 (round to nearest even), T a signed 64-bit integer; magnitudes below the
// normal range flush to zero.  Branch-free on the integer pipe: normalise |T| so that its top bit is
// bit 63, keep 53 bits, round on the 11 below them, and let the implicit bit (and a rounding carry)
// add into the exponent field.
__device__ __forceinline__ double xs_i64_to_double(long long T, int e2) {
  const unsigned long long sign = (unsigned long long)T & 0x8000000000000000ull;
  const unsigned long long a = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
  const int lz = __clzll((long long)a);
  const unsigned long long n = a << (lz & 63);                    // bit 63 set (a != 0)
  unsigned long long m = n >> 11;                                 // 53 bits, the implicit one on top
  const unsigned long long rb = (n >> 10) & 1ull, st = (n & 0x3FFull) != 0ull;
  m += rb & (st | (m & 1ull));
  const long long ex = (long long)(1023 + 63 - lz + e2);          // biased exponent of 2^(top bit)
  const unsigned long long bits = ((unsigned long long)(ex - 1) << 52) + m;
  if (a == 0ull || ex <= 0) return __longlong_as_double((long long)sign);
  if (ex >= 2047) return __longlong_as_double((long long)(sign | 0x7FF0000000000000ull));
  return __longlong_as_double((long long)(sign | bits));
}

}  // namespace mlg
