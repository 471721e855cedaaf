// fft_fixed.cuh — complex arithmetic in 64-bit fixed point for the plain form's FFTs (fftq.cu, fftqr.cu)
#pragma once
#include "fft_common.cuh"

namespace mlg {

struct qc { long long x, y; };   // a complex fixed-point value
__device__ __forceinline__ qc q_add(qc a, qc b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ qc q_sub(qc a, qc b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ qc q_conj(qc a) { return {a.x, -a.y}; }
__device__ __forceinline__ qc q_muli(qc a, int sgn) { return sgn > 0 ? qc{-a.y, a.x} : qc{a.y, -a.x}; }   // a (sgn i)

// x w for |x| <= 2^62 and a real constant w = (WH 2^31 + WL) 2^-61 below 1: with x = xh 2^31 + xl the products xh WH, xh WL
// and xl WH are summed in their places and xl WL, less than two units, is replaced by its mean WL / 2 (it spreads by 0.58
// units at most); the middle terms are rounded at the unit
template <int WH, int WL> __host__ __device__ __forceinline__ long long q_mulc(long long x) {
  const int xh = (int)(x >> 31), xl = (int)((unsigned)x & 0x7FFFFFFFu);
  const long long m = (long long)xh * WL + (long long)xl * WH + ((1ll << 29) + (WL >> 1));
  return (((long long)xh * WH) << 1) + (m >> 30);
}
// v w for a twiddle w = ((wx + i wy) 2^31 + (wz + i ww)) 2^-61 (low parts in [0, 2^31), or both parts of a component
// negated); |v| <= 2^61.5, so that the four middle products stay below 2^63
__host__ __device__ __forceinline__ qc q_mul(qc v, int4 w) {
  const int xh = (int)(v.x >> 31), xl = (int)((unsigned)v.x & 0x7FFFFFFFu);
  const int yh = (int)(v.y >> 31), yl = (int)((unsigned)v.y & 0x7FFFFFFFu);
  // (halves first: the low parts' difference can pass 32 bits where one is negated)
  long long a = (long long)((w.z >> 1) - (w.w >> 1)) + (1ll << 29), b = (long long)((w.z >> 1) + (w.w >> 1)) + (1ll << 29);
  a += (long long)xh * w.z; a += (long long)xl * w.x; a -= (long long)yh * w.w; a -= (long long)yl * w.y;
  b += (long long)xh * w.w; b += (long long)xl * w.y; b += (long long)yh * w.z; b += (long long)yl * w.x;
  return {(((long long)xh * w.x - (long long)yh * w.y) << 1) + (a >> 30),
          (((long long)xh * w.y + (long long)yh * w.x) << 1) + (b >> 30)};
}
__device__ __forceinline__ int4 q_tw(const int4* __restrict__ tw, int idx, int sgn) {   // tables hold exp(-2 pi i k / L)
  int4 w = __ldg(tw + idx);
  if (sgn > 0) { w.y = -w.y; w.w = -w.w; }
  return w;
}

// a line's scale: samples x_n become x_n 2^(NB - e1) for the first pass and are shifted right by sh after it, so that a
// result of 2^(NB - e) is 1
struct QScale { int e1, sh; };
// a thread's share of its line's statistics: the largest magnitude's high word, and the sum of the magnitudes in units of
// the largest one's power of two, in FP32 (the double's upper bits moved into place; what is 2^126 smaller counts as 0)
struct QStat { unsigned mx; float s; };
template <int N> __device__ __forceinline__ QStat q_stat(const double2* d) {
  QStat q{0u, 0.f};
#pragma unroll
  for (int i = 0; i < N; ++i)
    q.mx = max(q.mx, max((unsigned)__double2hiint(d[i].x) & 0x7FFFFFFFu, (unsigned)__double2hiint(d[i].y) & 0x7FFFFFFFu));
  const int sub = (int)(q.mx & 0x7FF00000u) - (126 << 20);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    q.s += __int_as_float(max((__double2hiint(d[i].x) & 0x7FFFFFFF) - sub, 0) << 3);
    q.s += __int_as_float(max((__double2hiint(d[i].y) & 0x7FFFFFFF) - sub, 0) << 3);
  }
  return q;
}

}  // namespace mlg
