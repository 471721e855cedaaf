// fftqr.cu — the plain form's FFTs in 64-bit fixed point (fftq.cu) of lengths that are no power of two: L = R1 R2 with R1 of 8, 9,
// 10, 12, 15, 16 and R2 of 2..6, 8, 9, 10, 12, 15, 16, from 18 to 240 points, in FFTE's conventions (fft.cu).
//
// Scaling, rounding and the lines that take the FP64 transform are as in fftq.cu; lines of 80 points and more have the finer
// unit of their own in the first pass, up to and with the twiddles between the passes.  The rounding is a quarter of the FP64
// transforms' (whose twiddle angles are rounded besides): in units of 2^-53 of a line's root mean square, FP64 beside it, z:
// 0.4-0.8 (0.9-2.8) at 48 points, 0.4-0.7 (1.1-3.1) at 240; phi: 0.5-0.8 (1.1-4.0) at np = 96, 0.5-0.7 (1.1-3.8) at 480.
//
// Shape: n = n2 + R2 n1, k = k1 + R1 k2, two register passes through shared memory.  A thread of the first pass takes the R1
// points of one n2, one of the second the R2 values of one k1; a transform of R points is done as P1 P2 points, P1 of 2..5,
// with the P1-point sums by additions, halvings and the constants of thirds and fifths.  TRL lines per CTA, max(R1, R2)
// threads a line.
// What bounds it: the integer pipe, as the power-of-two transforms.  The four transforms of a pair at 160 x 120 x
// 96: 334 us in FP64 -> 149 us.
#include "fft_fixed.cuh"
#include <cmath>

namespace mlg {

// sin(pi/3), sqrt(5)/4, sin(2pi/5), sin(pi/5) in units of 2^-61: upper and lower 31 bits
constexpr int Q_S3H = 929887696, Q_S3L = 1481419380, Q_R5H = 600239927, Q_R5L = 401909697;
constexpr int Q_S1H = 1021189158, Q_S1L = 1146421086, Q_S2H = 631129608, Q_S2L = 1968856558;

template <int H, int L> __device__ __forceinline__ qc q_scalec(qc a) { return {q_mulc<H, L>(a.x), q_mulc<H, L>(a.y)}; }
__device__ __forceinline__ qc q_half(qc a, int s) {   // a / 2^s, rounded
  const long long h = 1ll << (s - 1);
  return {(a.x + h) >> s, (a.y + h) >> s};
}
// P points in natural order; the constants of a fifth: cos(2pi/5), cos(4pi/5) = (-1 +- sqrt 5) / 4
template <int P> __device__ __forceinline__ void q_small(qc (&a)[P], int sgn) {
  if constexpr (P == 2) {
    const qc t = a[0];
    a[0] = q_add(t, a[1]);
    a[1] = q_sub(t, a[1]);
  } else if constexpr (P == 3) {
    const qc t = q_add(a[1], a[2]), m = q_sub(a[0], q_half(t, 1)), d = q_muli(q_scalec<Q_S3H, Q_S3L>(q_sub(a[1], a[2])), sgn);
    a[0] = q_add(a[0], t);
    a[1] = q_add(m, d);
    a[2] = q_sub(m, d);
  } else if constexpr (P == 4) {
    const qc t0 = q_add(a[0], a[2]), t1 = q_sub(a[0], a[2]), t2 = q_add(a[1], a[3]), t3 = q_muli(q_sub(a[1], a[3]), sgn);
    a[0] = q_add(t0, t2);
    a[2] = q_sub(t0, t2);
    a[1] = q_add(t1, t3);
    a[3] = q_sub(t1, t3);
  } else if constexpr (P == 5) {
    const qc t1 = q_add(a[1], a[4]), t2 = q_add(a[2], a[3]), t3 = q_sub(a[1], a[4]), t4 = q_sub(a[2], a[3]);
    const qc p = q_add(t1, t2), m = q_sub(a[0], q_half(p, 2)), d = q_scalec<Q_R5H, Q_R5L>(q_sub(t1, t2));
    const qc m1 = q_add(m, d), m2 = q_sub(m, d);
    const qc n1 = q_muli(q_add(q_scalec<Q_S1H, Q_S1L>(t3), q_scalec<Q_S2H, Q_S2L>(t4)), sgn);
    const qc n2 = q_muli(q_sub(q_scalec<Q_S2H, Q_S2L>(t3), q_scalec<Q_S1H, Q_S1L>(t4)), sgn);
    a[0] = q_add(a[0], p);
    a[1] = q_add(m1, n1);
    a[4] = q_sub(m1, n1);
    a[2] = q_add(m2, n2);
    a[3] = q_sub(m2, n2);
  }
}
// P1 P2 points in natural order, the twiddles exp(-+ 2 pi i j / (P1 P2)) at tw[j step]
template <int P1, int P2> __device__ __forceinline__ void q_comp(qc (&x)[P1 * P2], const int4* __restrict__ tw, int step, int sgn) {
  qc a[P2][P1];
#pragma unroll
  for (int i = 0; i < P1 * P2; ++i) a[i % P2][i / P2] = x[i];
#pragma unroll
  for (int r2 = 0; r2 < P2; ++r2) q_small<P1>(a[r2], sgn);
#pragma unroll
  for (int k1 = 0; k1 < P1; ++k1) {
    qc b[P2];
#pragma unroll
    for (int r2 = 0; r2 < P2; ++r2) b[r2] = (k1 && r2) ? q_mul(a[r2][k1], q_tw(tw, k1 * r2 * step, sgn)) : a[r2][k1];
    q_small<P2>(b, sgn);
#pragma unroll
    for (int r2 = 0; r2 < P2; ++r2) x[k1 + P1 * r2] = b[r2];
  }
}
template <> __device__ __forceinline__ void q_comp<2, 1>(qc (&x)[2], const int4* __restrict__, int, int sgn) { q_small<2>(x, sgn); }
template <> __device__ __forceinline__ void q_comp<3, 1>(qc (&x)[3], const int4* __restrict__, int, int sgn) { q_small<3>(x, sgn); }
template <> __device__ __forceinline__ void q_comp<4, 1>(qc (&x)[4], const int4* __restrict__, int, int sgn) { q_small<4>(x, sgn); }
template <> __device__ __forceinline__ void q_comp<5, 1>(qc (&x)[5], const int4* __restrict__, int, int sgn) { q_small<5>(x, sgn); }

struct QPlan { int L, r1, r2; };

// the line's scale from its n threads' shares, as q_scale (fftq.cu)
template <bool HALF> __device__ __forceinline__ bool qr_scale(const QStat* red, int lane, int TRL, int n, bool two, QScale& sc) {
  unsigned mx = 0;
  for (int q = 0; q < n; ++q) mx = max(mx, red[q * TRL + lane].mx);
  auto share = [&](int q) {   // moved to the line's unit by exact steps
    const QStat t = red[q * TRL + lane];
    const int d = min((int)(mx >> 20) - (int)(t.mx >> 20), 126);
    return t.s * __int_as_float((127 - d) << 23);
  };
  float s = 0.f, part = 0.f;
  for (int q = 0; q < n; ++q) {
    const float v = share(q);
    s += v;
    if (two) part = fmaxf(part, HALF ? v + share(q ? n - q : 0) : v);
  }
  auto bound = [](float x) { return (int)(__float_as_uint(x * 1.00006103515625f) >> 23) - 126; };
  const int es = bound(s);
  sc.e1 = (int)(mx >> 20) - 1022 + es;
  sc.sh = 0;
  if (two) {
    sc.sh = max(es - bound(part), 0);
    sc.e1 -= sc.sh;
  }
  return (mx == 0 || mx >= (100u << 20)) && mx < (2030u << 20);
}

// the first pass after its sums: twiddles between the passes, the common unit, and to shared memory at [k1][n2]
template <int R> __device__ __forceinline__ void qr_hand(const qc (&a)[R], qc* S, const int4* __restrict__ tw, int sgn, int n2, int r2,
                                                         int lane, int TRL, int sh) {
  const long long half = (1ll << sh) >> 1;
#pragma unroll
  for (int k1 = 0; k1 < R; ++k1) {
    qc v = a[k1];
    if (k1) v = q_mul(v, q_tw(tw, n2 * k1, sgn));
    v = {(v.x + half) >> sh, (v.y + half) >> sh};
    S[(k1 * r2 + n2) * TRL + lane] = v;
  }
}
// the second pass of thread k1: put(k, X_k)
template <int P1, int P2, class ST>
__device__ __forceinline__ void qr_second(const qc* S, const int4* __restrict__ tw, int sgn, const QPlan& pl, int k1, int lane, int TRL,
                                          bool sync, ST put) {
  constexpr int R = P1 * P2;
  qc b[R];
  if (k1 < pl.r1) {
#pragma unroll
    for (int i = 0; i < R; ++i) b[i] = S[(k1 * R + i) * TRL + lane];
    q_comp<P1, P2>(b, tw, pl.r1, sgn);
  }
  if (sync) __syncthreads();   // put goes to S
  if (k1 < pl.r1) {
#pragma unroll
    for (int i = 0; i < R; ++i) put(k1 + pl.r1 * i, b[i]);
  }
}
template <class ST>
__device__ __forceinline__ void qr_second_any(const qc* S, const int4* __restrict__ tw, int sgn, const QPlan& pl, int k1, int lane,
                                              int TRL, bool sync, ST put) {
  switch (pl.r2) {
#define QR(N, A, B) case N: qr_second<A, B>(S, tw, sgn, pl, k1, lane, TRL, sync, put); break;
    QR(2, 2, 1) QR(3, 3, 1) QR(4, 4, 1) QR(5, 5, 1) QR(6, 2, 3) QR(8, 4, 2) QR(9, 3, 3) QR(10, 2, 5) QR(12, 4, 3) QR(15, 3, 5) QR(16, 4, 4)
#undef QR
  }
}

// an FP64 transform of the CTA's lines for samples outside the fixed-point range: one radix at a time from S to the lines'
// own storage (point i at line + i st; its samples are in S) and back; the result is in S
__device__ void qr_line64(double2* S, double2* line, size_t st, bool ok, int L, const double2* __restrict__ tw, int sgn, int lane,
                          int TRL, int tt, int TT) {
  int rem = L;
  for (int ns = 1; ns < L;) {
    const int p = rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : 5;
    const RPass ps{(unsigned char)p, 1, (unsigned short)ns, (unsigned short)(L / p), ns > 1 ? (unsigned)(((1ull << 32) + ns - 1) / ns) : 0u};
    auto ld = [&](int i) { return S[i * TRL + lane]; };
    auto out = [&](int i, double2 v) { if (ok) line[(size_t)i * st] = v; };
    switch (p) {
      case 2: r_pass<double, 2, 1>(ps, L, tw, sgn, tt, TT, ld, out); break;
      case 3: r_pass<double, 3, 1>(ps, L, tw, sgn, tt, TT, ld, out); break;
      case 4: r_pass<double, 4, 1>(ps, L, tw, sgn, tt, TT, ld, out); break;
      default: r_pass<double, 5, 1>(ps, L, tw, sgn, tt, TT, ld, out); break;
    }
    __syncthreads();
    for (int i = tt; i < L; i += TT) S[i * TRL + lane] = ok ? line[(size_t)i * st] : make_double2(0.0, 0.0);
    __syncthreads();
    ns *= p;
    rem /= p;
  }
}

// z FFT (lines as zfft2_body), scaled
template <int P1, int P2>
__device__ __forceinline__ void zfft_qr_body(const FSet& fs, int nrdim, int npdim, const QPlan& pl, const int4* __restrict__ tw,
                                             const double2* __restrict__ tw64, int sgn, double scale, int nlines,
                                             unsigned char* smem_raw) {
  constexpr int R = P1 * P2, NB = 61;
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y, L = pl.L, r2 = pl.r2;
  qc* S = (qc*)smem_raw;
  QStat* red = (QStat*)(S + (L + 1) * TRL);
  const int gl = blockIdx.x * TRL + lane;     // line over the set; nlines per field
  const int f = gl / nlines, line = gl - f * nlines;
  const bool ok = f < fs.n;
  const size_t ps = (size_t)nrdim * npdim;
  double2* base = fset_e(fs, ok ? f : 0) + line;
  const bool mine = tt < r2;
  double2 d[R];
#pragma unroll
  for (int i = 0; i < R; ++i) d[i] = ok && mine ? base[(size_t)(tt + r2 * i) * ps] : make_double2(0.0, 0.0);
  if (mine) red[tt * TRL + lane] = q_stat<R>(d);
  __syncthreads();
  QScale sc;
  const bool fits = qr_scale<false>(red, lane, TRL, r2, L >= 80, sc);
  if (__syncthreads_or(!fits)) {
    double2* D = (double2*)smem_raw;
    if (mine) {
#pragma unroll
      for (int i = 0; i < R; ++i) D[(tt + r2 * i) * TRL + lane] = d[i];
    }
    __syncthreads();
    qr_line64(D, base, ps, ok, L, tw64, sgn, lane, TRL, tt, TT);
    if (ok)
      for (int i = tt; i < L; i += TT) base[(size_t)i * ps] = c_scale(D[i * TRL + lane], scale);
    return;
  }
  if (mine) {
    const int fb = 1085 - NB + sc.e1;
    qc a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = {xs_fixs(d[i].x, fb), xs_fixs(d[i].y, fb)};
    q_comp<P1, P2>(a, tw, r2, sgn);
    qr_hand<R>(a, S, tw, sgn, tt, r2, lane, TRL, sc.sh);
  }
  __syncthreads();
  const int eo = sc.e1 + sc.sh - NB;
  const bool one = scale == 1.0;
  qr_second_any(S, tw, sgn, pl, tt, lane, TRL, false, [&](int k, qc v) {
    double2 o = make_double2(xs_i64_to_double(v.x, eo), xs_i64_to_double(v.y, eo));
    if (!one) { o.x *= scale; o.y *= scale; }
    if (ok) base[(size_t)k * ps] = o;
  });
}
#define QR_FIRST(CALL)                                                                     \
  switch (pl.r1) {                                                                         \
    case 8: CALL(4, 2) break;                                                              \
    case 9: CALL(3, 3) break;                                                              \
    case 10: CALL(2, 5) break;                                                             \
    case 12: CALL(4, 3) break;                                                             \
    case 15: CALL(3, 5) break;                                                             \
    case 16: CALL(4, 4) break;                                                             \
  }
__global__ void __launch_bounds__(256) k_zfft_qr(FSet fs, int nrdim, int npdim, QPlan pl, const int4* __restrict__ tw,
                                                 const double2* __restrict__ tw64, int sgn, double scale, int nlines) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
#define Z(A, B) zfft_qr_body<A, B>(fs, nrdim, npdim, pl, tw, tw64, sgn, scale, nlines, smem_raw);
  QR_FIRST(Z)
#undef Z
}

// phi forward: packed reals (rows times rs[r] first, in FP64) -> X_0..X_L scaled, in place (lines (r, z)); the split as in
// k_pfft_fwd_q
template <int P1, int P2>
__device__ __forceinline__ void pfft_fwd_qr_body(const FSet& fs, int nrdim, int npdim, int nzdim, const QPlan& pl,
                                                 const int4* __restrict__ tw, const int4* __restrict__ twr,
                                                 const double2* __restrict__ tw64, const double2* __restrict__ twr64, double scale,
                                                 int nrs, unsigned char* smem_raw) {
  constexpr int R = P1 * P2, NB = 60;   // e and t double
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y, L = pl.L, r2 = pl.r2;
  qc* S = (qc*)smem_raw;
  QStat* red = (QStat*)(S + (L + 1) * TRL);
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const bool rsc = rs != nullptr && ok && r < nrs, mine = tt < r2;
  double2 d[R];
#pragma unroll
  for (int i = 0; i < R; ++i) d[i] = ok && mine ? base[(size_t)(tt + r2 * i) * nrdim] : make_double2(0.0, 0.0);
  if (rsc) {
    const double rv = rs[r];
#pragma unroll
    for (int i = 0; i < R; ++i) { d[i].x *= rv; d[i].y *= rv; }
  }
  if (mine) red[tt * TRL + lane] = q_stat<R>(d);
  __syncthreads();
  QScale sc;
  const bool fits = qr_scale<false>(red, lane, TRL, r2, L >= 80, sc);
  if (__syncthreads_or(!fits)) {
    double2* D = (double2*)smem_raw;
    if (mine) {
#pragma unroll
      for (int i = 0; i < R; ++i) D[(tt + r2 * i) * TRL + lane] = d[i];
    }
    __syncthreads();
    qr_line64(D, base, nrdim, ok, L, tw64, -1, lane, TRL, tt, TT);
    if (ok)
      for (int k = tt; k <= L; k += TT) {
        const double2 zk = D[(k == L ? 0 : k) * TRL + lane];
        double2 zc = D[(k == 0 ? 0 : L - k) * TRL + lane];
        zc.y = -zc.y;
        const double2 fe = c_scale(c_add(zk, zc), 0.5), fo = c_muli(c_scale(c_sub(zk, zc), 0.5), -1);   // (zk - zc)/(2i)
        base[(size_t)k * nrdim] = c_scale(c_add(fe, c_mul(load_tw<double>(twr64, k, -1), fo)), scale);
      }
    return;
  }
  if (mine) {
    const int fb = 1085 - NB + sc.e1;
    qc a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = {xs_fixs(d[i].x, fb), xs_fixs(d[i].y, fb)};
    q_comp<P1, P2>(a, tw, r2, -1);
    qr_hand<R>(a, S, tw, -1, tt, r2, lane, TRL, sc.sh);
  }
  __syncthreads();
  qr_second_any(S, tw, -1, pl, tt, lane, TRL, true, [&](int k, qc v) { S[k * TRL + lane] = v; });
  __syncthreads();
  if (!ok) return;
  const int eo = sc.e1 + sc.sh - NB - 1;
  for (int k = tt; 2 * k <= L; k += TT) {
    const qc zk = S[k * TRL + lane], zc = q_conj(S[(k ? L - k : 0) * TRL + lane]);
    const qc s = q_add(zk, zc), t = q_mul(q_muli(q_sub(zk, zc), -1), q_tw(twr, k, -1));
    base[(size_t)k * nrdim] = make_double2(xs_i64_to_double(s.x + t.x, eo) * scale, xs_i64_to_double(s.y + t.y, eo) * scale);
    if (k != L - k)
      base[(size_t)(L - k) * nrdim] = make_double2(xs_i64_to_double(s.x - t.x, eo) * scale, xs_i64_to_double(t.y - s.y, eo) * scale);
  }
}
__global__ void __launch_bounds__(256) k_pfft_fwd_qr(FSet fs, int nrdim, int npdim, int nzdim, QPlan pl, const int4* __restrict__ tw,
                                                     const int4* __restrict__ twr, const double2* __restrict__ tw64,
                                                     const double2* __restrict__ twr64, double scale, int nrs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
#define F(A, B) pfft_fwd_qr_body<A, B>(fs, nrdim, npdim, nzdim, pl, tw, twr, tw64, twr64, scale, nrs, smem_raw);
  QR_FIRST(F)
#undef F
}

// phi backward: X_0..X_L -> packed reals (unnormalised; rows times rs[r] last, in FP64), slot L <- np X_L, in place
template <int P1, int P2>
__device__ __forceinline__ void pfft_bwd_qr_body(const FSet& fs, int nrdim, int npdim, int nzdim, const QPlan& pl,
                                                 const int4* __restrict__ tw, const int4* __restrict__ twr,
                                                 const double2* __restrict__ tw64, const double2* __restrict__ twr64, double np_d,
                                                 int nrs, unsigned char* smem_raw) {
  constexpr int R = P1 * P2, NB = 60;
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y, L = pl.L, r2 = pl.r2;
  qc* S = (qc*)smem_raw;                       // [L + 1][TRL]
  QStat* red = (QStat*)(S + (L + 1) * TRL);
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const bool rsc = rs != nullptr && r < nrs, mine = tt < r2;
  const double rv = rsc ? rs[r] : 1.0;
  double2 d[R + 1];
#pragma unroll
  for (int i = 0; i < R; ++i) d[i] = ok && mine ? base[(size_t)(tt + r2 * i) * nrdim] : make_double2(0.0, 0.0);
  d[R] = ok && tt == 0 ? base[(size_t)L * nrdim] : make_double2(0.0, 0.0);
  const double2 nyq = d[R];
  if (tt == 0) { d[0].y = 0.0; d[R].y = 0.0; }   // the imaginary parts of X_0 and X_L do not enter
  if (mine) red[tt * TRL + lane] = q_stat<R + 1>(d);
  __syncthreads();
  QScale sc;
  const bool fits = qr_scale<true>(red, lane, TRL, r2, L >= 80, sc);
  if (__syncthreads_or(!fits)) {
    double2* D = (double2*)smem_raw;
    for (int k = tt; k < L; k += TT) {
      double2 xk = ok ? base[(size_t)k * nrdim] : make_double2(0.0, 0.0);
      double2 xc = ok ? base[(size_t)(L - k) * nrdim] : make_double2(0.0, 0.0);
      if (k == 0) { xk.y = 0; xc.y = 0; }
      xc.y = -xc.y;
      const double2 h = c_mul(c_sub(xk, xc), load_tw<double>(twr64, k, +1));   // exp(+2 pi i k / np)
      D[k * TRL + lane] = c_add(c_add(xk, xc), c_muli(h, 1));
    }
    __syncthreads();
    qr_line64(D, base, nrdim, ok, L, tw64, +1, lane, TRL, tt, TT);
    if (ok)
      for (int i = tt; i < L; i += TT) base[(size_t)i * nrdim] = rsc ? c_scale(D[i * TRL + lane], rv) : D[i * TRL + lane];
  } else {
    qc a[R];
    if (mine) {
      const int fb = 1085 - NB + sc.e1;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        a[i] = {xs_fixs(d[i].x, fb), xs_fixs(d[i].y, fb)};
        S[(tt + r2 * i) * TRL + lane] = a[i];
      }
      if (tt == 0) S[L * TRL + lane] = {xs_fixs(d[R].x, fb), 0};
    }
    __syncthreads();
    // V_k = X_k + conj X_(L-k) + i (X_k - conj X_(L-k)) exp(+2 pi i k / np), as in k_pfft_bwd_q
    if (mine) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int k = tt + r2 * i;
        const qc xc = q_conj(S[(L - k) * TRL + lane]);
        const qc g = q_add(a[i], xc), h = q_mul(q_sub(a[i], xc), q_tw(twr, k, +1));
        a[i] = q_add(g, q_muli(h, 1));
      }
    }
    __syncthreads();   // S read: free for the passes
    if (mine) {
      q_comp<P1, P2>(a, tw, r2, +1);
      qr_hand<R>(a, S, tw, +1, tt, r2, lane, TRL, sc.sh);
    }
    __syncthreads();
    const int eo = sc.e1 + sc.sh - NB;
    qr_second_any(S, tw, +1, pl, tt, lane, TRL, false, [&](int k, qc v) {
      double2 o = make_double2(xs_i64_to_double(v.x, eo), xs_i64_to_double(v.y, eo));
      if (rsc) { o.x *= rv; o.y *= rv; }
      if (ok) base[(size_t)k * nrdim] = o;
    });
  }
  if (ok && tt == 0) {
    double2 v = make_double2(nyq.x * np_d, nyq.y * np_d);
    if (rsc) { v.x *= rv; v.y *= rv; }
    base[(size_t)L * nrdim] = v;
  }
}
__global__ void __launch_bounds__(256) k_pfft_bwd_qr(FSet fs, int nrdim, int npdim, int nzdim, QPlan pl, const int4* __restrict__ tw,
                                                     const int4* __restrict__ twr, const double2* __restrict__ tw64,
                                                     const double2* __restrict__ twr64, double np_d, int nrs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
#define B(A, C) pfft_bwd_qr_body<A, C>(fs, nrdim, npdim, nzdim, pl, tw, twr, tw64, twr64, np_d, nrs, smem_raw);
  QR_FIRST(B)
#undef B
}

// ------------------------------------------------------------------------------------------------
// the split with the fewest threads a line, R1 first; false where there is none
static bool qr_plan(int L, QPlan& pl) {
  static const int first[] = {8, 9, 10, 12, 15, 16}, second[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16};
  int best = 17;
  for (int a : first)
    for (int b : second)
      if (a * b == L && std::max(a, b) < best) {
        best = std::max(a, b);
        pl = {L, a, b};
      }
  return best < 17;
}
bool fftqr_length(int L) {
  QPlan pl;
  return L >= 18 && (L & (L - 1)) != 0 && qr_plan(L, pl);
}
// Few lines are done sooner in FP64, one radix at a time (fftr.cu): a transform pair at 48 x 48 x 24 (2.8e4 points a
// transform) takes 78 us so and 84 us in fixed point, one at 64 x 60 x 30 (5.8e4) 87 and 80 us.
bool fftqr_pays(int L, long long lines) { return fftqr_length(L) && lines * L >= 40000; }
// 16 lines per CTA, fewer (at least two) where that leaves SMs without one
static int qr_lines(long long lines) {
  int tr = 16;
  while (tr > 2 && lines / tr < 152) tr /= 2;
  return tr;
}
static size_t qr_smem(int L, int TRL) { return (size_t)(L + 1) * TRL * sizeof(qc) + (size_t)16 * TRL * sizeof(QStat); }
template <class K> static int qr_attr(K k, size_t bytes) {
  if (bytes > 48 * 1024) MLG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return 0;
}
int launch_zfft_qr(const FSet& fs, int dir, double scale) {
  QPlan pl;
  if (!qr_plan(G.nz, pl)) return set_error(MLG_ESIZE, "vertical_fft: no fixed-point transform of this length");
  const int nlines = G.nrdim * G.npdim, TRL = qr_lines((long long)nlines * fs.n);
  const size_t sm = qr_smem(pl.L, TRL);
  MLG_TRY(qr_attr(k_zfft_qr, sm));
  k_zfft_qr<<<cdiv((long long)nlines * fs.n, TRL), dim3(TRL, std::max(pl.r1, pl.r2)), sm, G.stream>>>(
      fs, G.nrdim, G.npdim, pl, G.tw_zq, G.tw_zqd, dir, scale, nlines);
  MLG_LAUNCH();
  return 0;
}
int launch_pfft_qr(const FSet& fs, int dir, double scale) {
  QPlan pl;
  if (!qr_plan(G.nph, pl)) return set_error(MLG_ESIZE, "horizontal_fft: no fixed-point transform of this length");
  const long long lines = (long long)G.nrdim * G.nzdim * fs.n;
  const int TRL = qr_lines(lines), grid = cdiv(lines, TRL);
  const dim3 blk(TRL, std::max(pl.r1, pl.r2));
  const size_t sm = qr_smem(pl.L, TRL);
  if (dir < 0) {
    MLG_TRY(qr_attr(k_pfft_fwd_qr, sm));
    k_pfft_fwd_qr<<<grid, blk, sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, pl, G.tw_pq, G.tw_prq, G.tw_pqd, G.tw_prqd, scale, G.nr);
  } else {
    MLG_TRY(qr_attr(k_pfft_bwd_qr, sm));
    k_pfft_bwd_qr<<<grid, blk, sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, pl, G.tw_pq, G.tw_prq, G.tw_pqd, G.tw_prqd,
                                               (double)G.np, G.nr);
  }
  MLG_LAUNCH();
  return 0;
}

}  // namespace mlg
