// fftq.cu — the plain form's FFTs of power-of-two lengths (16..256 points) in 64-bit fixed point, in FFTE's conventions
// (fft.cu).
//
// Why: GB300 issues about 2 FP64 operations per clock per SM and 64 32-bit integer ones; a 64-bit addition takes two of the
// latter, a multiplication by a constant seven.  The FP64 transforms stood at that pipe: 218 us for the z transform of
// three fields at 192 x 128 x 128 (about 23 FP64 operations a sample), 275 and 307 us for the phi transforms, where the
// fields' way through HBM takes 23.  Now 80 us (z), 68 us (phi forward) and 79 us (phi backward).
//
// Scaling: every line has its own power of two.  With S >= sum_n (|re x_n| + |im x_n|), 2^es > S, the samples are rounded to
// integers X_n = x_n 2^(NB - es); no partial sum of a DFT exceeds sum |X_n| < 2^NB in modulus, so nothing overflows at any
// stage.  Sums are exact; a multiplication by a twiddle of 61 bits rounds to about the nearest integer; a result is
// rounded once to FP64.  From 128 points on the first pass has a finer unit of its own (q_scale).  The rounding is
// below the FP64 transforms' at every length: against extended precision, in units of 2^-53 of a line's root mean square
// (white, decaying and one-mode lines; FP64 beside it), z: 0.4-0.5 (0.9-1.7) at 64 points, 0.4-0.5 (1.1-2.0) at 256; phi:
// 0.5-0.6 (1.2-2.1) at np = 128, 0.5-0.6 (1.1-2.3) at 512.
// A block one of whose lines holds a non-finite or a huge sample (2^1007 and up) or none above 2^-922 (but not all zero)
// takes the FP64 transform.
//
// Shape: as the FP64 transforms (fft_common.cuh): TRL lines per CTA, R2 threads per line, L = R1 R2 in two register
// passes through shared memory.
#include "fft_fixed.cuh"

namespace mlg {

// cos(pi/4), cos(pi/8), sin(pi/8) in units of 2^-61: upper and lower 31 bits
constexpr int Q_C4H = 759250124, Q_C4L = 2134625425, Q_C8H = 992008094, Q_C8L = 848119337, Q_S8H = 410903206, Q_S8L = 1465168233;

// v exp(SGN 2 pi i j / 16), j = 0..7 a compile-time constant after unrolling
template <int SGN> __device__ __forceinline__ qc q_tw16(qc v, int j) {
  if (j == 0) return v;
  if (j == 4) return q_muli(v, SGN);
  if (j == 2 || j == 6) {   // (+-1 + SGN i) cos(pi/4)
    const long long x = j == 2 ? v.x : -v.x, y = j == 2 ? v.y : -v.y, sx = SGN > 0 ? v.x : -v.x, sy = SGN > 0 ? v.y : -v.y;
    return {q_mulc<Q_C4H, Q_C4L>(x - sy), q_mulc<Q_C4H, Q_C4L>(y + sx)};
  }
  const bool c8 = j == 1 || j == 7;   // |cos| = cos(pi/8) at j = 1, 7 and sin(pi/8) at 3, 5
  int ch = c8 ? Q_C8H : Q_S8H, cl = c8 ? Q_C8L : Q_S8L, sh = c8 ? Q_S8H : Q_C8H, sl = c8 ? Q_S8L : Q_C8L;
  if (j > 4) { ch = -ch; cl = -cl; }
  if (SGN < 0) { sh = -sh; sl = -sl; }
  return q_mul(v, make_int4(ch, sh, cl, sl));
}

// in-register DFT of N <= 16 points, as dft_reg: a[i] = X_bitrev(i)
template <int N, int SGN> __device__ __forceinline__ void q_dft(qc* a) {
#pragma unroll
  for (int len = N; len >= 2; len >>= 1) {
#pragma unroll
    for (int i = 0; i < N; i += len) {
#pragma unroll
      for (int k = 0; k < len / 2; ++k) {
        const qc u = a[i + k], v = a[i + k + len / 2];
        a[i + k] = q_add(u, v);
        a[i + k + len / 2] = q_tw16<SGN>(q_sub(u, v), k * (16 / len));
      }
    }
  }
}
// from 128 points on (q_scale)
template <int L> __host__ __device__ constexpr bool q_two_units() { return L >= 128; }

// the two passes, as fft2pass
template <int L, int SGN, int TRL>
__device__ __forceinline__ void q_fft2pass(qc* a, qc (*b)[Split<L>::R2], qc* S, const int4* __restrict__ tw, int w, int lane,
                                           int sh) {
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2;
  q_dft<R1, SGN>(a);
  const long long half = (1ll << sh) >> 1;
#pragma unroll
  for (int i = 0; i < R1; ++i) {
    const int k1 = bitrev(i, R1);
    qc v = a[i];
    if (k1) v = q_mul(v, q_tw(tw, (w * k1) & (L - 1), SGN));
    if (q_two_units<L>()) v = {(v.x + half) >> sh, (v.y + half) >> sh};
    S[(k1 * R2 + w) * TRL + lane] = v;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int k1 = w * Q + q;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) b[q][n2] = S[(k1 * R2 + n2) * TRL + lane];
    q_dft<R2, SGN>(b[q]);
  }
}

// the line's scale from its R2 threads' shares: sum |x| < 2^e over the line, and < 2^e1 over any one thread's samples
// (HALF: over those of threads w and R2 - w together), sh = e - e1; false where the line needs FP64.  A thread's samples
// are what the first pass sums: its own, finer unit keeps the rounding of the first pass' twiddles, which all later
// stages add up, below that of the second's (np = 512, white: 2.6 -> 0.6 units of 2^-53; it costs 2 % of the time)
template <int L, int TRL, bool HALF> __device__ __forceinline__ bool q_scale(const QStat* red, int lane, QScale& sc) {
  constexpr int R2 = Split<L>::R2;
  unsigned mx = 0;
#pragma unroll
  for (int q = 0; q < R2; ++q) mx = max(mx, red[q * TRL + lane].mx);
  float s = 0.f, part = 0.f, v[R2];
#pragma unroll
  for (int q = 0; q < R2; ++q) {
    const QStat t = red[q * TRL + lane];
    // t.s is in units of 2^(that share's exponent - 1022), in [0.5, 2 N): moved to the line's unit by exact steps
    const int d = min((int)(mx >> 20) - (int)(t.mx >> 20), 126);
    v[q] = t.s * __int_as_float((127 - d) << 23);
    s += v[q];
  }
  // the sums are low by up to 2^-20 a term (the words below the upper one, and the summation): s (1 + 2^-14) < 2^es
  auto bound = [](float x) { return (int)(__float_as_uint(x * 1.00006103515625f) >> 23) - 126; };
  const int es = bound(s);
  sc.e1 = (int)(mx >> 20) - 1022 + es;
  sc.sh = 0;
  if (q_two_units<L>()) {
#pragma unroll
    for (int q = 0; q < R2; ++q) part = fmaxf(part, HALF ? v[q] + v[(R2 - q) % R2] : v[q]);
    sc.sh = max(es - bound(part), 0);
    sc.e1 -= sc.sh;
  }
  return (mx == 0 || mx >= (100u << 20)) && mx < (2030u << 20);
}

// z FFT (lines as k_zfft2), scaled by 2^sexp
template <int L, int SGN, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, TRL * Split<L>::R2 == 256 ? 2 : 0) k_zfft_q(FSet fs, int nrdim, int npdim, const int4* __restrict__ tw,
                                                               const double2* __restrict__ tw64, int sexp, double scale,
                                                               int nlines) {
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2, NB = 61;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  qc* S = (qc*)smem_raw;
  QStat* red = (QStat*)(S + L * TRL);
  const int lane = threadIdx.x, w = threadIdx.y;
  const int gl = blockIdx.x * TRL + lane;     // line over the set; nlines per field
  const int f = gl / nlines, line = gl - f * nlines;
  const bool ok = f < fs.n;
  const size_t ps = (size_t)nrdim * npdim;
  double2* base = fset_e(fs, ok ? f : 0) + line;
  double2 d[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) d[n1] = ok ? base[(size_t)(w + R2 * n1) * ps] : make_double2(0.0, 0.0);
  red[w * TRL + lane] = q_stat<R1>(d);
  __syncthreads();
  QScale sc;
  const bool fits = q_scale<L, TRL, false>(red, lane, sc);
  if (__syncthreads_or(!fits)) {
    zfft2_body<double, L, SGN, TRL>(fs, nrdim, npdim, tw64, scale, 0, nlines, smem_raw);
    return;
  }
  const int fb = 1085 - NB + sc.e1;
  qc a[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) a[n1] = {xs_fixs(d[n1].x, fb), xs_fixs(d[n1].y, fb)};
  qc b[Q][R2];
  q_fft2pass<L, SGN, TRL>(a, b, S, tw, w, lane, sc.sh);
  if (!ok) return;
  const int eo = sc.e1 + sc.sh - NB + sexp;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i)
      base[(size_t)(k1 + R1 * bitrev(i, R2)) * ps] = make_double2(xs_i64_to_double(b[q][i].x, eo), xs_i64_to_double(b[q][i].y, eo));
  }
}

// φ forward: packed reals (rows times rs[r] first, in FP64) -> X_0..X_L scaled by 2^sexp, in place (lines (r, z)).  X_k and
// X_(L-k) come from the same sums: with e = Z_k + conj Z_(L-k), t = -i w_k (Z_k - conj Z_(L-k)), X_k = (e + t) / 2 and
// X_(L-k) = conj(e - t) / 2
template <int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, TRL * Split<L>::R2 == 256 ? 2 : 0) k_pfft_fwd_q(FSet fs, int nrdim, int npdim, int nzdim,
                                                                   const int4* __restrict__ tw, const int4* __restrict__ twr,
                                                                   const double2* __restrict__ tw64,
                                                                   const double2* __restrict__ twr64, int sexp, double scale,
                                                                   int nrs) {
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2, NB = 60;   // e and t double
  extern __shared__ __align__(16) unsigned char smem_raw[];
  qc* S = (qc*)smem_raw;
  QStat* red = (QStat*)(S + L * TRL);
  const int lane = threadIdx.x, w = threadIdx.y;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const bool rsc = rs != nullptr && ok && r < nrs;
  double2 d[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) d[n1] = ok ? base[(size_t)(w + R2 * n1) * nrdim] : make_double2(0.0, 0.0);
  if (rsc) {
    const double rv = rs[r];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) { d[n1].x *= rv; d[n1].y *= rv; }
  }
  red[w * TRL + lane] = q_stat<R1>(d);
  __syncthreads();
  QScale sc;
  const bool fits = q_scale<L, TRL, false>(red, lane, sc);
  if (__syncthreads_or(!fits)) {
    pfft_fwd2_body<double, L, TRL>(fs, nrdim, npdim, nzdim, tw64, twr64, scale, scale, 0.0, nrs, smem_raw);
    return;
  }
  const int fb = 1085 - NB + sc.e1;
  qc a[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) a[n1] = {xs_fixs(d[n1].x, fb), xs_fixs(d[n1].y, fb)};
  qc b[Q][R2];
  q_fft2pass<L, -1, TRL>(a, b, S, tw, w, lane, sc.sh);
  __syncthreads();   // every thread has read its pass-2 inputs: S takes the spectrum, Z_k at row k
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i) S[(k1 + R1 * bitrev(i, R2)) * TRL + lane] = b[q][i];
  }
  __syncthreads();
  if (!ok) return;
  const int eo = sc.e1 + sc.sh - NB + sexp - 1;
  for (int k = w; k <= L / 2; k += R2) {
    const qc zk = S[k * TRL + lane], zc = q_conj(S[((L - k) & (L - 1)) * TRL + lane]);
    const qc s = q_add(zk, zc), t = q_mul(q_muli(q_sub(zk, zc), -1), q_tw(twr, k, -1));
    base[(size_t)k * nrdim] = make_double2(xs_i64_to_double(s.x + t.x, eo), xs_i64_to_double(s.y + t.y, eo));
    if (k != L - k)
      base[(size_t)(L - k) * nrdim] = make_double2(xs_i64_to_double(s.x - t.x, eo), xs_i64_to_double(t.y - s.y, eo));
  }
}

// φ backward: X_0..X_L -> packed reals (unnormalised; rows times rs[r] last, in FP64), slot L <- np X_L, in place
template <int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, TRL * Split<L>::R2 == 256 ? 2 : 0) k_pfft_bwd_q(FSet fs, int nrdim, int npdim, int nzdim,
                                                                   const int4* __restrict__ tw, const int4* __restrict__ twr,
                                                                   const double2* __restrict__ tw64,
                                                                   const double2* __restrict__ twr64, double np_d, int nrs) {
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2, NB = 60;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  qc* S = (qc*)smem_raw;                       // [L + 1][TRL]
  QStat* red = (QStat*)(S + (L + 1) * TRL);
  const int lane = threadIdx.x, w = threadIdx.y;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  double2 d[R1 + 1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) d[n1] = ok ? base[(size_t)(w + R2 * n1) * nrdim] : make_double2(0.0, 0.0);
  d[R1] = ok && w == 0 ? base[(size_t)L * nrdim] : make_double2(0.0, 0.0);
  const double2 nyq = d[R1];
  if (w == 0) { d[0].y = 0.0; d[R1].y = 0.0; }   // the imaginary parts of X_0 and X_L do not enter
  red[w * TRL + lane] = q_stat<R1 + 1>(d);
  __syncthreads();
  QScale sc;
  const bool fits = q_scale<L, TRL, true>(red, lane, sc);
  // (a non-finite X_L reaches the output through slot L in either transform; a non-finite Im X_0 reaches nothing)
  if (__syncthreads_or(!fits)) {
    pfft_bwd2_body<double, L, TRL>(fs, nrdim, npdim, nzdim, tw64, twr64, np_d, nrs, smem_raw);
    return;
  }
  const int fb = 1085 - NB + sc.e1;
  qc a[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    a[n1] = {xs_fixs(d[n1].x, fb), xs_fixs(d[n1].y, fb)};
    S[(w + R2 * n1) * TRL + lane] = a[n1];
  }
  if (w == 0) S[L * TRL + lane] = {xs_fixs(d[R1].x, fb), 0};
  __syncthreads();
  // V_k = X_k + conj X_(L-k) + i (X_k - conj X_(L-k)) exp(+2 pi i k / np): twice the sums of |X| over the line at most,
  // counting each X_k of the half spectrum twice, so half the unit
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    const int k = w + R2 * n1;
    const qc xc = q_conj(S[(L - k) * TRL + lane]);
    const qc g = q_add(a[n1], xc), h = q_mul(q_sub(a[n1], xc), q_tw(twr, k, +1));
    a[n1] = q_add(g, q_muli(h, 1));
  }
  __syncthreads();   // S read: free for the passes
  qc b[Q][R2];
  q_fft2pass<L, +1, TRL>(a, b, S, tw, w, lane, sc.sh);
  if (!ok) return;
  const bool rsc = rs != nullptr && r < nrs;
  const double rv = rsc ? rs[r] : 1.0;
  const int eo = sc.e1 + sc.sh - NB;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i) {
      double2 v = make_double2(xs_i64_to_double(b[q][i].x, eo), xs_i64_to_double(b[q][i].y, eo));
      if (rsc) { v.x *= rv; v.y *= rv; }
      base[(size_t)(k1 + R1 * bitrev(i, R2)) * nrdim] = v;
    }
  }
  if (w == 0) {
    double2 v = make_double2(nyq.x * np_d, nyq.y * np_d);
    if (rsc) { v.x *= rv; v.y *= rv; }
    base[(size_t)L * nrdim] = v;
  }
}

// ------------------------------------------------------------------------------------------------
bool fftq_length(int L) { return L == 16 || L == 32 || L == 64 || L == 128 || L == 256; }

template <class K> static int q_smem(K k, size_t bytes) {
  if (bytes > 48 * 1024) MLG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return 0;
}

template <int L, int SGN> static int zfft_q(const FSet& fs, int sexp) {
  // 16 lines from 64 points on, so that several CTAs share an SM (two of the 256 threads of 256 points, held to 128 registers:
  // four transforms of three fields at 512 x 512 x 256 7.3 -> 6.0 ms)
  constexpr int TRL = L >= 64 ? 16 : 32, R2 = Split<L>::R2;
  const size_t sm = (size_t)L * TRL * sizeof(qc) + (size_t)R2 * TRL * sizeof(QStat);
  MLG_TRY(q_smem(k_zfft_q<L, SGN, TRL>, sm));
  const int nlines = G.nrdim * G.npdim;
  k_zfft_q<L, SGN, TRL><<<cdiv((long long)nlines * fs.n, TRL), dim3(TRL, R2), sm, G.stream>>>(
      fs, G.nrdim, G.npdim, G.tw_zq, G.tw_z, sexp, ldexp(1.0, sexp), nlines);
  MLG_LAUNCH();
  return 0;
}
int launch_zfft_q(const FSet& fs, int dir, int sexp) {
  switch (G.nz) {
#define ZQ(LEN) case LEN: return dir < 0 ? zfft_q<LEN, -1>(fs, sexp) : zfft_q<LEN, +1>(fs, sexp);
    ZQ(16) ZQ(32) ZQ(64) ZQ(128) ZQ(256)
#undef ZQ
  }
  return set_error(MLG_ESIZE, "vertical_fft: no fixed-point transform of this length");
}

template <int L> static int pfft_q(const FSet& fs, int dir, int sexp) {
  constexpr int TRL = L >= 64 ? 16 : 32, R2 = Split<L>::R2;
  const size_t sm = (size_t)(L + 1) * TRL * sizeof(qc) + (size_t)R2 * TRL * sizeof(QStat);
  const int grid = cdiv((long long)G.nrdim * G.nzdim * fs.n, TRL);
  if (dir < 0) {
    MLG_TRY(q_smem(k_pfft_fwd_q<L, TRL>, sm));
    k_pfft_fwd_q<L, TRL><<<grid, dim3(TRL, R2), sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, G.tw_pq, G.tw_prq, G.tw_p, G.tw_pr,
                                                                sexp, ldexp(1.0, sexp), G.nr);
  } else {
    MLG_TRY(q_smem(k_pfft_bwd_q<L, TRL>, sm));
    k_pfft_bwd_q<L, TRL><<<grid, dim3(TRL, R2), sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, G.tw_pq, G.tw_prq, G.tw_p, G.tw_pr,
                                                                (double)G.np, G.nr);
  }
  MLG_LAUNCH();
  return 0;
}
int launch_pfft_q(const FSet& fs, int dir, int sexp) {
  switch (G.nph) {
    case 16: return pfft_q<16>(fs, dir, sexp);
    case 32: return pfft_q<32>(fs, dir, sexp);
    case 64: return pfft_q<64>(fs, dir, sexp);
    case 128: return pfft_q<128>(fs, dir, sexp);
    case 256: return pfft_q<256>(fs, dir, sexp);
  }
  return set_error(MLG_ESIZE, "horizontal_fft: no fixed-point transform of this length");
}

}  // namespace mlg
