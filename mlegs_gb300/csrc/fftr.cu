// fftr.cu — FFTs of lengths that are no power of two in 16..256 (products of 2, 3 and 5; FFTE's conventions, fft.cu), in
// FP32 (mixed form) and FP64.
//
// Algorithm: Stockham autosort with the radices 4, then 2, 3, 5.  Consecutive stages are done together in registers where
// the product of their radices is at most 16: a thread loads the p1 p2 points of a butterfly pair, does the p1- and the
// p2-point transforms with their twiddles and stores once.  Lengths of up to three such passes' radices (60 = 4 3 | 5,
// 90 = 2 3 | 3 5, 96 = 4 4 | 2 3) take two: the first straight from the field, the last straight to it, with one exchange
// through shared memory between them.  The operations on a sample and their order are those of the one-stage-at-a-time
// transform, so that the results are the same to the last bit.
//
// Lines are taken flat over the fields of a set (as the power-of-two transforms, fft_common.cuh), TRL consecutive ones
// per CTA, and TT threads per line.
//
// What bounds it: FP32, latency (the fields of a step make less than one wave of CTAs, each load, transform, store once)
// and the issue slots, 150 instructions a sample, a third of them FP64-FP32 conversions; FP64, GB300's FP64 pipe (2 operations
// per clock per SM).  Sixty transforms of three fields at 96 x 120 x 90, mixed: 4 107 -> 2 084 us against one stage at a time
// through shared memory, field by field.
#include "fft_common.cuh"

namespace mlg {

constexpr int RP_MAX = 10;
struct RPlan { int L, n, flat; RPass s[RP_MAX]; };   // flat: the first pass loads to shared memory alone, the last stores alone

template <typename T, class LD, class ST>
__device__ __forceinline__ void r_pass_any(const RPass& ps, int L, const typename TW<T>::t* __restrict__ tw, int sgn, int tt,
                                           int TT, LD ld, ST st) {
  switch (ps.p1 * 8 + ps.p2) {
#define RP(A, B) case A * 8 + B: r_pass<T, A, B>(ps, L, tw, sgn, tt, TT, ld, st); break;
    RP(1, 1) RP(2, 1) RP(3, 1) RP(4, 1) RP(5, 1) RP(4, 4) RP(4, 2) RP(4, 3) RP(2, 3) RP(2, 5) RP(3, 3) RP(3, 5)
#undef RP
  }
}
// a line's passes: the first reads by ld, the last stores by st, through S0 and (three or more passes) S1, [L][TRL].  All of
// the CTA's threads have read by ld before the first st.
template <typename T, class LD, class ST>
__device__ __forceinline__ void r_fft(const RPlan& pl, typename CT<T>::t* S0, typename CT<T>::t* S1,
                                      const typename TW<T>::t* __restrict__ tw, int sgn, int lane, int TRL, int tt, int TT, LD ld,
                                      ST st) {
  typedef typename CT<T>::t C;
  if (pl.flat) for (int i = tt; i < pl.L; i += TT) S0[i * TRL + lane] = ld(i);
  else r_pass_any<T>(pl.s[0], pl.L, tw, sgn, tt, TT, ld, [&](int i, C v) { S0[i * TRL + lane] = v; });
  __syncthreads();
  for (int s = pl.flat ? 0 : 1; s < pl.n - (pl.flat ? 0 : 1); ++s) {
    const RPass& ps = pl.s[s];
    auto lds = [&](int i) -> C { return S0[i * TRL + lane]; };
    auto sts = [&](int i, C v) { S1[i * TRL + lane] = v; };
    switch (ps.p1) {
      case 2: r_pass<T, 2, 1>(ps, pl.L, tw, sgn, tt, TT, lds, sts); break;
      case 3: r_pass<T, 3, 1>(ps, pl.L, tw, sgn, tt, TT, lds, sts); break;
      case 4: r_pass<T, 4, 1>(ps, pl.L, tw, sgn, tt, TT, lds, sts); break;
      case 5: r_pass<T, 5, 1>(ps, pl.L, tw, sgn, tt, TT, lds, sts); break;
    }
    __syncthreads();
    C* t = S0; S0 = S1; S1 = t;
  }
  if (pl.flat) for (int i = tt; i < pl.L; i += TT) st(i, S0[i * TRL + lane]);
  else r_pass_any<T>(pl.s[pl.n - 1], pl.L, tw, sgn, tt, TT, [&](int i) -> C { return S0[i * TRL + lane]; }, st);
}

// z FFT (lines as zfft2_body)
template <typename T>
__global__ void __launch_bounds__(512) k_zfft_r(FSet fs, int nrdim, int npdim, const __grid_constant__ RPlan pl, const typename TW<T>::t* __restrict__ tw,
                                                int sgn, T scale, int m0, int nlines) {
  typedef typename CT<T>::t C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y;
  C* S0 = (C*)smem_raw;
  C* S1 = S0 + pl.L * TRL;
  const int gl = blockIdx.x * TRL + lane;     // line over the set; nlines per field
  const int f = gl / nlines, line = gl - f * nlines;
  const bool ok = f < fs.n;
  const size_t pst = (size_t)nrdim * npdim;
  double2* base = fset_e(fs, ok ? f : 0) + (size_t)nrdim * m0 + line;
  r_fft<T>(pl, S0, S1, tw, sgn, lane, TRL, tt, TT,
           [&](int i) -> C { return ok ? ld<T>(base + (size_t)i * pst) : mk<T>(0, 0); },
           [&](int i, C v) { if (ok) st<T>(base + (size_t)i * pst, c_scale(v, scale)); });
}

// phi forward: packed reals -> X_0..X_L (L = np/2) scaled, in place (lines (r, z)).  Mixed form: X_0 from the FP64 sum of
// the row, taken as ndc partial sums of every ndc-th point, the FP32 transform on the samples minus their FP64 mean
template <typename T>
__global__ void __launch_bounds__(512) k_pfft_fwd_r(FSet fs, int nrdim, int npdim, int nzdim, const __grid_constant__ RPlan pl,
                                                    const typename TW<T>::t* __restrict__ tw,
                                                    const typename TW<T>::t* __restrict__ twr, T scale, double scale_d,
                                                    double inv_np, int nrs, int ndc) {
  typedef typename CT<T>::t C;
  constexpr bool DC = std::is_same<T, float>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y, L = pl.L;
  double2* D = (double2*)smem_raw;             // mixed form: the samples in FP64; S1 takes their place
  C* S1 = (C*)smem_raw;
  C* S0 = DC ? (C*)(D + L * TRL) : S1 + L * TRL;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const double rv = (rs != nullptr && r < nrs) ? rs[r] : 1.0;   // scale_r of the input row
  double sum = 0.0, mu = 0.0;
  if (DC) {
    double* red = (double*)(S0 + L * TRL);
    for (int q = tt; q < ndc; q += TT) {
      double part = 0.0;
      for (int pt = q; pt < L; pt += ndc) {
        const double2 v = ok ? base[(size_t)pt * nrdim] : make_double2(0.0, 0.0);
        D[pt * TRL + lane] = v;
        part += fma(v.x, rv, v.y * rv);
      }
      red[q * TRL + lane] = part;
    }
    __syncthreads();
    for (int q = 0; q < ndc; ++q) sum += red[q * TRL + lane];
    mu = sum * inv_np;
  }
  C* res = (pl.n & 1) ? S0 : S1;               // where the last pass does not read
  r_fft<T>(pl, S0, S1, tw, -1, lane, TRL, tt, TT,
           [&](int i) -> C {
             const double2 d = DC ? D[i * TRL + lane] : ok ? base[(size_t)i * nrdim] : make_double2(0.0, 0.0);
             if (DC) return mk<T>((T)d2f_fast(fma(d.x, rv, -mu)), (T)d2f_fast(fma(d.y, rv, -mu)));
             return mk<T>((T)(d.x * rv), (T)(d.y * rv));
           },
           [&](int i, C v) { res[i * TRL + lane] = v; });
  __syncthreads();
  if (!ok) return;
  for (int k = tt; k <= L; k += TT) {
    C zk = res[(k == L ? 0 : k) * TRL + lane];
    C zc = res[(k == 0 ? 0 : L - k) * TRL + lane];
    zc.y = -zc.y;
    C fe = c_scale(c_add(zk, zc), (T)0.5);
    C fo = c_muli(c_scale(c_sub(zk, zc), (T)0.5), -1);   // (zk - zc)/(2i)
    C x = c_scale(c_add(fe, c_mul(load_tw<T>(twr, k, -1), fo)), scale);
    if (DC && k == 0) base[0] = make_double2(to_dbl(x.x) + sum * scale_d, to_dbl(x.y));
    else st<T>(base + (size_t)k * nrdim, x);
  }
}

// phi backward: X_0..X_L -> packed reals (unnormalised), slot L <- np X_L, in place; mixed form: Re X_0 left out of the FP32
// transform and added to every sample in FP64
template <typename T>
__global__ void __launch_bounds__(512) k_pfft_bwd_r(FSet fs, int nrdim, int npdim, int nzdim, const __grid_constant__ RPlan pl,
                                                    const typename TW<T>::t* __restrict__ tw,
                                                    const typename TW<T>::t* __restrict__ twr, double np_d, int nrs) {
  typedef typename CT<T>::t C;
  constexpr bool DC = std::is_same<T, float>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x, tt = threadIdx.y, TRL = blockDim.x, TT = blockDim.y, L = pl.L;
  C* S0 = (C*)smem_raw;
  C* S1 = S0 + L * TRL;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  const bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const double rv = (rs != nullptr && r < nrs) ? rs[r] : 1.0;   // scale_r of the output row
  double2 nyq = make_double2(0, 0);
  double dc = 0.0;
  if (ok && tt == 0) nyq = base[(size_t)L * nrdim];
  if (DC && ok) dc = base[0].x;
  // X_k enters V_k and V_(L-k): read and rounded once, through shared memory
  for (int i = tt; i <= L; i += TT) {
    C v = ok ? ld<T>(base + (size_t)i * nrdim) : mk<T>(0, 0);
    if (i == 0 || i == L) { v.y = 0; if (DC && i == 0) v.x = 0; }
    S1[i * TRL + lane] = v;
  }
  __syncthreads();
  r_fft<T>(pl, S0, S1, tw, +1, lane, TRL, tt, TT,
           [&](int k) -> C {
             const C xk = S1[k * TRL + lane];
             C xc = S1[(L - k) * TRL + lane];
             xc.y = -xc.y;
             C g = c_add(xk, xc);
             C h = c_mul(c_sub(xk, xc), load_tw<T>(twr, k, +1));   // exp(+2 pi i k / np)
             return c_add(g, c_muli(h, 1));
           },
           [&](int i, C y) {
             if (!ok) return;
             double2 v;
             if (DC) v = make_double2(to_dbl(y.x) + dc, to_dbl(y.y) + dc);
             else v = make_double2((double)y.x, (double)y.y);
             base[(size_t)i * nrdim] = make_double2(v.x * rv, v.y * rv);
           });
  if (ok && tt == 0) base[(size_t)L * nrdim] = make_double2(nyq.x * np_d * rv, nyq.y * np_d * rv);
}

// ------------------------------------------------------------------------------------------------
constexpr int R_FLAT = 32;   // short lengths: one loop over the radices, less code to fetch (32 x 24 mixed: 21 -> 18.5 us)
// the passes of a length: the radices 4, 2, 3, 5 in this order, the first two and the last two of them in one pass where
// their product is at most 16 (not if `single`); at least two passes (a copy, radix 1, stands in)
static int r_plan(int L, RPlan& pl, bool single = false) {
  int f[32], nf = 0, rem = L;
  while (rem > 1) {
    const int p = rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : rem % 5 == 0 ? 5 : 0;
    if (p == 0) return set_error(MLG_ESIZE, "fft: length with a factor other than 2, 3 and 5");
    f[nf++] = p;
    rem /= p;
  }
  pl.L = L;
  pl.n = 0;
  pl.flat = single && L <= R_FLAT && nf > 0;
  int ns = 1;
  auto add = [&](int p1, int p2) {
    if (pl.n < RP_MAX)
      pl.s[pl.n] = {(unsigned char)p1, (unsigned char)p2, (unsigned short)ns, (unsigned short)(L / (p1 * p2)),
                    ns > 1 ? (unsigned)(((1ull << 32) + ns - 1) / ns) : 0u};
    ++pl.n;
    ns *= p1 * p2;
  };
  if (pl.flat) {
    for (int i = 0; i < nf; ++i) add(f[i], 1);
    return 0;
  }
  int a = 0, b = nf;
  if (!single && nf >= 3 && f[0] * f[1] <= 16) { add(f[0], f[1]); a = 2; }
  else { add(nf > 0 ? f[0] : 1, 1); a = nf > 0 ? 1 : 0; }
  const bool lp = !single && nf - a >= 2 && f[nf - 2] * f[nf - 1] <= 16;
  b = nf - (lp ? 2 : nf - a >= 1 ? 1 : 0);
  for (int i = a; i < b; ++i) add(f[i], 1);
  if (lp) add(f[nf - 2], f[nf - 1]);
  else add(b < nf ? f[b] : 1, 1);
  if (pl.n > RP_MAX || L > 65535) return set_error(MLG_ESIZE, "fft: length too large");
  return 0;
}
// lines per CTA: 32, fewer where shared memory (`bytes` a line) would pass 96 KiB
static int r_lines(size_t bytes, int most = 32) {
  int tr = most;
  while (tr > 1 && tr * bytes > 96 * 1024) tr /= 2;
  return tr;
}
// at most: so many that a set of few lines still has a CTA for every SM, but no fewer than two, one 32-byte sector an access
static int r_spread(long long lines) {
  int tr = 32;
  while (tr > 2 && lines / tr < 152) tr /= 2;
  return tr;
}
// With fewer lines than a CTA of 32 for every SM, issue slots are idle and a line's chain of operations is the time: a
// thread then takes one radix at a time (288 lines of 90 points in FP64: 28 -> 14 us; transforms at 40 x 400 x 20, plain:
// 204 -> 133 us)
static bool r_narrow(int most) { return most < 32; }
// threads per line: the fewest thread steps over the passes, or (narrow) the shortest chain of steps
static int r_threads(const RPlan& pl, int lines, bool narrow = false) {
  int best = 1;
  long long cost = -1;
  const int most = std::min(512 / lines, 128);
  for (int t = std::min(5, most); t <= most; ++t) {
    long long c = 0;
    for (int i = 0; i < pl.n; ++i) c += (long long)cdiv(pl.s[i].m, t) * (narrow ? 1 : t) * pl.s[i].p1 * pl.s[i].p2;
    if (cost < 0 || c < cost || (c == cost && !narrow)) { cost = c; best = t; }
  }
  return best;
}
template <class K> static int r_smem(K k, size_t bytes) {
  if (bytes > 48 * 1024) MLG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return 0;
}

template <typename T>
int launch_zfft_r(const FSet& fs, const typename TW<T>::t* tw, int dir, double scale, int m0, int nm,
                  cudaStream_t stream) {
  const int nlines = G.nrdim * nm, most = r_spread((long long)nlines * fs.n);
  RPlan pl;
  MLG_TRY(r_plan(G.nz, pl, r_narrow(most)));
  const size_t per = (size_t)(pl.n > 2 || pl.flat ? 2 : 1) * pl.L * sizeof(typename CT<T>::t);
  const int TRL = r_lines(per, most), TT = r_threads(pl, TRL, r_narrow(most));
  MLG_TRY(r_smem(k_zfft_r<T>, per * TRL));
  k_zfft_r<T><<<cdiv((long long)nlines * fs.n, TRL), dim3(TRL, TT), per * TRL, stream>>>(fs, G.nrdim, G.npdim, pl, tw, dir,
                                                                                       (T)scale, m0, nlines);
  MLG_LAUNCH();
  return 0;
}
// the FP64 sum's partial sums: as many as a CTA of 256 threads over the lines of two FP32 buffers in 96 KiB has threads a line
static int r_dc_parts(int L) {
  const int tr = r_lines(2 * (size_t)L * sizeof(float2));
  return std::max(1, std::min(256 / tr, std::max(L / 2, 1)));
}
template <typename T>
int launch_pfft_r(const FSet& fs, const typename TW<T>::t* tw, const typename TW<T>::t* twr, int dir, double scale) {
  const int most = r_spread((long long)G.nrdim * G.nzdim * fs.n);
  RPlan pl;
  MLG_TRY(r_plan(G.nph, pl, r_narrow(most)));
  const int ndc = std::is_same<T, float>::value ? r_dc_parts(pl.L) : 0;
  const size_t buf = (size_t)pl.L * sizeof(typename CT<T>::t);
  const size_t per = dir > 0 ? 2 * buf + sizeof(typename CT<T>::t)
                             : ndc > 0 ? pl.L * sizeof(double2) + buf + ndc * sizeof(double) : 2 * buf;
  const int TRL = r_lines(per, most);
  int TT = r_threads(pl, TRL, r_narrow(most));
  if (r_narrow(most)) TT = std::max(TT, std::min(std::min(512 / TRL, 64), pl.L + 1));   // one load a thread where they are staged
  const unsigned grid = cdiv((long long)G.nrdim * G.nzdim * fs.n, TRL);
  if (dir < 0) {
    MLG_TRY(r_smem(k_pfft_fwd_r<T>, per * TRL));
    k_pfft_fwd_r<T><<<grid, dim3(TRL, TT), per * TRL, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, pl, tw, twr, (T)scale, scale,
                                                                1.0 / G.np, G.nr, ndc);
  } else {
    MLG_TRY(r_smem(k_pfft_bwd_r<T>, per * TRL));
    k_pfft_bwd_r<T><<<grid, dim3(TRL, TT), per * TRL, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, pl, tw, twr, (double)G.np, G.nr);
  }
  MLG_LAUNCH();
  return 0;
}
template int launch_zfft_r<float>(const FSet&, const float2*, int, double, int, int, cudaStream_t);
template int launch_zfft_r<double>(const FSet&, const double2*, int, double, int, int, cudaStream_t);
template int launch_pfft_r<float>(const FSet&, const float2*, const float2*, int, double);
template int launch_pfft_r<double>(const FSet&, const double2*, const double2*, int, double);

}  // namespace mlg
