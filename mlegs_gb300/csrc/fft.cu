// fft.cu — φ and z FFTs of a field (horizontal_fft_forward/backward, mlegs_scalar_ops.f90:1567-1717;
// vertical_fft_forward/backward, :1721-1848) in FFTE's conventions:
//   forward  X_k = sum_j x_j exp(-2 pi i jk/N), then scaled 1/N (the reference divides after FFTE);
//   backward unnormalised sum with exp(+2 pi i jk/N) (FFTE's 1/N undone by the reference's *N).
// The φ transform is real: PPP stores two real samples per complex slot, z_j = f(2j) + i f(2j+1),
// which is exactly the input of a half-length complex FFT; the usual split step turns its result
// into X_0..X_{N/2}.  Backward, the last complex slot keeps N times its input (FFTE's zdfft2d never
// writes A(NX/2+1), zdfft2d.f:119-128, and the reference then multiplies by N, :1705).
//
// Mixed form (T = float): the DC coefficient of a transform line is carried in FP64 and the FP32 FFT
// runs on the mean-free residual.  Forward, the line's FP64 sum gives the k = 0 output and its mean is
// subtracted (in FP64) before the samples are rounded to FP32; backward, the k = 0 input is left out of
// the FP32 transform and added (in FP64) to every output sample.  A vortex field is dominated by its
// axisymmetric, axially uniform mean flow; without this the FP32 rounding of that mean (relative
// 2^-24 of an O(1) value) would land on every other wavenumber, where the perturbation lives.  The
// φ lines all get it (their DC is the m = 0 coefficient).  The z lines of the m = 0 plane run in FP64.
//
// Layout: a field is (nrdim, npdim, nzdim) with r fastest.  Both transforms run along a strided
// dimension; a CTA takes TR consecutive r (the contiguous batch, so every global access is a run of
// TR*16 bytes) and TT threads per transform, keeps the TR transforms in shared memory as
// [point][TR] and runs a Stockham autosort FFT (radix 4, 2, 3, 5) between two shared buffers.
#include "common.cuh"
#include "fft_common.cuh"
#include <cmath>

namespace mlg {

// the mixed form's FFT arithmetic: FP32 or double-float
#ifndef MLG_MIXED_FFT_DF
#define MLG_MIXED_FFT_DF 0
#endif
typedef std::conditional<MLG_MIXED_FFT_DF != 0, dfl, float>::type MixFT;

// Stockham FFT over the TR transforms held in s0 ([L][TR]); result left in *res.
template <typename T>
__device__ void stockham(typename CT<T>::t* s0, typename CT<T>::t* s1, typename CT<T>::t** res, int L, int TR,
                         int tr, int tt, int TT, const typename TW<T>::t* tw, int sgn) {
  typedef typename CT<T>::t C;
  C* src = s0;
  C* dst = s1;
  int rem = L;
  for (int ns = 1; ns < L;) {
    int p = (rem % 4 == 0) ? 4 : (rem % 2 == 0) ? 2 : (rem % 3 == 0) ? 3 : 5;
    int m = L / p;
    int span = ns * p, twstep = L / span;
    for (int j = tt; j < m; j += TT) {
      int k = j % ns;
      C a[5];
#pragma unroll
      for (int r = 0; r < 5; ++r)
        if (r < p) a[r] = src[(j + r * m) * TR + tr];
      if (k) {
#pragma unroll
        for (int r = 1; r < 5; ++r)
          if (r < p) a[r] = c_mul(a[r], load_tw<T>(tw, (k * r * twstep) % L, sgn));
      }
      dft_small<T>(a, p, sgn);
      int base = (j / ns) * span + k;
#pragma unroll
      for (int r = 0; r < 5; ++r)
        if (r < p) dst[(base + r * ns) * TR + tr] = a[r];
    }
    __syncthreads();
    C* t = src; src = dst; dst = t;
    ns = span;
    rem /= p;
  }
  *res = src;
}

// z FFT of columns (r, m): points at stride nrdim*npdim; the grid covers m = m0, m0+1, ...
template <typename T>
__global__ void k_vfft(double2* __restrict__ e, int nrdim, int npdim, int L, int TR,
                       const typename TW<T>::t* __restrict__ tw, int sgn, T scale, int m0) {
  typedef typename CT<T>::t C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s0 = (C*)smem_raw;
  C* s1 = s0 + (size_t)L * TR;
  int tr = threadIdx.x, tt = threadIdx.y, TT = blockDim.y;
  int r = blockIdx.x * TR + tr;
  int m = blockIdx.y + m0;
  bool ok = r < nrdim;
  size_t pstride = (size_t)nrdim * npdim;
  double2* base = e + r + (size_t)nrdim * m;
  for (int pt = tt; pt < L; pt += TT) s0[pt * TR + tr] = ok ? ld<T>(base + pt * pstride) : mk<T>(0, 0);
  __syncthreads();
  C* res;
  stockham<T>(s0, s1, &res, L, TR, tr, tt, TT, tw, sgn);
  if (ok)
    for (int pt = tt; pt < L; pt += TT) st<T>(base + pt * pstride, c_scale(res[pt * TR + tr], (T)scale));
}

// φ forward: packed reals -> X_0..X_{L} (L = np/2) scaled 1/np, in place.  Mixed form: X_0 from the
// FP64 sum of the row, the FP32 FFT on the samples minus their FP64 mean.
template <typename T>
__global__ void k_hfft_fwd(double2* __restrict__ e, int nrdim, int npdim, int L, int TR,
                           const typename TW<T>::t* __restrict__ tw, const typename TW<T>::t* __restrict__ twr, T scale,
                           double scale_d, double inv_np, const double* __restrict__ rs, int nrs) {
  typedef typename CT<T>::t C;
  constexpr bool DC = std::is_same<T, float>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s0 = (C*)smem_raw;
  C* s1 = s0 + (size_t)L * TR;
  int tr = threadIdx.x, tt = threadIdx.y, TT = blockDim.y;
  int r = blockIdx.x * TR + tr;
  int z = blockIdx.y;
  bool ok = r < nrdim;
  double2* base = e + r + (size_t)nrdim * npdim * z;
  const double rv = (rs != nullptr && ok && r < nrs) ? rs[r] : 1.0;   // scale_r of the input row
  double sum = 0.0, mu = 0.0;
  if (DC) {
    double* red = (double*)(s1 + (size_t)L * TR);
    double part = 0.0;
    if (ok)
      for (int pt = tt; pt < L; pt += TT) { double2 v = base[(size_t)pt * nrdim]; part += v.x * rv + v.y * rv; }
    red[tt * TR + tr] = part;
    __syncthreads();
    for (int q = 0; q < TT; ++q) sum += red[q * TR + tr];
    mu = sum * inv_np;
  }
  for (int pt = tt; pt < L; pt += TT) {
    C v = mk<T>(0, 0);
    if (ok) {
      if (DC) {
        double2 d = base[(size_t)pt * nrdim];
        v = mk<T>((T)d2f_fast(d.x * rv - mu), (T)d2f_fast(d.y * rv - mu));
      } else {
        double2 d = base[(size_t)pt * nrdim];
        v = mk<T>((T)(d.x * rv), (T)(d.y * rv));
      }
    }
    s0[pt * TR + tr] = v;
  }
  __syncthreads();
  C* res;
  stockham<T>(s0, s1, &res, L, TR, tr, tt, TT, tw, -1);
  if (!ok) return;
  for (int k = tt; k <= L; k += TT) {
    C zk = res[(k % L) * TR + tr];
    C zc = res[((L - k) % L) * TR + tr];
    zc.y = -zc.y;
    C fe = c_scale(c_add(zk, zc), (T)0.5);
    C fo = c_muli(c_scale(c_sub(zk, zc), (T)0.5), -1);   // (zk - zc)/(2i)
    typename TW<T>::t wd = twr[k];
    C w = mk<T>(wd.x, wd.y);
    C x = c_scale(c_add(fe, c_mul(w, fo)), (T)scale);
    if (DC && k == 0) {
      base[0] = make_double2(f2d_fast((float)x.x) + sum * scale_d, f2d_fast((float)x.y));
    } else {
      st<T>(base + (size_t)k * nrdim, x);
    }
  }
}

// φ backward: X_0..X_L -> packed reals (unnormalised); slot L <- np * X_L (input), in place.  Mixed
// form: Re X_0 is left out of the FP32 FFT and added to every sample in FP64.
template <typename T>
__global__ void k_hfft_bwd(double2* __restrict__ e, int nrdim, int npdim, int L, int TR,
                           const typename TW<T>::t* __restrict__ tw, const typename TW<T>::t* __restrict__ twr, double np_d,
                           const double* __restrict__ rs, int nrs) {
  typedef typename CT<T>::t C;
  constexpr bool DC = std::is_same<T, float>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s0 = (C*)smem_raw;
  C* s1 = s0 + (size_t)L * TR;
  int tr = threadIdx.x, tt = threadIdx.y, TT = blockDim.y;
  int r = blockIdx.x * TR + tr;
  int z = blockIdx.y;
  bool ok = r < nrdim;
  double2* base = e + r + (size_t)nrdim * npdim * z;
  double2 nyq = make_double2(0, 0);
  double dc = 0.0;
  if (ok && tt == 0) nyq = base[(size_t)L * nrdim];
  if (DC && ok) dc = base[0].x;
  for (int k = tt; k < L; k += TT) {
    C v = mk<T>(0, 0);
    if (ok) {
      C xk = ld<T>(base + (size_t)k * nrdim);
      C xc = ld<T>(base + (size_t)(L - k) * nrdim);
      if (k == 0) { xk.y = 0; xc.y = 0; if (DC) xk.x = 0; }
      xc.y = -xc.y;
      C g = c_add(xk, xc);
      typename TW<T>::t wd = twr[k];
      C w = mk<T>(wd.x, -wd.y);   // exp(+2 pi i k / np)
      C h = c_mul(c_sub(xk, xc), w);
      v = c_add(g, c_muli(h, 1));
    }
    s0[k * TR + tr] = v;
  }
  __syncthreads();
  C* res;
  stockham<T>(s0, s1, &res, L, TR, tr, tt, TT, tw, +1);
  if (!ok) return;
  const double rv = (rs != nullptr && r < nrs) ? rs[r] : 1.0;   // scale_r of the output row
  for (int pt = tt; pt < L; pt += TT) {
    C y = res[pt * TR + tr];
    double2 v;
    if (DC) v = make_double2(f2d_fast((float)y.x) + dc, f2d_fast((float)y.y) + dc);
    else v = make_double2((double)y.x, (double)y.y);
    base[(size_t)pt * nrdim] = make_double2(v.x * rv, v.y * rv);
  }
  if (tt == 0) base[(size_t)L * nrdim] = make_double2(nyq.x * np_d * rv, nyq.y * np_d * rv);
}

template <typename T, int L, int SGN, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2) k_zfft2(FSet fs, int nrdim, int npdim,
                                                              const typename TW<T>::t* __restrict__ tw, T scale, int m0,
                                                              int nlines) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  zfft2_body<T, L, SGN, TRL>(fs, nrdim, npdim, tw, scale, m0, nlines, smem_raw);
}
template <typename T, int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2) k_pfft_fwd2(FSet fs, int nrdim, int npdim, int nzdim,
                                                                  const typename TW<T>::t* __restrict__ tw,
                                                                  const typename TW<T>::t* __restrict__ twr, T scale,
                                                                  double scale_d, double inv_np, int nrs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pfft_fwd2_body<T, L, TRL>(fs, nrdim, npdim, nzdim, tw, twr, scale, scale_d, inv_np, nrs, smem_raw);
}
template <typename T, int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2) k_pfft_bwd2(FSet fs, int nrdim, int npdim, int nzdim,
                                                                  const typename TW<T>::t* __restrict__ tw,
                                                                  const typename TW<T>::t* __restrict__ twr, double np_d,
                                                                  int nrs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pfft_bwd2_body<T, L, TRL>(fs, nrdim, npdim, nzdim, tw, twr, np_d, nrs, smem_raw);
}

// a host-side scale factor in the transform's arithmetic (double-float: hi = the FP32 rounding, lo =
// the FP32 rounding of the rest)
template <typename T> static T host_scale(double v) { return (T)v; }
template <> dfl host_scale<dfl>(double v) { const float h = (float)v; return dfl(h, (float)(v - (double)h)); }

// the twiddle tables of a transform's arithmetic: phi (L = np/2), phi post-processing (np), z (nz)
template <typename T> struct TwTab;
template <> struct TwTab<double> {
  static const double2* p() { return G.tw_p; }
  static const double2* pr() { return G.tw_pr; }
  static const double2* z() { return G.tw_z; }
};
template <> struct TwTab<float> {
  static const float2* p() { return G.tw_p32; }
  static const float2* pr() { return G.tw_pr32; }
  static const float2* z() { return G.tw_z32; }
};
template <> struct TwTab<dfl> {
  static const float4* p() { return G.tw_pdf; }
  static const float4* pr() { return G.tw_prdf; }
  static const float4* z() { return G.tw_zdf; }
};

static int pick_tr(int L, size_t elem) {
  // two shared buffers of L*TR complex values, at most 96 KB
  int tr = 32;
  while (tr > 1 && 2ull * L * tr * elem > 96 * 1024) tr /= 2;
  return tr;
}

template <typename T>
static int set_smem(const void* fn, size_t bytes) {
  if (bytes > 48 * 1024) MLG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return 0;
}

static FSet fset1(cd* e, const double* rs = nullptr) {
  FSet fs{};
  fs.e[0] = e; fs.rs[0] = rs; fs.n = 1;
  return fs;
}

template <typename T, int L, int SGN, int TRL>
static int zfft2_launch(const FSet& fs, double scale, int m0, int nm, cudaStream_t stream) {
  size_t sm = (size_t)L * TRL * sizeof(typename CT<T>::t);
  MLG_TRY(set_smem<T>((const void*)k_zfft2<T, L, SGN, TRL>, sm));
  const int nlines = G.nrdim * nm;
  dim3 grid(cdiv((long long)nlines * fs.n, TRL)), blk(TRL, Split<L>::R2);
  k_zfft2<T, L, SGN, TRL><<<grid, blk, sm, stream>>>(fs, G.nrdim, G.npdim, TwTab<T>::z(), host_scale<T>(scale), m0,
                                                     nlines);
  MLG_LAUNCH();
  return 0;
}
template <typename T, int L, int TRL>
static int zfft2_dir(const FSet& fs, int dir, double scale, int m0, int nm, cudaStream_t stream) {
  return dir < 0 ? zfft2_launch<T, L, -1, TRL>(fs, scale, m0, nm, stream) : zfft2_launch<T, L, +1, TRL>(fs, scale, m0, nm, stream);
}
template <typename T, int TRL>
static int zfft2_any(const FSet& fs, int dir, double scale, int m0, int nm, cudaStream_t stream) {
  switch (G.nz) {
    case 16: return zfft2_dir<T, 16, TRL>(fs, dir, scale, m0, nm, stream);
    case 32: return zfft2_dir<T, 32, TRL>(fs, dir, scale, m0, nm, stream);
    case 64: return zfft2_dir<T, 64, TRL>(fs, dir, scale, m0, nm, stream);
    case 128: return zfft2_dir<T, 128, TRL>(fs, dir, scale, m0, nm, stream);
    case 256: return zfft2_dir<T, 256, TRL>(fs, dir, scale, m0, nm, stream);
  }
  return -1;
}
static bool pow2_fast(int L) { return L == 16 || L == 32 || L == 64 || L == 128 || L == 256; }

template <typename T>
static int vfft_t(const FSet& fs, int dir, double scale, int m0, int nm, int tr_max, cudaStream_t stream) {
  int L = G.nz;
  if (L <= 1 || nm <= 0) return 0;
  if (pow2_fast(L)) {
    if (tr_max >= 32) return zfft2_any<T, 32>(fs, dir, scale, m0, nm, stream);
    // a single plane (m = 0): four lines per CTA, so that its few hundred lines spread over most SMs
    return tr_max >= 8 ? zfft2_any<T, 8>(fs, dir, scale, m0, nm, stream) : zfft2_any<T, 4>(fs, dir, scale, m0, nm, stream);
  }
  if constexpr (std::is_same<T, dfl>::value) {
    return vfft_t<double>(fs, dir, scale, m0, nm, tr_max, stream);   // other lengths: the FP64 Stockham kernel
  } else {
  int TR = std::min(pick_tr(L, sizeof(typename CT<T>::t)), tr_max);
  int TT = std::max(1, std::min(256 / TR, L / 2));
  size_t sm = 2ull * L * TR * sizeof(typename CT<T>::t);
  MLG_TRY(set_smem<T>((const void*)k_vfft<T>, sm));
  dim3 grid(cdiv(G.nrdim, TR), nm), blk(TR, TT);
  for (int f = 0; f < fs.n; ++f) {   // other lengths: the Stockham kernel, field by field
    k_vfft<T><<<grid, blk, sm, stream>>>(fs.e[f], G.nrdim, G.npdim, L, TR, TwTab<T>::z(), dir, (T)scale, m0);
    MLG_LAUNCH();
  }
  return 0;
  }
}

// plain form: FP64.  Mixed form: m >= 1 in FP32; the m = 0 lines (the axisymmetric part, with the mean
// flow in its k = 0 coefficient) in FP64, in small CTAs so that they spread over the SMs.
static int vfft_any(const FSet& fs, int dir, double scale) {
  kt_begin(1);
  if (G.precision == MLG_MIXED) {
    MLG_TRY(side_fork());
    MLG_TRY(vfft_t<double>(fs, dir, scale, 0, 1, 2, G.side));
    MLG_TRY(vfft_t<MixFT>(fs, dir, scale, 1, G.npdim - 1, 32, G.stream));
    MLG_TRY(side_join());
  } else {
    int sexp;
    if (fftq_length(G.nz) && std::frexp(scale, &sexp) == 0.5) MLG_TRY(launch_zfft_q(fs, dir, sexp - 1));
    else MLG_TRY(vfft_t<double>(fs, dir, scale, 0, G.npdim, 32, G.stream));
  }
  kt_end(1, 2.0 * fs.n * G.fsize * 16);
  return 0;
}

int launch_vfft_buf(cd* e, int dir) { return vfft_any(fset1(e), dir, dir < 0 ? 1.0 / G.nz : 1.0); }
// sum_j x_j exp(dir 2 pi i jk/nz) * scale, any direction and scale (the adjoint's FFTs)
int launch_vfft_scaled(cd* e, int dir, double scale) { return vfft_any(fset1(e), dir, scale); }
int launch_vfft(Scalar& s, int dir) { return launch_vfft_buf(s.e, dir); }
// the z transform of n fields in one pass (forward scaled by 1/nz)
int launch_vfft_multi(Scalar* const* s, int n, int dir) {
  if (n < 1 || n > FS_MAX) return set_error(MLG_EPARAM, "vertical_fft: 1 to 6 fields per batch");
  FSet fs{};
  for (int i = 0; i < n; ++i) { fs.e[i] = s[i]->e; fs.rs[i] = nullptr; }
  fs.n = n;
  return vfft_any(fs, dir, dir < 0 ? 1.0 / G.nz : 1.0);
}

template <typename T, int L>
static int pfft2_launch(const FSet& fs, int dir, double scale) {
  constexpr int TRL = 32;
  constexpr bool DC = !std::is_same<T, double>::value;
  size_t sm = (size_t)L * TRL * sizeof(typename CT<T>::t) + (DC && dir < 0 ? (size_t)Split<L>::R2 * TRL * sizeof(double) : 0);
  dim3 grid(cdiv((long long)G.nrdim * G.nzdim * fs.n, TRL)), blk(TRL, Split<L>::R2);
  if (dir < 0) {
    MLG_TRY(set_smem<T>((const void*)k_pfft_fwd2<T, L, TRL>, sm));
    k_pfft_fwd2<T, L, TRL><<<grid, blk, sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, TwTab<T>::p(),
                                                        TwTab<T>::pr(), host_scale<T>(scale), scale, 1.0 / G.np, G.nr);
  } else {
    MLG_TRY(set_smem<T>((const void*)k_pfft_bwd2<T, L, TRL>, sm));
    k_pfft_bwd2<T, L, TRL><<<grid, blk, sm, G.stream>>>(fs, G.nrdim, G.npdim, G.nzdim, TwTab<T>::p(),
                                                        TwTab<T>::pr(), (double)G.np, G.nr);
  }
  MLG_LAUNCH();
  return 0;
}

template <typename T>
static int hfft_t(const FSet& fs, int dir, double scale) {
  int L = G.nph;
  if (G.np <= 1) return 0;
  kt_begin(1);
  if constexpr (std::is_same<T, double>::value) {   // the plain form
    int sexp = 1;
    if (fftq_length(L) && (dir > 0 || std::frexp(scale, &sexp) == 0.5)) {
      MLG_TRY(launch_pfft_q(fs, dir, dir > 0 ? 0 : sexp - 1));
      kt_end(1, 2.0 * fs.n * G.fsize * 16);
      return 0;
    }
  }
  if (pow2_fast(L)) {
    switch (L) {
      case 16: MLG_TRY((pfft2_launch<T, 16>(fs, dir, scale))); break;
      case 32: MLG_TRY((pfft2_launch<T, 32>(fs, dir, scale))); break;
      case 64: MLG_TRY((pfft2_launch<T, 64>(fs, dir, scale))); break;
      case 128: MLG_TRY((pfft2_launch<T, 128>(fs, dir, scale))); break;
      case 256: MLG_TRY((pfft2_launch<T, 256>(fs, dir, scale))); break;
    }
    kt_end(1, 2.0 * fs.n * G.fsize * 16);
    return 0;
  }
  if constexpr (std::is_same<T, dfl>::value) {
    kt_end(1, 0.0);
    return hfft_t<double>(fs, dir, scale);   // other lengths: the FP64 Stockham kernels
  } else {
  int TR = pick_tr(L, sizeof(typename CT<T>::t));
  int TT = std::max(1, std::min(256 / TR, std::max(L / 2, 1)));
  constexpr bool DC = std::is_same<T, float>::value;
  size_t sm = 2ull * L * TR * sizeof(typename CT<T>::t) + (DC ? (size_t)TT * TR * sizeof(double) : 0);
  dim3 grid(cdiv(G.nrdim, TR), G.nzdim), blk(TR, TT);
  if (dir < 0) MLG_TRY(set_smem<T>((const void*)k_hfft_fwd<T>, sm));
  else MLG_TRY(set_smem<T>((const void*)k_hfft_bwd<T>, sm));
  for (int f = 0; f < fs.n; ++f) {   // other lengths: the Stockham kernels, field by field
    if (dir < 0) {
      k_hfft_fwd<T><<<grid, blk, sm, G.stream>>>(fs.e[f], G.nrdim, G.npdim, L, TR, TwTab<T>::p(),
                                                  TwTab<T>::pr(), (T)scale,
                                                  scale, 1.0 / G.np, fs.rs[f], G.nr);
    } else {
      k_hfft_bwd<T><<<grid, blk, sm, G.stream>>>(fs.e[f], G.nrdim, G.npdim, L, TR, TwTab<T>::p(),
                                                  TwTab<T>::pr(), (double)G.np, fs.rs[f], G.nr);
    }
    MLG_LAUNCH();
  }
  kt_end(1, 2.0 * fs.n * G.fsize * 16);
  return 0;
  }
}

int launch_hfft(Scalar& s, int dir) { return launch_hfft_rs(s, dir, nullptr); }
// with rs: the rows i < nr of the field times rs[i] before the forward transform / after the
// backward one (scale_r folded into the transform)
int launch_hfft_rs(Scalar& s, int dir, const double* rs) {
  Scalar* ps = &s;
  return launch_hfft_multi(&ps, &rs, 1, dir);
}
// the phi transform of n fields in one pass, field i's rows times rs[i] (before the forward / after
// the backward transform) where rs[i] is not null
int launch_hfft_multi(Scalar* const* s, const double* const* rs, int n, int dir) {
  if (n < 1 || n > FS_MAX) return set_error(MLG_EPARAM, "horizontal_fft: 1 to 6 fields per batch");
  FSet fs{};
  for (int i = 0; i < n; ++i) {
    if (G.npchop + s[i]->off[1] > G.npdim)
      return set_error(MLG_ECHOP, dir < 0 ? "horizontal_fft_forward: chopping in p too large"
                                          : "horizontal_fft_fbackard: chopping in p too large");
    fs.e[i] = s[i]->e; fs.rs[i] = rs ? rs[i] : nullptr;
  }
  fs.n = n;
  return G.precision == MLG_MIXED ? hfft_t<MixFT>(fs, dir, 1.0 / G.np) : hfft_t<double>(fs, dir, 1.0 / G.np);
}
static FSet fset_n(cd* const* e, int n) {
  FSet fs{};
  for (int i = 0; i < n; ++i) { fs.e[i] = e[i]; fs.rs[i] = nullptr; }
  fs.n = n;
  return fs;
}
// the real-to-half-complex sum scaled by `scale` instead of 1/np (the adjoint's FFTs), of n <= 6 buffers
int launch_hfft_fwd_scaled_n(cd* const* e, int n, double scale) {
  if (n < 1 || n > FS_MAX) return set_error(MLG_EPARAM, "horizontal_fft: 1 to 6 fields per batch");
  const FSet fs = fset_n(e, n);
  return G.precision == MLG_MIXED ? hfft_t<MixFT>(fs, -1, scale) : hfft_t<double>(fs, -1, scale);
}
int launch_hfft_fwd_scaled(cd* e, double scale) { return launch_hfft_fwd_scaled_n(&e, 1, scale); }
// the half-complex-to-real sum (unnormalised, Nyquist slot kept times np), on n <= 6 raw buffers
int launch_hfft_bwd_buf_n(cd* const* e, int n) {
  if (n < 1 || n > FS_MAX) return set_error(MLG_EPARAM, "horizontal_fft: 1 to 6 fields per batch");
  const FSet fs = fset_n(e, n);
  return G.precision == MLG_MIXED ? hfft_t<MixFT>(fs, +1, 1.0) : hfft_t<double>(fs, +1, 1.0);
}
int launch_hfft_bwd_buf(cd* e) { return launch_hfft_bwd_buf_n(&e, 1); }
// the z sum of n <= 6 buffers, any direction and scale
int launch_vfft_scaled_n(cd* const* e, int n, int dir, double scale) {
  if (n < 1 || n > FS_MAX) return set_error(MLG_EPARAM, "vertical_fft: 1 to 6 fields per batch");
  return vfft_any(fset_n(e, n), dir, scale);
}

}  // namespace mlg
