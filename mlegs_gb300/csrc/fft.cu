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
// dimension; a CTA takes TRL consecutive lines (the contiguous batch, so every global access is a run of
// TRL*16 bytes) and several threads per line, which exchange through shared memory as [point][TRL].
// Lengths: powers of two from 16 to 256 here (the mixed form) and in fftq.cu (the plain one); others in fftr.cu and, for the
// plain form where they split into two passes, in fftqr.cu.
#include "common.cuh"
#include "fft_common.cuh"
#include <cmath>

namespace mlg {

// the mixed form's FFT arithmetic: FP32 or double-float
#ifndef MLG_MIXED_FFT_DF
#define MLG_MIXED_FFT_DF 0
#endif
typedef std::conditional<MLG_MIXED_FFT_DF != 0, dfl, float>::type MixFT;

// CTAs an SM is to hold, of 256 threads (80 and 64 registers a thread instead of 95 to 120 and 80); smaller CTAs are left to the
// compiler, whose choice is the faster there
constexpr int fft_ctas(int threads, int n) { return threads == 256 ? n : 0; }

template <typename T, int L, int SGN, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, fft_ctas(TRL * Split<L>::R2, 4)) k_zfft2(FSet fs, int nrdim, int npdim,
                                                              const typename TW<T>::t* __restrict__ tw, T scale, int m0,
                                                              int nlines) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  zfft2_body<T, L, SGN, TRL>(fs, nrdim, npdim, tw, scale, m0, nlines, smem_raw);
}
template <typename T, int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, fft_ctas(TRL * Split<L>::R2, 3)) k_pfft_fwd2(FSet fs, int nrdim, int npdim, int nzdim,
                                                                  const typename TW<T>::t* __restrict__ tw,
                                                                  const typename TW<T>::t* __restrict__ twr, T scale,
                                                                  double scale_d, double inv_np, int nrs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pfft_fwd2_body<T, L, TRL>(fs, nrdim, npdim, nzdim, tw, twr, scale, scale_d, inv_np, nrs, smem_raw);
}
template <typename T, int L, int TRL>
__global__ void __launch_bounds__(TRL * Split<L>::R2, fft_ctas(TRL * Split<L>::R2, 3)) k_pfft_bwd2(FSet fs, int nrdim, int npdim, int nzdim,
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
  // of fftr.cu's transforms in the plain form: correctly rounded where the kit has them (lengths whose larger sets run in
  // fixed point): of 690 lines at np = 60 the worst phi backward is 4.4 units of 2^-53 with rounded angles, below 4 so
  static bool plain() { return G.precision != MLG_MIXED; }
  static const double2* rp() { return plain() && G.tw_pqd ? G.tw_pqd : G.tw_p; }
  static const double2* rpr() { return plain() && G.tw_prqd ? G.tw_prqd : G.tw_pr; }
  static const double2* rz() { return plain() && G.tw_zqd ? G.tw_zqd : G.tw_z; }
};
template <> struct TwTab<float> {
  static const float2* p() { return G.tw_p32; }
  static const float2* pr() { return G.tw_pr32; }
  static const float2* z() { return G.tw_z32; }
  static const float2* rp() { return G.tw_p32; }
  static const float2* rpr() { return G.tw_pr32; }
  static const float2* rz() { return G.tw_z32; }
};
template <> struct TwTab<dfl> {
  static const float4* p() { return G.tw_pdf; }
  static const float4* pr() { return G.tw_prdf; }
  static const float4* z() { return G.tw_zdf; }
};

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

// lines per CTA: 16 from 64 points on, so that several CTAs of 128 or 256 threads share an SM and one loads while another
// computes (32 lines of 256 points, 512 threads at 86 to 120 registers, left an SM with one: 12 transforms of three fields at
// 512 x 512 x 256, mixed, 15.3 -> 12.9 ms, and 10.9 with fft_ctas)
constexpr int fft_lines(int L) { return L >= 64 ? 16 : 32; }

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
template <typename T, int MOST>
static int zfft2_any(const FSet& fs, int dir, double scale, int m0, int nm, cudaStream_t stream) {
  switch (G.nz) {
    case 16: return zfft2_dir<T, 16, std::min(MOST, fft_lines(16))>(fs, dir, scale, m0, nm, stream);
    case 32: return zfft2_dir<T, 32, std::min(MOST, fft_lines(32))>(fs, dir, scale, m0, nm, stream);
    case 64: return zfft2_dir<T, 64, std::min(MOST, fft_lines(64))>(fs, dir, scale, m0, nm, stream);
    case 128: return zfft2_dir<T, 128, std::min(MOST, fft_lines(128))>(fs, dir, scale, m0, nm, stream);
    case 256: return zfft2_dir<T, 256, std::min(MOST, fft_lines(256))>(fs, dir, scale, m0, nm, stream);
  }
  return -1;
}
static bool pow2_fast(int L) { return L == 16 || L == 32 || L == 64 || L == 128 || L == 256; }

template <typename T>
static int vfft_t(const FSet& fs, int dir, double scale, int m0, int nm, cudaStream_t stream) {
  int L = G.nz;
  if (L <= 1 || nm <= 0) return 0;
  if (pow2_fast(L)) {
    // FP64: the mixed form's m = 0 plane alone, four lines per CTA, so that its few hundred lines spread over most SMs (a plain
    // field's lines are in fixed point, but for a scale that is no power of two)
    if constexpr (!std::is_same<T, double>::value) return zfft2_any<T, 32>(fs, dir, scale, m0, nm, stream);
    else if (nm == 1) return zfft2_any<T, 4>(fs, dir, scale, m0, nm, stream);
  }
  if constexpr (std::is_same<T, dfl>::value) {
    return vfft_t<double>(fs, dir, scale, m0, nm, stream);   // other lengths: FP64
  } else {
    return launch_zfft_r<T>(fs, TwTab<T>::rz(), dir, scale, m0, nm, stream);
  }
}

// plain form: FP64.  Mixed form: m >= 1 in FP32; the m = 0 lines (the axisymmetric part, with the mean
// flow in its k = 0 coefficient) in FP64, in small CTAs so that they spread over the SMs.
static int vfft_any(const FSet& fs, int dir, double scale) {
  kt_begin(1);
  if (G.precision == MLG_MIXED) {
    MLG_TRY(side_fork());
    MLG_TRY(vfft_t<double>(fs, dir, scale, 0, 1, G.side));
    MLG_TRY(vfft_t<MixFT>(fs, dir, scale, 1, G.npdim - 1, G.stream));
    MLG_TRY(side_join());
  } else {
    int sexp;
    if (fftq_length(G.nz) && std::frexp(scale, &sexp) == 0.5) MLG_TRY(launch_zfft_q(fs, dir, sexp - 1));
    else if (fftqr_pays(G.nz, (long long)G.nrdim * G.npdim * fs.n)) MLG_TRY(launch_zfft_qr(fs, dir, scale));
    else MLG_TRY(vfft_t<double>(fs, dir, scale, 0, G.npdim, G.stream));
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
  constexpr int TRL = fft_lines(L);
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
    if (fftqr_pays(L, (long long)G.nrdim * G.nzdim * fs.n)) {
      MLG_TRY(launch_pfft_qr(fs, dir, scale));
      kt_end(1, 2.0 * fs.n * G.fsize * 16);
      return 0;
    }
  }
  if constexpr (!std::is_same<T, double>::value) {
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
  }
  if constexpr (std::is_same<T, dfl>::value) {
    kt_end(1, 0.0);
    return hfft_t<double>(fs, dir, scale);   // other lengths: FP64
  } else {
    MLG_TRY(launch_pfft_r<T>(fs, TwTab<T>::rp(), TwTab<T>::rpr(), dir, scale));
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
