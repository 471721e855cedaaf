// fft_common.cuh — the FFTs' small transforms, typed loads and stores, and the register two-pass transforms of
// power-of-two lengths (fft.cu: FP32 and FP64; fftq.cu: fixed point, with the FP64 transforms for lines outside its
// range).
#pragma once
#include "common.cuh"
#include "dfloat.cuh"
#include "xs_common.cuh"
#include <type_traits>

namespace mlg {

template <typename T> struct CT;
template <> struct CT<double> { typedef double2 t; };
template <> struct CT<float> { typedef float2 t; };
template <> struct CT<dfl> { typedef dfl2 t; };

template <typename T> __device__ __forceinline__ typename CT<T>::t mk(T a, T b);
template <> __device__ __forceinline__ double2 mk<double>(double a, double b) { return make_double2(a, b); }
template <> __device__ __forceinline__ float2 mk<float>(float a, float b) { return make_float2(a, b); }
template <> __device__ __forceinline__ dfl2 mk<dfl>(dfl a, dfl b) { dfl2 r; r.x = a; r.y = b; return r; }

template <typename C> __device__ __forceinline__ C c_add(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C c_sub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C> __device__ __forceinline__ C c_mul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
template <typename C> __device__ __forceinline__ C c_muli(C a, int sgn) {  // a * (sgn * i), exact
  C r; r.x = sgn > 0 ? -a.y : a.y; r.y = sgn > 0 ? a.x : -a.x; return r;
}
template <typename C, typename T> __device__ __forceinline__ C c_scale(C a, T s) { C r; r.x = a.x * s; r.y = a.y * s; return r; }

// twiddle tables hold exp(-2 pi i k/L) (FP64 for the plain form; FP32, or double-float as (re hi,
// re lo, im hi, im lo), for the mixed form); sgn > 0 conjugates
template <typename T> struct TW;
template <> struct TW<double> { typedef double2 t; };
template <> struct TW<float> { typedef float2 t; };
template <> struct TW<dfl> { typedef float4 t; };
template <typename T>
__device__ __forceinline__ typename CT<T>::t load_tw(const typename TW<T>::t* tw, int idx, int sgn) {
  typename TW<T>::t w = tw[idx];
  return mk<T>(w.x, sgn < 0 ? w.y : -w.y);
}
template <>
__device__ __forceinline__ dfl2 load_tw<dfl>(const float4* tw, int idx, int sgn) {
  const float4 w = tw[idx];
  const dfl im(w.z, w.w);
  return mk<dfl>(dfl(w.x, w.y), sgn < 0 ? im : -im);
}
// h + l rounded to FP64 on the integer pipe, for a normalised double-float (|l| <= ulp(h)/2, so l's
// exponent is at least 23 below h's): both significands in one 64-bit integer, h's at bits 38..61,
// then one rounding; GB300's FP64 pipe (about 2 operations per clock per SM) stays free
__device__ __forceinline__ double df_to_double(float h, float l) {
  const unsigned bh = __float_as_uint(h), bl = __float_as_uint(l);
  const int eh = (int)((bh >> 23) & 0xFFu), el = (int)((bl >> 23) & 0xFFu);
  if (eh == 0) return f2d_fast(l);
  long long X = (long long)((bh & 0x7FFFFFu) | 0x800000u) << 38;
  if (bh >> 31) X = -X;
  const int d = eh - el;
  if (el != 0 && d < 62) {
    const long long ml = (long long)((bl & 0x7FFFFFu) | 0x800000u);
    const long long L = d <= 38 ? (ml << (38 - d)) : (ml >> (d - 38));
    X += (bl >> 31) ? -L : L;
  }
  return xs_i64_to_double(X, eh - 150 - 38);
}
// a transform value to FP64 (FP32 and double-float on the integer pipe)
__device__ __forceinline__ double to_dbl(double v) { return v; }
__device__ __forceinline__ double to_dbl(float v) { return f2d_fast(v); }
__device__ __forceinline__ double to_dbl(dfl v) { return df_to_double(v.h, v.l); }

// a double-float sample in the transform's arithmetic
template <typename T> __device__ __forceinline__ T from_df(dfl v);
template <> __device__ __forceinline__ float from_df<float>(dfl v) { return v.h; }
template <> __device__ __forceinline__ dfl from_df<dfl>(dfl v) { return v; }

// small DFTs, sign sgn = -1 forward, +1 backward
template <typename T>
__device__ __forceinline__ void dft_small(typename CT<T>::t* a, int p, int sgn) {
  typedef typename CT<T>::t C;
  if (p == 2) {
    C t = a[0]; a[0] = c_add(t, a[1]); a[1] = c_sub(t, a[1]);
  } else if (p == 4) {
    C t0 = c_add(a[0], a[2]), t1 = c_sub(a[0], a[2]), t2 = c_add(a[1], a[3]), t3 = c_muli(c_sub(a[1], a[3]), sgn);
    a[0] = c_add(t0, t2); a[2] = c_sub(t0, t2); a[1] = c_add(t1, t3); a[3] = c_sub(t1, t3);
  } else if (p == 3) {
    const T c1 = (T)-0.5, s1 = (T)0.86602540378443864676372317075294;  // cos(2pi/3), sin(2pi/3)
    C t1 = c_add(a[1], a[2]), t2 = c_sub(a[1], a[2]);
    C m1 = c_add(a[0], c_scale(t1, c1));
    C m2 = c_muli(c_scale(t2, s1), sgn);
    a[0] = c_add(a[0], t1); a[1] = c_add(m1, m2); a[2] = c_sub(m1, m2);
  } else if (p == 5) {
    const T c1 = (T)0.30901699437494742410229341718282, c2 = (T)-0.80901699437494742410229341718282;
    const T s1 = (T)0.95105651629515357211643933337938, s2 = (T)0.58778525229247312916870595463907;
    C t1 = c_add(a[1], a[4]), t2 = c_add(a[2], a[3]), t3 = c_sub(a[1], a[4]), t4 = c_sub(a[2], a[3]);
    C m1 = c_add(a[0], c_add(c_scale(t1, c1), c_scale(t2, c2)));
    C m2 = c_add(a[0], c_add(c_scale(t1, c2), c_scale(t2, c1)));
    C n1 = c_muli(c_add(c_scale(t3, s1), c_scale(t4, s2)), sgn);
    C n2 = c_muli(c_sub(c_scale(t3, s2), c_scale(t4, s1)), sgn);
    a[0] = c_add(a[0], c_add(t1, t2));
    a[1] = c_add(m1, n1); a[4] = c_sub(m1, n1);
    a[2] = c_add(m2, n2); a[3] = c_sub(m2, n2);
  }
}

template <typename T> __device__ __forceinline__ typename CT<T>::t ld(const double2* p);
template <> __device__ __forceinline__ double2 ld<double>(const double2* p) { return *p; }
template <> __device__ __forceinline__ float2 ld<float>(const double2* p) { return ld_c32(p); }
template <> __device__ __forceinline__ dfl2 ld<dfl>(const double2* p) {
  const double2 v = *p;
  return mk<dfl>(dfl(v.x), dfl(v.y));
}
template <typename T> __device__ __forceinline__ void st(double2* p, typename CT<T>::t v);
template <> __device__ __forceinline__ void st<double>(double2* p, double2 v) { *p = v; }
template <> __device__ __forceinline__ void st<float>(double2* p, float2 v) { st_c32(p, v); }
template <> __device__ __forceinline__ void st<dfl>(double2* p, dfl2 v) { *p = make_double2(to_dbl(v.x), to_dbl(v.y)); }

// ------------------------------------------------------------------------------------------------
// Power-of-two lengths 16..256: two passes through registers.  L = R1 * R2, n = n2 + R2 n1,
// k = k1 + R1 k2:  X_k = sum_n2 w_L^(n2 k1) [sum_n1 x_n w_R1^(n1 k1)] w_R2^(n2 k2).
// A CTA holds TRL lines (consecutive r: every global access is a run of TRL*16 bytes) and R2 threads
// per line; pass 1: each thread loads R1 points of its line and does the R1-point DFT in registers,
// multiplies by w_L^(n2 k1) and stores to shared memory [k1][n2][line]; pass 2: each thread does
// R1/R2 DFTs of R2 points and writes the results.  Every element is read and written once in HBM and
// once in shared memory, with compile-time index arithmetic.

// cos and sin of 2 pi j / 16 (j mod 16)
__host__ __device__ constexpr double cos16(int j) {
  return (j & 15) == 0 ? 1.0 : (j & 15) == 1 ? 0.92387953251128675613 : (j & 15) == 2 ? 0.70710678118654752440
       : (j & 15) == 3 ? 0.38268343236508977173 : (j & 15) == 4 ? 0.0 : (j & 15) == 5 ? -0.38268343236508977173
       : (j & 15) == 6 ? -0.70710678118654752440 : (j & 15) == 7 ? -0.92387953251128675613 : (j & 15) == 8 ? -1.0
       : (j & 15) == 9 ? -0.92387953251128675613 : (j & 15) == 10 ? -0.70710678118654752440
       : (j & 15) == 11 ? -0.38268343236508977173 : (j & 15) == 12 ? 0.0 : (j & 15) == 13 ? 0.38268343236508977173
       : (j & 15) == 14 ? 0.70710678118654752440 : 0.92387953251128675613;
}
__host__ __device__ constexpr double sin16(int j) { return cos16(j - 4); }

// v * exp(SGN 2 pi i j / 16)
template <typename T, int SGN>
__device__ __forceinline__ typename CT<T>::t tw16(typename CT<T>::t v, int j) {
  typedef typename CT<T>::t C;
  j &= 15;
  if (j == 0) return v;
  if (j == 8) { C r; r.x = -v.x; r.y = -v.y; return r; }
  if (j == 4) return c_muli(v, SGN);
  if (j == 12) return c_muli(v, -SGN);
  C w; w.x = (T)cos16(j); w.y = (T)(SGN * sin16(j));
  return c_mul(v, w);
}

__host__ __device__ constexpr int bitrev(int i, int n) {   // bit reversal of i in log2(n) bits
  int r = 0;
  for (int b = 1; b < n; b <<= 1) { r = (r << 1) | (i & 1); i >>= 1; }
  return r;
}

// in-register DFT of N <= 16 points, sign SGN: radix-2 decimation in frequency, fully unrolled, so
// every register index is a compile-time constant; the result comes out in bit-reversed order,
// a[i] = X_bitrev(i), and the callers fold the reversal into their memory addresses
template <typename T, int N, int SGN>
__device__ __forceinline__ void dft_reg(typename CT<T>::t* a) {
  typedef typename CT<T>::t C;
#pragma unroll
  for (int len = N; len >= 2; len >>= 1) {
#pragma unroll
    for (int i = 0; i < N; i += len) {
#pragma unroll
      for (int k = 0; k < len / 2; ++k) {
        C u = a[i + k], v = a[i + k + len / 2];
        a[i + k] = c_add(u, v);
        a[i + k + len / 2] = tw16<T, SGN>(c_sub(u, v), k * (16 / len));
      }
    }
  }
}

template <int L> struct Split;            // L = R1 * R2, R1 >= R2, R1 <= 16
template <> struct Split<16> { static constexpr int R1 = 4, R2 = 4; };
template <> struct Split<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct Split<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct Split<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct Split<256> { static constexpr int R1 = 16, R2 = 16; };

// the two passes on a CTA's lines; a[] holds the R1 inputs of this thread (n1 order); on return
// b[q][i] holds X_(k1 + R1 bitrev(i)) for k1 = w*(R1/R2) + q
template <typename T, int L, int SGN, int TRL>
__device__ __forceinline__ void fft2pass(typename CT<T>::t* a, typename CT<T>::t (*b)[Split<L>::R2],
                                         typename CT<T>::t* S, const typename TW<T>::t* __restrict__ tw, int w,
                                         int lane) {
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2;
  dft_reg<T, R1, SGN>(a);
#pragma unroll
  for (int i = 0; i < R1; ++i) {
    const int k1 = bitrev(i, R1);
    typename CT<T>::t v = a[i];
    if (k1) v = c_mul(v, load_tw<T>(tw, (w * k1) & (L - 1), SGN));
    S[(k1 * R2 + w) * TRL + lane] = v;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    int k1 = w * Q + q;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) b[q][n2] = S[(k1 * R2 + n2) * TRL + lane];
    dft_reg<T, R2, SGN>(b[q]);
  }
}

// a set of fields transformed by one launch (the components of a vector field, stage by stage): their
// lines are taken flat, field after field, so that one launch has enough blocks to fill the GPU
constexpr int FS_MAX = 6;
struct FSet {
  double2* e[FS_MAX];
  const double* rs[FS_MAX];   // per field: the row scaling of the phi transforms, or null
  int n;
};
// field f's pointers by a chain of selects: an indexed access to the kernel parameter would copy the
// whole set to local memory
__device__ __forceinline__ double2* fset_e(const FSet& fs, int f) {
  double2* p = fs.e[0];
#pragma unroll
  for (int q = 1; q < FS_MAX; ++q) p = f == q ? fs.e[q] : p;
  return p;
}
__device__ __forceinline__ const double* fset_rs(const FSet& fs, int f) {
  const double* p = fs.rs[0];
#pragma unroll
  for (int q = 1; q < FS_MAX; ++q) p = f == q ? fs.rs[q] : p;
  return p;
}

// z FFT: the lines (r, m) of m in [m0, m0 + nm) taken flat, line r + nrdim*(m - m0) at offset
// r + nrdim*m (so a block's lanes read one run of consecutive offsets and no block is left ragged at
// the end of an m), points at stride nrdim*npdim
template <typename T, int L, int SGN, int TRL>
__device__ __forceinline__ void zfft2_body(const FSet& fs, int nrdim, int npdim,
                                            const typename TW<T>::t* __restrict__ tw, T scale, int m0, int nlines,
                                            unsigned char* smem_raw) {
  typedef typename CT<T>::t C;
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2;
  C* S = (C*)smem_raw;
  int lane = threadIdx.x, w = threadIdx.y;
  const int gl = blockIdx.x * TRL + lane;     // line over the set; nlines per field
  const int f = gl / nlines, line = gl - f * nlines;
  bool ok = f < fs.n;
  size_t ps = (size_t)nrdim * npdim;
  double2* base = fset_e(fs, ok ? f : 0) + (size_t)nrdim * m0 + line;
  C a[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) a[n1] = ok ? ld<T>(base + (size_t)(w + R2 * n1) * ps) : mk<T>(0, 0);
  C b[Q][R2];
  fft2pass<T, L, SGN, TRL>(a, b, S, tw, w, lane);
  if (!ok) return;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i) st<T>(base + (size_t)(k1 + R1 * bitrev(i, R2)) * ps, c_scale(b[q][i], scale));
  }
}

// φ forward: packed reals -> X_0..X_L scaled, in place (lines (r, z)); mixed form: X_0 from the FP64
// sum of the row, the FP32 transform on the samples minus their FP64 mean
template <typename T, int L, int TRL>
__device__ __forceinline__ void pfft_fwd2_body(const FSet& fs, int nrdim, int npdim, int nzdim,
                                                                  const typename TW<T>::t* __restrict__ tw,
                                                                  const typename TW<T>::t* __restrict__ twr, T scale,
                                                                  double scale_d, double inv_np, int nrs, unsigned char* smem_raw) {
  typedef typename CT<T>::t C;
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2;
  constexpr bool DC = !std::is_same<T, double>::value;
  C* S = (C*)smem_raw;
  double* red = (double*)(smem_raw + (size_t)L * TRL * sizeof(C));
  int lane = threadIdx.x, w = threadIdx.y;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  const bool rsc = rs != nullptr && ok && r < nrs;   // the row's samples times rs[r] first (scale_r)
  const double rv = rsc ? rs[r] : 1.0;
  C a[R1];
  double sum = 0.0;
  if constexpr (DC) {
    // the row scale, the row sum and the mean subtraction in double-float (about 47 bits, on the FP32
    // and integer pipes; FP64 would occupy GB300's narrow FP64 pipe with 4-6 operations per sample);
    // the samples less their mean are then rounded to FP32 for the transform
    dfl dx[R1], dy[R1];
    dfl part(0);
    const dfl rvd = rsc ? dfl(rv) : dfl(1);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      const double2 v = ok ? base[(size_t)(w + R2 * n1) * nrdim] : make_double2(0.0, 0.0);
      dx[n1] = dfl(v.x);
      dy[n1] = dfl(v.y);
      if (rsc) { dx[n1] = dx[n1] * rvd; dy[n1] = dy[n1] * rvd; }
      part = part + dx[n1] + dy[n1];
    }
    dfl* redf = reinterpret_cast<dfl*>(red);
    redf[w * TRL + lane] = part;
    __syncthreads();
    dfl sd(0);
#pragma unroll
    for (int q = 0; q < R2; ++q) sd = sd + redf[q * TRL + lane];
    const dfl mu = sd * dfl((float)inv_np, 0.f);   // inv_np = 1/np, a power of two for these lengths
    sum = f2d_fast(sd.h) + f2d_fast(sd.l);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) a[n1] = mk<T>(from_df<T>(dx[n1] - mu), from_df<T>(dy[n1] - mu));
  } else {
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      if (rsc) {
        double2 d = base[(size_t)(w + R2 * n1) * nrdim];
        a[n1] = mk<T>((T)(d.x * rv), (T)(d.y * rv));
      } else {
        a[n1] = ok ? ld<T>(base + (size_t)(w + R2 * n1) * nrdim) : mk<T>(0, 0);
      }
    }
  }
  C b[Q][R2];
  fft2pass<T, L, -1, TRL>(a, b, S, tw, w, lane);
  __syncthreads();   // every thread has read its pass-2 inputs: S can take the spectrum
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i) S[(k1 * R2 + bitrev(i, R2)) * TRL + lane] = b[q][i];   // Z_(k1 + R1 k2)
  }
  __syncthreads();
  if (!ok) return;
  auto Z = [&](int k) -> C { return S[((k % R1) * R2 + k / R1) * TRL + lane]; };
  for (int k = w; k <= L; k += R2) {
    C zk = Z(k & (L - 1));
    C zc = Z((L - k) & (L - 1));
    zc.y = -zc.y;
    C fe = c_scale(c_add(zk, zc), (T)0.5);
    C fo = c_muli(c_scale(c_sub(zk, zc), (T)0.5), -1);   // (zk - zc)/(2i)
    C x = c_scale(c_add(fe, c_mul(load_tw<T>(twr, k, -1), fo)), scale);
    bool dc0 = false;
    if constexpr (DC) dc0 = k == 0;
    if (dc0) base[0] = make_double2(to_dbl(x.x) + sum * scale_d, to_dbl(x.y));
    else st<T>(base + (size_t)k * nrdim, x);
  }
}

// φ backward: X_0..X_L -> packed reals (unnormalised), slot L <- np X_L, in place; mixed form: Re X_0
// left out of the FP32 transform and added to every sample in FP64
template <typename T, int L, int TRL>
__device__ __forceinline__ void pfft_bwd2_body(const FSet& fs, int nrdim, int npdim, int nzdim,
                                                                  const typename TW<T>::t* __restrict__ tw,
                                                                  const typename TW<T>::t* __restrict__ twr, double np_d,
                                                                  int nrs, unsigned char* smem_raw) {
  typedef typename CT<T>::t C;
  constexpr int R1 = Split<L>::R1, R2 = Split<L>::R2, Q = R1 / R2;
  constexpr bool DC = !std::is_same<T, double>::value;
  C* S = (C*)smem_raw;
  int lane = threadIdx.x, w = threadIdx.y;
  const int per = nrdim * nzdim;               // the lines (r, z) of a field taken flat: r + nrdim*z
  const int gl = blockIdx.x * TRL + lane;
  const int f = gl / per, line = gl - f * per;
  bool ok = f < fs.n;
  const int r = line % nrdim, z = line / nrdim;
  double2* base = fset_e(fs, ok ? f : 0) + r + (size_t)nrdim * npdim * z;
  const double* rs = ok ? fset_rs(fs, f) : nullptr;
  double2 nyq = make_double2(0, 0);
  double dc = 0.0;
  if (ok && w == 0) nyq = base[(size_t)L * nrdim];
  if (DC && ok) dc = base[0].x;
  C a[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    int k = w + R2 * n1;
    C v = mk<T>(0, 0);
    if (ok) {
      C xk = ld<T>(base + (size_t)k * nrdim);
      C xc = ld<T>(base + (size_t)(L - k) * nrdim);
      if (k == 0) { xk.y = 0; xc.y = 0; if (DC) xk.x = 0; }
      xc.y = -xc.y;
      C g = c_add(xk, xc);
      C h = c_mul(c_sub(xk, xc), load_tw<T>(twr, k, +1));   // exp(+2 pi i k / np)
      v = c_add(g, c_muli(h, 1));
    }
    a[n1] = v;
  }
  C b[Q][R2];
  fft2pass<T, L, +1, TRL>(a, b, S, tw, w, lane);
  if (!ok) return;
  const bool rsc = rs != nullptr && r < nrs;   // every slot of the row times rs[r] last (scale_r)
  const double rv = rsc ? rs[r] : 1.0;
  const double dcr = dc * rv;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    int k1 = w * Q + q;
#pragma unroll
    for (int i = 0; i < R2; ++i) {
      C y = b[q][i];
      double2* o = base + (size_t)(k1 + R1 * bitrev(i, R2)) * nrdim;
      double2 v;
      if constexpr (DC) {
        // (y + dc) rv as one FMA per component
        v = rsc ? make_double2(fma(to_dbl(y.x), rv, dcr), fma(to_dbl(y.y), rv, dcr))
                : make_double2(to_dbl(y.x) + dc, to_dbl(y.y) + dc);
      } else {
        v = make_double2((double)y.x, (double)y.y);
        if (rsc) { v.x *= rv; v.y *= rv; }
      }
      *o = v;
    }
  }
  if (w == 0) {
    double2 v = make_double2(nyq.x * np_d, nyq.y * np_d);
    if (rsc) { v.x *= rv; v.y *= rv; }
    base[(size_t)L * nrdim] = v;
  }
}

// ------------------------------------------------------------------------------------------------
// Other lengths: one or two Stockham stages in registers
struct RPass { unsigned char p1, p2; unsigned short ns, m; unsigned magic; };   // radices, points combined before it, butterfly pairs, ceil(2^32 / ns)
// a b with the roundings fixed (one product of each component is rounded, the other is added to it unrounded), so that it does
// not depend on how a compiler contracts the sums: an FP32 transform's last bits reach the spectrum of a mixed run
template <typename C> __device__ __forceinline__ C r_mul(C a, C b) {
  C r;
  r.x = fma(a.x, b.x, -(a.y * b.y));
  r.y = fma(a.y, b.x, a.x * b.y);
  return r;
}
// one pass over a line's L points: butterfly pair j takes the points j + m i, i < p1 p2, as p2 transforms of radix p1 over
// groups combined ns at a time, then p1 of radix p2
template <typename T, int P1, int P2, class LD, class ST>
__device__ __forceinline__ void r_pass(const RPass& ps, int L, const typename TW<T>::t* __restrict__ tw, int sgn, int tt,
                                       int TT, LD ld, ST st) {
  typedef typename CT<T>::t C;
  constexpr int R = P1 * P2;
  const int m = ps.m, ns = ps.ns;
  const int st2 = ns == 1 ? m : (int)__umulhi((unsigned)m, ps.magic), st1 = st2 * P2;   // L / (ns p1 p2), L / (ns p1)
  for (int j = tt; j < m; j += TT) {
    const int q = ns == 1 ? j : (int)__umulhi((unsigned)j, ps.magic), k = j - q * ns;
    C a[P2][P1];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i % P2][i / P2] = ld(j + m * i);
    if (k) {
#pragma unroll
      for (int r1 = 1; r1 < P1; ++r1) {
        const C w = load_tw<T>(tw, k * r1 * st1, sgn);
#pragma unroll
        for (int r2 = 0; r2 < P2; ++r2) a[r2][r1] = r_mul(a[r2][r1], w);
      }
    }
#pragma unroll
    for (int r2 = 0; r2 < P2; ++r2) dft_small<T>(a[r2], P1, sgn);
    const int base = q * ns * R + k;
#pragma unroll
    for (int r1 = 0; r1 < P1; ++r1) {
      C b[P2];
#pragma unroll
      for (int r2 = 0; r2 < P2; ++r2) b[r2] = a[r2][r1];
      const int kb = k + r1 * ns;
      if (P2 > 1 && kb) {
#pragma unroll
        for (int r2 = 1; r2 < P2; ++r2) b[r2] = r_mul(b[r2], load_tw<T>(tw, kb * r2 * st2, sgn));
      }
      dft_small<T>(b, P2, sgn);
#pragma unroll
      for (int r2 = 0; r2 < P2; ++r2) st(base + ns * (r1 + r2 * P1), b[r2]);
    }
  }
}

// fixed-point transforms of power-of-two lengths (fftq.cu), the plain form's: z (scale 2^sexp), phi forward (2^sexp) and
// backward
int launch_zfft_q(const FSet& fs, int dir, int sexp);
int launch_pfft_q(const FSet& fs, int dir, int sexp);
// and of products of two of 2..6, 8, 9, 10, 12, 15 and 16 (fftqr.cu), with any FP64 scale
int launch_zfft_qr(const FSet& fs, int dir, double scale);
int launch_pfft_qr(const FSet& fs, int dir, double scale);
// transforms of other lengths (fftr.cu), FP32 and FP64: z on the planes m0 .. m0 + nm - 1, phi
// forward (scaled) and backward
template <typename T>
int launch_zfft_r(const FSet& fs, const typename TW<T>::t* tw, int dir, double scale, int m0, int nm,
                  cudaStream_t stream);
template <typename T>
int launch_pfft_r(const FSet& fs, const typename TW<T>::t* tw, const typename TW<T>::t* twr, int dir, double scale);

}  // namespace mlg
