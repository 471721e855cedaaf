// xs_radial.cu — the radial Legendre contractions as exact-slice products on the 5th-generation tensor
// cores (rtrans_forward, mlegs_scalar_ops.f90:1852-1927; rtrans_backward, :1931-2008).
//
// Method (the Ozaki scheme of error-free matrix products).  Every row of the table operand A has a
// power-of-two scale 2^EA (|A(row, k)| < 2^EA) and every column of the field operand B one of 2^EB;
// both are cut into NS signed digits of w bits,
//   A(row, k) ~ 2^(EA - nb) sum_t a_t 2^(w (NS-1-t)),   nb = w NS,  a_t integer, |a_t| < 2^w,
// by rounding A 2^(nb - EA) to an integer (so the representation error is at most 2^(EA - nb - 1)).  Every digit is
// an exact BF16 and every digit product an exact FP32 integer.  The products of one digit order
// d = t + s are summed over K in their own FP32 accumulator in tensor memory,
//   G_d = sum_{t+s=d} sum_k a_t(row, k) b_s(k, n),
// which stays exact while K (d+1) (largest digit product) <= 2^24.  Orders d < NO = NS are kept; the epilogue forms the
// integer T = sum_d G_d 2^(w (NO-1-d)) in 64 bits (its lowest bits shifted out where it would not fit) and rounds
// T 2^(EA + EB + const) once to FP64, on the integer pipe.
// The result differs from the exact product of the FP64 operands by what the dropped orders hold, about 2^-(nb - 2) of
// max|A(row,:)| max|B(:,n)|: 63 bits, in eight or nine balanced digits, for the plain form, 42 bits for the mixed form.  Where
// FP64 sums were the plain form's alternative (nine digits), the outputs whose terms are all small beside those maxima, points
// near the axis for one, are found by a contraction of the magnitudes and summed again in FP64 (xs_least_sum, k_xs_again): each
// output is as near to the exact sum of its terms as an FP64 sum.  A column of the plain form with a NaN or an infinity gives
// NaN, or what an FP64 sum gives (nine digits).  No floating-point rounding happens anywhere else: the forward fold f(i) +- f(nr-1-i) is an exact
// integer sum of the two rounded samples, and the quadrature weights are folded into the table (A = pf w, one FP64
// rounding at kit init).
//
// Forward: per m and row parity par, C_par(t, n) = sum_{i < nr/2} A_par(t, i) B_par(i, n) with
//   A_par(t, i) = pf(i, 2t+par, m) w(i),  B_par(i, n) = f(i) + (-1)^par f(nr-1-i)  (n: re/im of z),
//   c(2t+par, m, z) = C_par(t, n); one column scale per n for both parities (the fold may double),
//   one row scale per (par, t).
// Backward: D_par(i, n) = sum_t A_par(i, t) B_par(t, n) with A_par(i, t) = pf(i, 2t+par, m),
//   B_par(t, n) = c(2t+par, m, z); f(i) = D_0 + D_1, f(nr-1-i) = D_0 - D_1, formed exactly in the
//   integers, so both parities share one row scale per i and one column scale per n; the log term
//   ln * lnx(i) is added at m = 0 (trans, :194).
//
// Engine: a persistent grid of one CTA per SM.  A work item is one (m, tile of NZ complex z columns); the CTA
//  * bulk-copies the item's FP64 field columns (NZ runs of consecutive r, each contiguous in HBM) into
//    shared memory on the TMA engine, completing on an mbarrier, and scans them for the column scales;
//  * per row tile, parity and K chunk of 16: the table digits arrive by one bulk copy (pre-split at kit init in the
//    UMMA canonical no-swizzle K-major layout), the digit warps cut the field digits from shared memory into the same
//    layout (each warp's 32 stores in 32 banks), and one thread issues the chunk's tcgen05.mma and commits.  The field
//    digits lie side by side (digit s at rows s N .. s N + N-1 of the B operand) and so do the accumulators of the
//    orders, so table digit t meets all field digits s <= NO-1-t in one MMA of M = 128, N = (NO - t) 2 NZ, K = 16 whose
//    column block s lands on order t + s: NO MMAs per stage instead of NO (NO+1)/2, and each table tile is read
//    from shared memory once;
//  * reads the NO accumulators of a parity back with tcgen05.ld and, after the second parity, writes FP64 results.
// Every wait is bounded (about a second of SM clock): a timeout sets the library's timeout word and the
// CTA stops issuing work, waits (bounded) for what it issued, frees its tensor memory and returns.
#include "common.cuh"
#include "tc_common.cuh"
#include "xs_common.cuh"
#include <cstdint>

namespace mlg {

constexpr int XS_KC = 16;                         // K per chunk: one MMA K step
constexpr int XS_THREADS = 896;
constexpr int XS_ATILE = 128 * XS_KC * 2;         // 4 KiB: 128 rows x 16 K of BF16
constexpr int XS_SBO = XS_KC * 16;                // between 8-row core-matrix groups
constexpr int XS_LBO = 128;                       // between the two 8-K core matrices of a row group
__host__ __device__ constexpr int xs_off(int row, int k) {
  return (row >> 3) * XS_SBO + (k >> 3) * XS_LBO + (row & 7) * 16 + (k & 7) * 2;
}

// ------------------------------------------------------------------------------------------------
// kit-time table images
// fwd rows (par, t), K = i: A = pf(i, 2t+par, m) w(i); bwd rows i, K = t: A = pf(i, 2t+par, m)
__device__ __forceinline__ double xs_a(const double* __restrict__ pf, const double* __restrict__ w, int mode, int row,
                                       int k, int par, int m, int nn, int nrh, int ne) {
  const int i = mode == 0 ? k : row, t = mode == 0 ? row : k, j = 2 * t + par;
  if (j >= nn || i >= nrh) return 0.0;
  const double v = pf[i + (size_t)nrh * (j + (size_t)ne * m)];
  return mode == 0 ? v * w[i] : v;
}

// row scales: fwd aexp[(m * 2 + par) * nrp + t], bwd aexp[m * nrp + i] (both parities); -2000: all zero
__global__ void k_xs_aexp(const double* __restrict__ pf, const double* __restrict__ w, int* __restrict__ aexp, int mode,
                          int nrh, int ne, int nrc, int nrp, int nk, int bal) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y, nn = max(min(nrc, nrc - m), 0);
  if (row >= nrp) return;
  for (int p = 0; p < (mode == 0 ? 2 : 1); ++p) {
    unsigned long long mx = 0;
    for (int par = (mode == 0 ? p : 0); par <= (mode == 0 ? p : 1); ++par)
      for (int k = 0; k < nk; ++k) {
        unsigned long long v = (unsigned long long)__double_as_longlong(xs_a(pf, w, mode, row, k, par, m, nn, nrh, ne)) &
                               0x7FFFFFFFFFFFFFFFull;
        mx = v > mx ? v : mx;
      }
    aexp[(size_t)(mode == 0 ? m * 2 + p : m) * nrp + row] = !mx ? -2000 : bal ? xs_ebound_bal((unsigned)(mx >> 32)) : xs_ebound(mx);
  }
}

// the digit configuration of a digit count: 6 or 9 digits of 7 bits, 7 or 10 of 6, 8 of 8; eight and nine digits are
// balanced
template <int NS> __host__ __device__ constexpr int xs_w() { return NS == 8 ? 8 : NS == 7 || NS == 10 ? 6 : 7; }
template <int NS> __host__ __device__ constexpr bool xs_bal() { return NS == 8 || NS == 9; }
template <int NS> __host__ __device__ constexpr int xs_nb() { return xs_bal<NS>() ? 63 : xs_w<NS>() * NS; }
// nine digits carry a magnitude tile beside them (xs_least_sum); it costs 7 % (velocity and vorticity at 512 x 512 x 256:
// 17.0 -> 18.2 ms, where FP64 sums took 159)
template <int NS> __host__ __device__ constexpr int xs_mag() { return NS == 9 ? 1 : 0; }

// digit tiles of 128 rows x 16 K: [m][row tile mt][par][chunk kc][digit t, then the magnitudes]
template <int NS>
__global__ void k_xs_table(const double* __restrict__ pf, const double* __restrict__ w, const int* __restrict__ aexp,
                           uint16_t* __restrict__ img, int mode, int nrh, int ne, int nrc, int nmt, int nkc, int nrp) {
  constexpr int W = xs_w<NS>();
  const size_t blk = blockIdx.x;   // (m * nmt + mt) * nkc + kc
  const int kc = (int)(blk % nkc), mt = (int)((blk / nkc) % nmt), m = (int)(blk / ((size_t)nkc * nmt));
  const int nn = max(min(nrc, nrc - m), 0);
  constexpr int TILES = NS + xs_mag<NS>();
  uint8_t* base = (uint8_t*)img + ((blk / nkc) * 2 * nkc + kc) * (size_t)(TILES * XS_ATILE);
  const size_t pstep = (size_t)nkc * TILES * XS_ATILE;   // from the even to the odd parity
  for (int idx = threadIdx.x; idx < 2 * 128 * XS_KC; idx += blockDim.x) {
    const int k = idx % XS_KC, r = (idx / XS_KC) % 128, par = idx / (XS_KC * 128);
    const int row = mt * 128 + r, kk = kc * XS_KC + k;
    int E = -2000;
    double a = 0.0;
    if (row < nrp) {
      E = aexp[(size_t)(mode == 0 ? m * 2 + par : m) * nrp + row];
      a = xs_a(pf, w, mode, row, kk, par, m, nn, nrh, ne);
    }
    const long long A = xs_fix(a, E, xs_nb<NS>());
    const unsigned long long X = (unsigned long long)A + (xs_bal<NS>() ? xs_bias<NS, W>() : 0ull);
    xs_static_for<NS>([&](auto tc) {
      constexpr int t = decltype(tc)::value;
      *(uint16_t*)(base + par * pstep + t * XS_ATILE + xs_off(r, k)) = (uint16_t)xs_digit2<NS, W, xs_bal<NS>(), t>(X, X);
    });
    if (xs_mag<NS>()) *(uint16_t*)(base + par * pstep + NS * XS_ATILE + xs_off(r, k)) = (uint16_t)xs_mag2(A, A);
  }
}

// ------------------------------------------------------------------------------------------------
// up to XS_NF fields with the same chop, transformed by one launch (the components of a vector field)
constexpr int XS_NF = 3;
struct XsArgs {
  const double2* in[XS_NF];
  double2* out[XS_NF];
  const double* lnp[XS_NF];
  const uint16_t* img;
  const int* aexp;
  const double* lnx;
  int* status;
  int add_ln, nf, nr, nrh, nrdim, npdim, nzdim, nrc, m0, npc, nmt, nkc, nrp, rawk;
  int aent, bst, nraw;   // ring sizes: table entries and field-digit stages (one parity of a chunk), field-column buffers
  int sent;              // and magnitude tiles
  unsigned* again;       // nine digits: the outputs to be summed again, a word of 32 rows (xs_word)
  int ngrp;
  float least;           // xs_least_sum
};
// the word of the rows 32 g .. 32 g + 31 (of parity par, forward) of column (m, z) of field f
__device__ __forceinline__ size_t xs_word(const XsArgs& a, int mode, int f, int m, int par, int g, int z) {
  return ((((size_t)f * a.npc + m) * (mode == 0 ? 2 : 1) + par) * a.ngrp + g) * a.nzdim + z;
}
// field f's pointer without an indexed access to the kernel parameters (which would copy them to local
// memory)
template <class P> __device__ __forceinline__ P xs_sel(const P (&p)[XS_NF], int f) {
  return f == 0 ? p[0] : (f == 1 ? p[1] : p[2]);
}

__device__ __forceinline__ bool xs_wait(uint64_t* bar, uint32_t phase, bool& ok) {
  if (!ok) return false;
  ok = mbar_wait(bar, phase);
  return ok;
}
// a bounded wait whose outcome every lane of the warp shares (the warp-collective operations that
// follow need the whole warp)
__device__ __forceinline__ bool xs_wait_w(uint64_t* bar, uint32_t phase, bool& ok) {
  xs_wait(bar, phase, ok);
  ok = __all_sync(0xFFFFFFFFu, ok);
  return ok;
}

// Warp roles of the contraction kernel (896 threads, one CTA per SM):
//   warp 0        the table entries and magnitude tiles, by bulk copy (one thread)
//   warp 1        MMA issue and the tensor-memory allocation
//   warps 2, 3    the items' field columns, by bulk copy (one thread), and their scales
//   warps 4..11   field digits, in two groups that take the stages in turn
//   warps 12..27  epilogue: tensor memory -> 64-bit order sums -> FP64 results
// A work unit is one parity of a row tile of an item: its accumulators are NO N columns, so that two sets fit tensor
// memory (one with nine digits and 32 columns) and the MMAs of a unit run while the epilogue reads the one before.
// Every hand-off is an mbarrier: the table entries, their magnitude tiles and the field-digit stages (one parity of a chunk
// each) are rings, the field columns are one buffer (the next item's columns land while the MMAs and the epilogue of this one run).  The
// epilogue keeps the even parity's sums in registers and writes both parities' results after the odd unit.
// What bounds it (clock64 traces, 192 points, six digits, about 13 000 cycles an item): the integer pipe, on which the
// digits, the order sums and the conversions take about 8 000 of them; the MMAs need 4 000 (7 400 while one lane issued
// them from a branch: 3.70 ms below).  A cluster of two CTAs sharing the table entries by multicast measured the same.
// Ten steps' radial transforms at 192 x 128 x 128, mixed: 4.27 -> 3.49 ms against eight-warp epilogues that released both
// parities together and reduced the scales themselves (20 700 cycles an item); 512 x 512 x 256, two mixed steps:
// 22.4 -> 15.1 ms; plain: 2.48 -> 1.70 ms for four steps.
constexpr int XS_SBMAX = 4, XS_AEMAX = 8, XS_MEMAX = 2;   // ring sizes (at most)
constexpr int XS_CXS = 4;                   // column-scale slots (items)
constexpr int XS_NSW = 2, XS_NDW = 8, XS_NEW = 16;   // scale warps (2, 3), digit warps (4..11), epilogue warps (12..27)
constexpr int XS_NG = 2;                    // groups of digit warps (at most the digit stages: a group waits at most one phase ahead)
constexpr int XS_NEPI = XS_NEW * 32;
constexpr int XS_NBAR = 4 + 2 * XS_AEMAX + 2 * XS_MEMAX + 2 * XS_SBMAX + 4 + 2 * XS_CXS;
static_assert(2 + XS_NSW + XS_NDW + XS_NEW == XS_THREADS / 32, "warp roles");

// MODE 0 forward, 1 backward; NS digits (and orders), NZ complex z columns per item
// right shift of the unsigned digits' 64-bit order sums: |G_d| < 2^24 / (pairs) keeps sum_d G_d 2^(w (NS-1-d) - ESH)
// below 2^62
template <int NS> __host__ __device__ constexpr int xs_esh() {
  return 24 + xs_w<NS>() * (NS - 1) - 62 > 0 ? 24 + xs_w<NS>() * (NS - 1) - 62 : 0;
}
// The plain form's order sums.  A fixed shift that keeps K max|A| max|B| within 64 bits would cut the sums at 2^-52 of
// max|A| max|B|, far above what the digits hold (2^-61, the dropped orders), and rows whose largest table entries meet
// small coefficients (the innermost points, where the Legendre functions grow like a power of the degree) would lose
// bits that FP64 keeps.  So the sum of the orders from 2 on, L = sum_{d>=2} G_d 2^(w (NO-1-d) - low), is formed exactly
// (but for the last order's `low` bits), and added to C = G_0 2^w + G_1 with the smallest shift that fits:
// T = C 2^(cb - esh) + (L >> esh), cb = w (NO-2) - low.
// low: |G_2| <= K (2^(2w-2) + 2 2^(w+6)) and the orders below it keep |L| < 2^63 (8 digits: 3 2^21 2^40) or, with K <=
// 372 and nine digits, 2^22.9 2^(42 - 3)
template <int NS> __host__ __device__ constexpr int xs_low() { return NS == 9 ? 3 : 0; }
template <int NS> __host__ __device__ constexpr int xs_cb() { return xs_w<NS>() * (NS - 2) - xs_low<NS>(); }
// the shift for a sum with |C| = mx: |T| <= (mx + 2^16) 2^(cb - esh) < 2^62 (|L| 2^-cb <= 2^16), so that the sum of two
// fits 64 bits too; at most 15, since |C| < 2^30 (nine digits, K <= 372) or 2^29 (eight, K <= 113)
template <int NS> __device__ __forceinline__ int xs_order_shift(int mx) {
  return max(32 - __clz(mx + 65536) + xs_cb<NS>() - 62, 0);
}
// T += v 2^SH (floor for SH < 0), SH a compile-time constant: one wide multiply-add for 0 <= SH <= 30
template <int SH> __device__ __forceinline__ void xs_acc(long long& T, int v) {
  if constexpr (SH > 30) T += (long long)v << SH;
  else if constexpr (SH >= 0) T += (long long)v * (long long)(1 << SH);
  else T += (long long)v >> (-SH);
}
template <int NO, int W, int ESH, int D> __device__ __forceinline__ void xs_acc_order(long long& T, uint32_t g) {
  xs_acc<W * (NO - 1 - D) - ESH>(T, xs_f2i(__uint_as_float(g)));
}

// CW consecutive columns of tensor memory into each lane (no wait)
template <int CW> __device__ __forceinline__ void xs_tmem_ld(uint32_t taddr, uint32_t* r) {
  static_assert(CW == 4 || CW == 8, "columns of an epilogue warp");
  if constexpr (CW == 8) tmem_ld8_nw(taddr, r);
  else tmem_ld4_nw(taddr, r);
}

template <int MODE, int NS, int NZ>
__global__ void __launch_bounds__(XS_THREADS, 1) k_xs_rtrans(XsArgs a) {
  constexpr int NO = NS;
  constexpr int W = xs_w<NS>(), ESH = xs_esh<NS>(), nb = xs_nb<NS>();
  constexpr bool BAL = xs_bal<NS>();
  constexpr bool PLAIN = NS >= 8;                 // else the mixed form's digits
  constexpr int N = 2 * NZ;                       // real columns (MMA N per digit)
  constexpr int BT = N * XS_KC * 2;               // B digit tile bytes
  constexpr int AENT = NS * XS_ATILE;             // a table entry: the digits of one parity of a chunk
  constexpr bool MAG = xs_mag<NS>() != 0;         // with magnitude sums
  constexpr int TILES = NS + xs_mag<NS>();        // tiles of a table entry's image and of a digit stage
  constexpr int BSTAGE = TILES * BT;
  constexpr int ACC = (NO + xs_mag<NS>()) * N;    // accumulator columns of a unit
  constexpr int TB = 2 * ACC <= 512 ? 2 : 1;      // sets of them
  constexpr int TUSE = TB * ACC;
  constexpr int TCOLS = TUSE <= 128 ? 128 : TUSE <= 256 ? 256 : 512;
  constexpr int NBLK = (N / 8) * 2;               // digit blocks per stage
  constexpr int NG = XS_NG, GW = XS_NDW / NG;     // digit groups, warps of a group
  constexpr int CW = N / 4;                       // columns of an epilogue warp
  static_assert(ACC <= 512, "accumulators exceed tensor memory");
  static_assert(N == 16 || N == 32, "MMA N per digit");
  static_assert(NBLK % GW == 0, "digit blocks per warp");
  extern __shared__ __align__(1024) uint8_t xs_smem_raw[];
  uint8_t* sbase = (uint8_t*)(((uintptr_t)xs_smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t AE = (uint32_t)a.aent, SB = (uint32_t)a.bst, ME = MAG ? (uint32_t)a.sent : 0u;
  const int RB = a.nraw;
  uint8_t* sA = sbase;                                   // [AE][AENT]
  uint8_t* sM = sA + AE * AENT;                          // [ME][XS_ATILE]
  uint8_t* sB = sM + ME * XS_ATILE;                      // [SB][BSTAGE]
  double* raw0 = (double*)(sB + SB * BSTAGE);            // [RB][NZ][rawk] complex (re, im)
  const size_t rawsz = (size_t)2 * NZ * a.rawk;
  int* colexp = (int*)(raw0 + RB * rawsz);               // [XS_CXS][N], by item
  uint64_t* bars = (uint64_t*)(colexp + XS_CXS * N);
  uint64_t* bar_rf = bars;                 // [RB] field columns landed
  uint64_t* bar_re = bars + 2;             // [RB] field columns consumed (digit threads)
  uint64_t* bar_af = bars + 4;             // [AE] table entry landed
  uint64_t* bar_ae = bar_af + XS_AEMAX;    // [AE] table entry consumed (MMA commit)
  uint64_t* bar_mf = bar_ae + XS_AEMAX;    // [ME] magnitude tile landed
  uint64_t* bar_me = bar_mf + XS_MEMAX;    // [ME] magnitude tile consumed (MMA commit)
  uint64_t* bar_bf = bar_me + XS_MEMAX;    // [SB] digit stage written (the group's digit threads)
  uint64_t* bar_be = bar_bf + XS_SBMAX;    // [SB] digit stage consumed (MMA commit)
  uint64_t* bar_tf = bar_be + XS_SBMAX;    // [TB] accumulators complete (MMA commit)
  uint64_t* bar_te = bar_tf + 2;           // [TB] accumulators read (epilogue threads)
  uint64_t* bar_cx = bar_te + 2;           // [XS_CXS] column scales written (scale threads)
  uint64_t* bar_ce = bar_cx + XS_CXS;      // [XS_CXS] column scales read (epilogue threads: the item's last readers)
  uint32_t* tslot = (uint32_t*)(bar_ce + XS_CXS);

  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;   // warp: uniform
  if (tid < XS_NBAR) {   // a barrier per thread
    const int i = tid;
    const uint64_t* q = bars + i;
    mbar_init(bars + i, q == bar_re || q == bar_re + 1 ? XS_NDW * 32
                        : q >= bar_bf && q < bar_be    ? GW * 32
                        : q >= bar_te && q < bar_cx    ? XS_NEPI
                        : q >= bar_cx && q < bar_ce    ? XS_NSW * 32
                        : q >= bar_ce                  ? XS_NEPI
                                                       : 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tslot, TCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  bool ok = true;

  // the CTA's items (field, m, z tile), item = ((m - m0) nzt + z tile) nf + field, those without rows
  // skipped; every role walks the same sequence
  const int nzt = (a.nzdim + NZ - 1) / NZ;
  const int nitems = (a.npc - a.m0) * nzt * a.nf;
  auto item_m = [&](int item) { return a.m0 + item / (nzt * a.nf); };
  auto item_z0 = [&](int item) { return ((item / a.nf) % nzt) * NZ; };
  auto item_f = [&](int item) { return item % a.nf; };
  auto item_nn = [&](int item) { const int m = item_m(item); return max(min(a.nrc, a.nrc - m), 0); };
  auto next_item = [&](int item) {
    for (item += gridDim.x; item < nitems && item_nn(item) == 0; item += gridDim.x) {}
    return item;
  };
  int first = blockIdx.x;
  while (first < nitems && item_nn(first) == 0) first += gridDim.x;
  // per item: K extent (fwd radial points, bwd rows of the even parity), chunks, output rows, row tiles
  auto geom = [&](int nn, int& nkc_m, int& nrows, int& nmt_m) {
    const int kext = MODE == 0 ? a.nrh : (nn + 1) / 2;
    nkc_m = (kext + XS_KC - 1) / XS_KC;
    nrows = MODE == 0 ? (nn + 1) / 2 : a.nrh;
    nmt_m = (nrows + 127) / 128;
  };

  if (warp == 0) {
    // ---- producer
    if (lane == 0) {
      uint32_t c = 0, s = 0, ph = 0, cm = 0, sm = 0, pm = 0;   // table entries and magnitude tiles issued, ring slots and phases
      for (int item = first; item < nitems && ok; item = next_item(item)) {
        const int m = item_m(item);
        int nkc_m, nrows, nmt_m;
        geom(item_nn(item), nkc_m, nrows, nmt_m);
        for (int mt = 0; mt < nmt_m && ok; ++mt)
          for (int par = 0; par < 2 && ok; ++par) {
            const uint8_t* img_u = (const uint8_t*)a.img + (((size_t)m * a.nmt + mt) * 2 + par) * a.nkc * (size_t)(TILES * XS_ATILE);
            for (int kc = 0; kc < nkc_m; ++kc, ++c) {
              if (c >= AE && !xs_wait(&bar_ae[s], ph ^ 1u, ok)) break;
              mbar_expect_tx(&bar_af[s], AENT);
              const uint8_t* ent = img_u + (size_t)kc * (TILES * XS_ATILE);
              bulk_g2s(sA + s * AENT, ent, AENT, &bar_af[s]);
              if (++s == AE) { s = 0; ph ^= 1u; }
              if constexpr (MAG) {
                if (cm >= ME && !xs_wait(&bar_me[sm], pm ^ 1u, ok)) { ++c; break; }
                mbar_expect_tx(&bar_mf[sm], XS_ATILE);
                bulk_g2s(sM + sm * XS_ATILE, ent + AENT, XS_ATILE, &bar_mf[sm]);
                ++cm;
                if (++sm == ME) { sm = 0; pm ^= 1u; }
              }
            }
          }
      }
      // the copies issued complete on their own: wait (bounded) for the last of them, so that no copy
      // is in flight when the CTA's shared memory goes away (at once in a run without a timeout)
      for (uint32_t j = c > AE ? c - AE : 0; j < c; ++j) {
        bool ok2 = true;
        xs_wait(&bar_af[j % AE], (j / AE) & 1, ok2);
      }
      if constexpr (MAG) {
        for (uint32_t j = cm > ME ? cm - ME : 0; j < cm; ++j) {
          bool ok2 = true;
          xs_wait(&bar_mf[j % ME], (j / ME) & 1, ok2);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issue (the whole warp, one elected lane issuing)
    const uint32_t el = elect_lane();
    uint32_t sa = 0, pa = 0, sm = 0, pm = 0, sb = 0, pb = 0, u = 0, last = 0, plast = 0, mlast = 0, pmlast = 0;
    bool any = false, many = false;
    for (int item = first; item < nitems && ok; item = next_item(item)) {
      int nkc_m, nrows, nmt_m;
      geom(item_nn(item), nkc_m, nrows, nmt_m);
      for (int v = 0; v < 2 * nmt_m && ok; ++v, ++u) {   // units: row tile v / 2, parity v % 2
        // the unit's accumulators, once the epilogue has read what they held TB units before
        const uint32_t tb = u % TB;
        if (u >= (uint32_t)TB && !xs_wait_w(&bar_te[tb], ((u - TB) / TB) & 1, ok)) break;
        const uint32_t tacc = tmem + tb * (uint32_t)ACC;
        for (int kc = 0; kc < nkc_m; ++kc) {
          if (!xs_wait_w(&bar_bf[sb], pb, ok)) break;
          if (!xs_wait_w(&bar_af[sa], pa, ok)) break;
          tc_fence_after();
          const uint32_t a0 = smem_u32(sA) + sa * AENT, b0 = smem_u32(sB) + sb * BSTAGE;
          // table digit t times the field digits s = 0 .. NO-1-t in one MMA of N (NO - t) columns (two where that
          // passes the 256 columns of an MMA): the field digits lie side by side in shared memory and the orders
          // d = t + s side by side in tensor memory, so the product of digit s lands on order t + s
#pragma unroll
          for (int t = 0; t < NO; ++t) {
            const uint64_t ad = sdesc(a0 + t * XS_ATILE, XS_LBO, XS_SBO);
            constexpr int NB1 = 256 / N;   // digits of one MMA
            const int n1 = NO - t < NB1 ? NO - t : NB1;
            umma_bf16(tacc + (uint32_t)(t * N), ad, sdesc(b0, XS_LBO, XS_SBO), idesc_bf16(128, n1 * N),
                      (kc > 0 || t > 0) ? 1u : 0u, el);
            if (NO - t > NB1)
              umma_bf16(tacc + (uint32_t)((t + NB1) * N), ad, sdesc(b0 + NB1 * BT, XS_LBO, XS_SBO),
                        idesc_bf16(128, (NO - t - NB1) * N), (kc > 0 || t > 0) ? 1u : 0u, el);
          }
          umma_commit(&bar_ae[sa], el);
          last = sa; plast = pa; any = true;
          if (++sa == AE) { sa = 0; pa ^= 1u; }
          if constexpr (MAG) {   // the magnitudes' product, after the orders
            if (!xs_wait_w(&bar_mf[sm], pm, ok)) break;
            tc_fence_after();
            umma_bf16(tacc + (uint32_t)(NO * N), sdesc(smem_u32(sM) + sm * XS_ATILE, XS_LBO, XS_SBO), sdesc(b0 + NS * BT, XS_LBO, XS_SBO),
                      idesc_bf16(128, N), kc > 0 ? 1u : 0u, el);
            umma_commit(&bar_me[sm], el);
            mlast = sm; pmlast = pm; many = true;
            if (++sm == ME) { sm = 0; pm ^= 1u; }
          }
          umma_commit(&bar_be[sb], el);
          if (++sb == SB) { sb = 0; pb ^= 1u; }
        }
        if (ok) umma_commit(&bar_tf[tb], el);
      }
    }
    if (any) {   // the MMAs issued have finished (bounded) before tensor memory is freed
      bool ok2 = true;
      xs_wait_w(&bar_ae[last], plast, ok2);
    }
    if (MAG && many) {
      bool ok2 = true;
      xs_wait_w(&bar_me[mlast], pmlast, ok2);
    }
  } else if (warp < 2 + XS_NSW) {
    // ---- column scales from the largest magnitudes' high words of the re and im parts: |x| < 2^(exponent field - 1022),
    // and the forward folds may double.  Lane 0 of the first of the two warps also copies the field columns: with two
    // buffers the next item's as soon as this item's scales are out, so that they land while its digits are cut (issued
    // behind the item's table entries they came late: 20 500 cycles an item)
    int nraw = 0;   // copies issued
    auto copy_columns = [&](int item, int ii) {
      if (warp != 2 || lane != 0 || item >= nitems) return;
      const int rb = ii % RB, m = item_m(item), z0 = item_z0(item), kraw = MODE == 0 ? a.nr : item_nn(item);
      const double2* fin = xs_sel(a.in, item_f(item)) + (size_t)a.nrdim * (m + (size_t)a.npdim * z0);
      // once the digit threads are done with the item that had the buffer before
      if (ii >= RB && !xs_wait(&bar_re[rb], (ii / RB - 1) & 1, ok)) return;
      fence_async_smem();
      const int nzc = max(min(NZ, a.nzdim - z0), 0);
      mbar_expect_tx(&bar_rf[rb], (uint32_t)(nzc * kraw) * 16u);
      for (int zz = 0; zz < nzc; ++zz)
        bulk_g2s(raw0 + rb * rawsz + (size_t)2 * zz * a.rawk, fin + (size_t)a.nrdim * a.npdim * zz, (uint32_t)kraw * 16u,
                 &bar_rf[rb]);
      ++nraw;
    };
    int ii = 0;
    if (RB > 1) copy_columns(first, 0);
    for (int item = first; item < nitems && ok; item = next_item(item), ++ii) {
      const int slot = ii % XS_CXS, rb = ii % RB;
      if (ii >= XS_CXS && !xs_wait_w(&bar_ce[slot], (ii / XS_CXS - 1) & 1, ok)) break;
      if (RB > 1 && !xs_wait_w(&bar_rf[rb], (ii / RB) & 1, ok)) break;
      const int z0 = item_z0(item);
      const int kraw = MODE == 0 ? a.nr : item_nn(item);
      int* cxw = colexp + slot * N;
      // eight columns per warp, four lanes per column, their loads independent (a column after the other, reduced over the
      // whole warp, took 4 600 cycles an item alone and 12 000 beside the other warps)
      const int zz = (warp - 2) * 8 + (lane >> 2);
      unsigned mr = 0, mi = 0;
      if (zz < NZ && z0 + zz < a.nzdim) {
        // (re lo, re hi, im lo, im hi); with one column buffer read from global memory, ahead of the copy, so that the scan
        // does not stand between the copy and the digits
        auto scan = [&](const int4* col) {
#pragma unroll 8
          for (int i = lane & 3; i < kraw; i += 4) {
            const int4 v = col[i];
            mr = max(mr, (unsigned)v.y & 0x7FFFFFFFu);
            mi = max(mi, (unsigned)v.w & 0x7FFFFFFFu);
          }
        };
        if (RB > 1) scan((const int4*)(raw0 + rb * rawsz + (size_t)2 * zz * a.rawk));
        else scan((const int4*)(xs_sel(a.in, item_f(item)) + (size_t)a.nrdim * (item_m(item) + (size_t)a.npdim * (z0 + zz))));
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        mr = max(mr, __shfl_xor_sync(0xFFFFFFFFu, mr, o));
        mi = max(mi, __shfl_xor_sync(0xFFFFFFFFu, mi, o));
      }
      if ((lane & 3) == 0 && zz < NZ) {
        constexpr int fold = MODE == 0 ? 1 : 0;
        // an all-subnormal column counts as zero
        auto scale = [](unsigned h) {
          if (PLAIN && xs_nonfin(h)) return XS_NONFIN;
          return (h >> 20) ? (BAL ? xs_ebound_bal(h) : (int)(h >> 20) - 1022) + fold : -2000;
        };
        cxw[2 * zz] = scale(mr);
        cxw[2 * zz + 1] = scale(mi);
      }
      mbar_arrive(&bar_cx[slot]);
      if (RB > 1) copy_columns(next_item(item), ii + 1);
      else copy_columns(item, ii);
      ok = __all_sync(0xFFFFFFFFu, ok);
    }
    // no copy is in flight when the CTA's shared memory goes away (bounded; at once in a run without a timeout)
    for (int j = max(nraw - RB, 0); j < nraw; ++j) {
      bool ok2 = true;
      xs_wait(&bar_rf[j % RB], (j / RB) & 1, ok2);
    }
  } else if (warp < 2 + XS_NSW + XS_NDW) {
    // ---- field digits
    const int dw = (warp - 2 - XS_NSW) % GW, grp = (warp - 2 - XS_NSW) / GW;
    uint32_t c = 0, s = 0, ph = 0;
    int ii = 0;
    for (int item = first; item < nitems && ok; item = next_item(item), ++ii) {
      const int z0 = item_z0(item), nn = item_nn(item);
      int nkc_m, nrows, nmt_m;
      geom(nn, nkc_m, nrows, nmt_m);
      const int* cx = colexp + (ii % XS_CXS) * N;
      if (!xs_wait_w(&bar_cx[ii % XS_CXS], (ii / XS_CXS) & 1, ok)) break;
      const int rb = ii % RB;
      const double* raw = raw0 + rb * rawsz;
      if (!xs_wait_w(&bar_rf[rb], (ii / RB) & 1, ok)) break;
      // a warp writes (8 columns, 4 K pairs) blocks, each its 32 four-byte stores in 32 banks; the warp's blocks
      // unrolled, so that their independent chains interleave.  The columns' shift bases once per item.
      int base[NBLK / GW];
#pragma unroll
      for (int bi = 0; bi < NBLK / GW; ++bi) {
        const int n = ((dw + bi * GW) % (N / 8)) * 8 + (lane & 7);
        base[bi] = xs_fix_base(cx[n], nb, z0 + (n >> 1) < a.nzdim);
      }
      for (int v = 0; v < 2 * nmt_m && ok; ++v) {
        const int par = v & 1;
        for (int kc = 0; kc < nkc_m; ++kc, ++c) {
          if ((int)(c % NG) == grp) {   // the group's stage
            if (c >= SB && !xs_wait_w(&bar_be[s], ph ^ 1u, ok)) break;
            uint8_t* bst = sB + s * BSTAGE;
#pragma unroll
            for (int bi = 0; bi < NBLK / GW; ++bi) {
              const int blk = dw + bi * GW, ng = blk % (N / 8), kh = blk / (N / 8);
              const int n = ng * 8 + (lane & 7), kp = kh * 4 + (lane >> 3), zz = n >> 1;
              const double* col = raw + (size_t)2 * zz * a.rawk + (n & 1);
              const int off = xs_off(n, 2 * kp);
              unsigned long long x[2];
              long long xm[2];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int k = kc * XS_KC + 2 * kp + h;
                long long X = 0;
                if (MODE == 0) {
                  // B_par(i) = f(i) + (-1)^par f(nr-1-i), exact in the integers
                  if (k < a.nrh) {
                    const long long x2 = xs_fixs(col[2 * (a.nr - 1 - k)], base[bi]);
                    X = xs_fixs(col[2 * k], base[bi]) + (par ? -x2 : x2);
                  }
                } else {
                  // B_par(t) = c(2t + par)
                  const int j = 2 * k + par;
                  if (j < nn) X = xs_fixs(col[2 * j], base[bi]);
                }
                xm[h] = X;
                x[h] = (unsigned long long)X + (BAL ? xs_bias<NS, W>() : 0ull);
              }
              if constexpr (MAG) *(uint32_t*)(bst + NS * BT + off) = xs_mag2(xm[0], xm[1]);
              xs_static_for<NS>([&](auto tc) {
                constexpr int t = decltype(tc)::value;
                *(uint32_t*)(bst + t * BT + off) = xs_digit2<NS, W, BAL, t>(x[0], x[1]);
              });
            }
            fence_async_smem();
            mbar_arrive(&bar_bf[s]);
          }
          if (++s == SB) { s = 0; ph ^= 1u; }
        }
      }
      mbar_arrive(&bar_re[rb]);   // done with the item's field columns
    }
  } else {
    // ---- epilogue: warp e reads TMEM lanes 32 (e % 4) .. +31 (rows of the tile) and the column group e / 4; the
    // orders are combined exactly in 64-bit integers on the integer pipe, and the sums rounded once to FP64
    const int ew = warp - 2 - XS_NSW - XS_NDW, lq = warp & 3, cg = ew >> 2;
    const uint32_t lrow = (uint32_t)(lq * 32) << 16;
    uint32_t u = 0;
    int ii = 0;
    for (int item = first; item < nitems && ok; item = next_item(item), ++ii) {
      const int m = item_m(item), z0 = item_z0(item), nn = item_nn(item);
      double2* fout = xs_sel(a.out, item_f(item));
      int nkc_m, nrows, nmt_m;
      geom(nn, nkc_m, nrows, nmt_m);
      // the item's column scales: written before its digits were cut, and so before its accumulators were complete
      if (!xs_wait_w(&bar_cx[ii % XS_CXS], (ii / XS_CXS) & 1, ok)) break;
      const int* cx = colexp + (ii % XS_CXS) * N + cg * CW;
      for (int mt = 0; mt < nmt_m && ok; ++mt) {
        const int row = mt * 128 + lq * 32 + lane;
        const bool live = mt * 128 + lq * 32 < nrows;   // a warp of rows past the tile's rows reads nothing
        // the row exponents, loaded before the wait so that their latency hides behind it
        int EA[2] = {-2000, -2000};
        if (MODE == 0) {
          if (row < nrows) {
            EA[0] = a.aexp[(size_t)(m * 2) * a.nrp + row];
            EA[1] = a.aexp[(size_t)(m * 2 + 1) * a.nrp + row];
          }
        } else if (row < a.nrh) {
          EA[0] = a.aexp[(size_t)m * a.nrp + row];
        }
        // T 2^(row exp + column exp + eo + esh): the products carry 2^(-2 nb), the orders' unit is
        // 2^(2 w (NS-1) - w (NO-1)).  The mixed form's sums fit 64 bits with a fixed shift; the plain form's take the
        // shift esh that each sum itself allows (xs_order_shift): a column's small sums would lose bits to a neighbour's
        // large ones in a common shift
        constexpr int eo = (BAL ? xs_low<NS>() : ESH) + W * (2 * (NS - 1) - (NO - 1)) - 2 * nb;
        auto value = [&](long long t, int E, int ea, int e) {   // E: the column's scale
          if (PLAIN && E == XS_NONFIN) return __longlong_as_double(0x7FF8000000000000ll);
          return ea > -2000 && E > -2000 ? xs_i64_to_double(t, ea + E + e) : 0.0;
        };
        long long T[2][CW];            // order sums
        uint32_t esh[2] = {0, 0};      // balanced: the columns' shifts, four bits each (backward: esh[0] for both parities)
        uint32_t small[2] = {0, 0};    // magnitude sums below the least, a bit a column
#pragma unroll
        for (int par = 0; par < 2; ++par, ++u) {
          const uint32_t tb = u % TB;
          if (!xs_wait_w(&bar_tf[tb], (u / TB) & 1, ok)) break;
          tc_fence_after();
          const uint32_t tcol = tmem + tb * (uint32_t)ACC + lrow + (uint32_t)(cg * CW);
#pragma unroll
          for (int c = 0; c < CW; ++c) T[par][c] = 0;
          if (live) {
            // two orders per load batch
            xs_static_for<(NO + 1 - (BAL ? 2 : 0)) / 2>([&](auto dc) {
              constexpr int D = 2 * decltype(dc)::value + (BAL ? 2 : 0), D2 = D + 1 < NO ? D + 1 : D;
              uint32_t g[CW], h[CW];
              xs_tmem_ld<CW>(tcol + (uint32_t)(D * N), g);
              if constexpr (D2 != D) xs_tmem_ld<CW>(tcol + (uint32_t)(D2 * N), h);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < CW; ++c) {
                xs_acc_order<NO, W, BAL ? xs_low<NS>() : ESH, D>(T[par][c], g[c]);
                if constexpr (D2 != D) xs_acc_order<NO, W, BAL ? xs_low<NS>() : ESH, D2>(T[par][c], h[c]);
              }
            });
            if constexpr (BAL) {
              // C = G_0 2^w + G_1, then T = C 2^(cb - esh) + (L >> esh)
              uint32_t g[CW], h[CW];
              xs_tmem_ld<CW>(tcol, g);
              xs_tmem_ld<CW>(tcol + (uint32_t)N, h);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < CW; ++c) {
                const int C = xs_f2i(__uint_as_float(g[c])) * (1 << W) + xs_f2i(__uint_as_float(h[c]));
                int es = xs_order_shift<NS>(abs(C));
                if (MODE == 1 && par == 1) {   // the two parities are added: the same shift for both
                  const int e0 = (int)(esh[0] >> (4 * c)) & 15;
                  es = max(es, e0);
                  T[0][c] >>= es - e0;
                  esh[0] = (esh[0] & ~(15u << (4 * c))) | ((uint32_t)es << (4 * c));
                } else {
                  esh[par] |= (uint32_t)es << (4 * c);
                }
                T[par][c] = ((long long)C << (xs_cb<NS>() - es)) + (T[par][c] >> es);
              }
              if constexpr (MAG) {
                xs_tmem_ld<CW>(tcol + (uint32_t)(NO * N), g);
                tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < CW; ++c) small[par] |= __uint_as_float(g[c]) < a.least ? 1u << c : 0u;
              }
            }
          }
          tc_fence_before();
          mbar_arrive(&bar_te[tb]);
        }
        if (!ok) break;
        if (MAG && live) {
          // the outputs whose terms are all small beside their row's and column's largest entries, and those of columns with
        // non-finite samples, for k_xs_again
#pragma unroll
          for (int par = 0; par < (MODE == 0 ? 2 : 1); ++par) {
            const uint32_t sm = MODE == 0 ? small[par] : small[0] & small[1];
            const bool rok = MODE == 0 ? 2 * row + par < nn : row < a.nrh;
#pragma unroll
            for (int c = 0; c < CW; c += 2) {
              const int zo = z0 + ((cg * CW + c) >> 1);
              if (zo >= a.nzdim) continue;
              const bool few = (EA[par] > -2000 && (((sm >> c) & 1 && cx[c] > -2000) || ((sm >> (c + 1)) & 1 && cx[c + 1] > -2000))) ||
                               cx[c] == XS_NONFIN || cx[c + 1] == XS_NONFIN;
              const unsigned word = __ballot_sync(0xFFFFFFFFu, rok && few);
              if (lane == 0) a.again[xs_word(a, MODE, item_f(item), m, par, mt * 4 + lq, zo)] = word;
            }
          }
        }
        if (MODE == 0 ? row < nrows : row < a.nrh) {
          // the log term is added at m = 0 only: an integer test per item, so that the other items
          // issue no FP64 compares or (predicated) FP64 additions on GB300's narrow FP64 pipe
          const bool ln_here = MODE == 1 && a.add_ln && m == 0;
#pragma unroll
          for (int c = 0; c < CW; c += 2) {
            const int zo = z0 + ((cg * CW + c) >> 1);
            if (zo >= a.nzdim) continue;
            double2* o = fout + (size_t)a.nrdim * (m + (size_t)a.npdim * zo);
            if (MODE == 0) {
#pragma unroll
              for (int par = 0; par < 2; ++par) {
                if (2 * row + par >= nn) continue;
                double v[2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                  v[h] = value(T[par][c + h], cx[c + h], EA[par], eo + ((int)(esh[par] >> (4 * (c + h))) & 15));
                o[2 * row + par] = make_double2(v[0], v[1]);
              }
            } else {
              double v[4];   // f(i) re, im; f(nr-1-i) re, im
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                // f(i) = D_0 + D_1, f(nr-1-i) = D_0 - D_1: both parities share the scales
                const int e = eo + ((int)(esh[0] >> (4 * (c + h))) & 15);
                v[h] = value(T[0][c + h] + T[1][c + h], cx[c + h], EA[0], e);
                v[2 + h] = value(T[0][c + h] - T[1][c + h], cx[c + h], EA[0], e);
              }
              if (ln_here) {
                const double lnv = *xs_sel(a.lnp, item_f(item));
                v[0] += lnv * a.lnx[row];
                v[2] += lnv * a.lnx[a.nr - 1 - row];
              }
              o[row] = make_double2(v[0], v[1]);
              o[a.nr - 1 - row] = make_double2(v[2], v[3]);
            }
          }
        }
      }
      if (ok) mbar_arrive(&bar_ce[ii % XS_CXS]);   // this thread is done with the item's column scales
    }
  }
  if (!ok) atomicExch(a.status, 2);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TCOLS);
}

// ------------------------------------------------------------------------------------------------
// The marked outputs of the nine-digit form, summed in FP64 (as the FP64 kernels of radial.cu sum, term after term, backward).
// Few and scattered, or whole regions (the points near the axis where the functions of high m vanish), so each warp takes words
// from all over the grid, XS_AGAIN (a prime) apart.  Backward: a lane per row of the word, the table read along the rows.
// Forward: a marked row after the other, the lanes over the radial points.  Nothing marked: 4 us.
template <int MODE>
__global__ void __launch_bounds__(XS_AGAIN_T) k_xs_again(XsArgs a, const double* __restrict__ pf, const double* __restrict__ w, int ne,
                                                  size_t nwords) {
  const int lane = threadIdx.x & 31;
  const size_t nw = XS_AGAIN, wid = (size_t)blockIdx.x * (XS_AGAIN_T / 32) + (threadIdx.x >> 5);
  if (wid >= nw) return;
  int f, m, par, g, z;
  auto place = [&](size_t idx) {
    z = (int)(idx % a.nzdim); idx /= a.nzdim;
    g = (int)(idx % a.ngrp); idx /= a.ngrp;
    if (MODE == 0) { par = (int)(idx & 1); idx >>= 1; } else par = 0;
    m = (int)(idx % a.npc);
    f = (int)(idx / a.npc);
  };
  for (size_t base = wid; base < nwords; base += 32 * nw) {
    const size_t mine = base + nw * lane;
    unsigned word = 0;
    if (mine < nwords) {
      place(mine);
      const int nn = max(min(a.nrc, a.nrc - m), 0);
      if (m >= a.m0 && nn > 0 && g * 32 < (MODE == 0 ? (nn + 1) / 2 : a.nrh)) word = a.again[mine];   // (others are not written)
    }
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, word != 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const unsigned rows = __shfl_sync(0xFFFFFFFFu, word, src);
      place(base + nw * src);
      const int nn = max(min(a.nrc, a.nrc - m), 0);
      const size_t off = (size_t)a.nrdim * (m + (size_t)a.npdim * z);
      const double2* in = xs_sel(a.in, f) + off;
      double2* out = xs_sel(a.out, f) + off;
      const double* tab = pf + (size_t)a.nrh * ne * m;
      if (MODE == 1) {
        const int i = min(g * 32 + lane, a.nrh - 1);
        double er = 0.0, ei = 0.0, dr = 0.0, di = 0.0;
#pragma unroll 4
        for (int j = 0; j + 1 < nn; j += 2) {
          const double ve = __ldg(tab + i + (size_t)a.nrh * j), vo = __ldg(tab + i + (size_t)a.nrh * (j + 1));
          const double2 ce = __ldg(in + j), co = __ldg(in + j + 1);
          er = fma(ve, ce.x, er); ei = fma(ve, ce.y, ei);
          dr = fma(vo, co.x, dr); di = fma(vo, co.y, di);
        }
        if (nn & 1) {
          const double ve = __ldg(tab + i + (size_t)a.nrh * (nn - 1));
          const double2 ce = __ldg(in + nn - 1);
          er = fma(ve, ce.x, er); ei = fma(ve, ce.y, ei);
        }
        if ((rows >> lane) & 1) {
          out[i] = make_double2(er + dr, ei + di);
          out[a.nr - 1 - i] = make_double2(er - dr, ei - di);
        }
      } else {
        const double sgn = par ? -1.0 : 1.0;
        for (unsigned left = rows; left; left &= left - 1) {
          const int j = 2 * (g * 32 + __ffs(left) - 1) + par;
          if (j >= nn) break;   // (words that a contraction which ran out of time left unwritten)
          double re = 0.0, im = 0.0;
          for (int i = lane; i < a.nrh; i += 32) {
            const double v = __ldg(tab + i + (size_t)a.nrh * j), wi = __ldg(w + i);
            const double2 p = __ldg(in + i), q = __ldg(in + a.nr - 1 - i);
            re = fma(v, (p.x + sgn * q.x) * wi, re);
            im = fma(v, (p.y + sgn * q.y) * wi, im);
          }
#pragma unroll
          for (int o = 16; o; o >>= 1) {
            re += __shfl_xor_sync(0xFFFFFFFFu, re, o);
            im += __shfl_xor_sync(0xFFFFFFFFu, im, o);
          }
          if (lane == 0) out[j] = make_double2(re, im);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
struct XsImg {
  uint16_t* p = nullptr;
  int* aexp = nullptr;
  unsigned* again = nullptr;
  size_t bytes = 0, abytes = 0, gbytes = 0;
  int nrc = -1, npc = -1, ns = 0, nmt = 0, nkc = 0, nrp = 0;
};
static XsImg g_xs[2][2];   // [mode][plain/mixed]
static void xs_drop(XsImg& t) {
  if (t.p) dfree(t.p, t.bytes);
  if (t.aexp) dfree(t.aexp, t.abytes);
  if (t.again) dfree(t.again, t.gbytes);
  t = XsImg();
}

void xs_free() {
  for (auto& r : g_xs)
    for (auto& t : r) xs_drop(t);
}

// the digit configuration: FP64-grade (plain: 63 bits) or the mixed form's 42 bits, with the widest digits whose
// orders stay exact.  The mixed form
// needs 42 bits: its transform errors are deterministic, so a slowly changing flow meets the same
// error step after step and they add up along a run; with 35-bit slices the backward transforms alone
// left the vortex step's nonlinear term 9.6e-7 from the FP64 form after 1000 steps at 192 x 128 x 128,
// with 42 bits the whole mixed step stayed within 7e-7.  The plain form
// needs more than 53 bits: the rounding is relative to the column maximum, and the nonlinear term's
// curl cancellation magnifies what that loses on small entries (at 192 x 128 x 128 the vortex step's
// nonlinear term differed from the FP64 reference by 5e-10 with 49-bit and 2.4e-11 with 56-bit digits).
// On grids of up to 284 points it takes eight balanced digits up to 113 terms and ten unsigned ones of 6 bits, with a fixed
// 64-bit shift that cuts the sums at 2^-52 of max|A| max|B|, beyond; on larger grids nine balanced digits with magnitude sums.
// returns the digit count (its width is xs_w's), 0 where no configuration is exact
static int xs_rawk(int nrc) { return std::max(G.nr, nrc) | 1; }   // odd: the staged columns start in different banks
static int xs_cfg(int kmax, int nrc, bool plain) {
  const double lim = 16777216.0;
  if (plain) {
    if (xs_rawk(nrc) <= 285) return kmax <= 113 ? 8 : 10;   // 8 128 128 K <= 2^24 up to 128
    if (xs_order_bound(9, 7, 1, kmax) <= XS_EXACT) return 9;   // up to 372
  } else {
    // (larger grids' sums are FP64 in this form too: 740 points with seven digits, 892 with six)
    if (6.0 * kmax * 128 * 128 < lim) return xs_rawk(nrc) <= 893 ? 6 : 0;
    if (7.0 * kmax * 64 * 64 < lim) return xs_rawk(nrc) <= 741 ? 7 : 0;
  }
  return 0;
}

static size_t xs_smem(int ns, int nz, int rawk, int aent, int bst, int nraw, int sent) {
  const int n = 2 * nz;
  return 1024 + aent * (size_t)(ns * XS_ATILE) + sent * (size_t)XS_ATILE + bst * (size_t)((ns + (sent > 0)) * n * XS_KC * 2) +
         nraw * (size_t)2 * nz * rawk * sizeof(double) + XS_CXS * n * sizeof(int) + 512;
}
constexpr size_t XS_SMEM_MAX = 227 * 1024;
// The work items and rings of a digit count: 16 complex z columns per item where shared memory holds one buffer of field
// columns beside two digit stages and two table entries (up to 512 points in the plain form), else 8: half the columns
// per table entry means twice the table traffic, through L2 and shared memory, for the same result (512 points, seven
// digits: 19.1 ms for two steps' backward transforms with 8 columns, 13.8 ms with 16).  Two column buffers where they fit
// (up to 256 points), so that an item's columns land and are scanned while the one before is cut; then digit stages, at
// most four (six measured the same), and table entries in what is left.
struct XsPlan { int nz, aent, bst, nraw, sent; };
// `few`: no more items than half the SMs; halved, they take less time each (24 x 20 x 12, plain: 17.1 and 21.1 us forward and
// backward with 16 columns, 14.9 and 17.2 with 8).
static bool xs_plan(int ns, int rawk, XsPlan& p, bool few = false) {
  for (int nz = G.nzdim > 8 && !few ? 16 : 8; nz >= 8; nz /= 2)
    for (int nraw = 2; nraw >= 1; --nraw)
      for (int sb = XS_SBMAX; sb >= 2; --sb)
        for (int me = ns == 9 ? XS_MEMAX : 0; me >= (ns == 9 ? 1 : 0); --me)
          for (int ae = XS_AEMAX; ae >= 2; --ae)
            if (xs_smem(ns, nz, rawk, ae, sb, nraw, me) <= XS_SMEM_MAX) { p = {nz, ae, sb, nraw, me}; return true; }
  return false;
}
// whether the exact-slice contraction covers this kit: the orders stay exact and the rings fit
bool xs_supported(int mode, int nrc, bool plain) {
  const int ns = xs_cfg(mode == 0 ? G.nrh : (nrc + 1) / 2, nrc, plain);
  XsPlan p;
  return ns > 0 && xs_plan(ns, xs_rawk(nrc), p);
}

static size_t xs_words(int mode, int nf, int npc, int ngrp) { return (size_t)nf * npc * (mode == 0 ? 2 : 1) * ngrp * G.nzdim; }
template <int MODE, int NS, int NZ>
static int xs_launch(const XsArgs& args, int nitems) {
  const size_t sm = xs_smem(NS, NZ, args.rawk, args.aent, args.bst, args.nraw, args.sent);
  if (sm > XS_SMEM_MAX) return set_error(MLG_ESIZE, "radial contraction: shared-memory stage too large");
  auto kern = k_xs_rtrans<MODE, NS, NZ>;
  MLG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  kern<<<std::min(nitems, 152), XS_THREADS, sm, G.stream>>>(args);
  MLG_LAUNCH();
  if constexpr (xs_mag<NS>() != 0) {
    k_xs_again<MODE><<<cdiv(XS_AGAIN, XS_AGAIN_T / 32), XS_AGAIN_T, 0, G.stream>>>(args, G.pf, G.w, G.ne,
                                                                                 xs_words(MODE, args.nf, args.npc, args.ngrp));
    MLG_LAUNCH();
  }
  return 0;
}

// the table images of a chop: made on its first transform; MLG_EALLOC where there is no room for them
int xs_prepare(int mode, int nrc, int npc, bool plain) {
  const int nrows = mode == 0 ? (nrc + 1) / 2 : G.nrh, kmax = mode == 0 ? G.nrh : (nrc + 1) / 2, ns = xs_cfg(kmax, nrc, plain);
  const int nmt = cdiv(nrows, 128), nkc = cdiv(kmax, XS_KC), nrp = nmt * 128;
  XsImg& im = g_xs[mode][plain ? 0 : 1];
  if (im.nrc == nrc && im.npc == npc && im.p && im.ns == ns) return 0;
  xs_drop(im);
  im.bytes = (size_t)npc * nmt * nkc * 2 * (ns + (ns == 9)) * XS_ATILE;
  im.abytes = (size_t)npc * (mode == 0 ? 2 : 1) * nrp * sizeof(int);
  im.gbytes = ns == 9 ? xs_words(mode, XS_NF, npc, cdiv(nrows, 32)) * sizeof(unsigned) : 0;
  if (int rc = dmalloc_all({{(void**)&im.p, im.bytes}, {(void**)&im.aexp, im.abytes}, {(void**)&im.again, im.gbytes}})) return rc;
  k_xs_aexp<<<dim3(cdiv(nrp, 128), npc), 128, 0, G.stream>>>(G.pf, G.w, im.aexp, mode, G.nrh, G.ne, nrc, nrp, kmax,
                                                                 ns == 8 || ns == 9 ? 1 : 0);
  MLG_LAUNCH();
  const int nblk_t = npc * nmt * nkc;
  switch (ns) {
    case 6: k_xs_table<6><<<nblk_t, 256, 0, G.stream>>>(G.pf, G.w, im.aexp, im.p, mode, G.nrh, G.ne, nrc, nmt, nkc, nrp); break;
    case 7: k_xs_table<7><<<nblk_t, 256, 0, G.stream>>>(G.pf, G.w, im.aexp, im.p, mode, G.nrh, G.ne, nrc, nmt, nkc, nrp); break;
    case 8: k_xs_table<8><<<nblk_t, 256, 0, G.stream>>>(G.pf, G.w, im.aexp, im.p, mode, G.nrh, G.ne, nrc, nmt, nkc, nrp); break;
    case 10: k_xs_table<10><<<nblk_t, 256, 0, G.stream>>>(G.pf, G.w, im.aexp, im.p, mode, G.nrh, G.ne, nrc, nmt, nkc, nrp); break;
    default: k_xs_table<9><<<nblk_t, 256, 0, G.stream>>>(G.pf, G.w, im.aexp, im.p, mode, G.nrh, G.ne, nrc, nmt, nkc, nrp); break;
  }
  MLG_LAUNCH();
  im.nrc = nrc; im.npc = npc; im.ns = ns; im.nmt = nmt; im.nkc = nkc; im.nrp = nrp;
  return 0;
}

// mode 0 forward, 1 backward, for m0 <= m < npc; out's rows that it writes are overwritten, the rest left
int xs_rtrans_multi(int mode, const cd* const* in, cd* const* out, int nf, int nrc, int npc, int m0,
                    const double* const* lnp, bool add_ln, bool plain) {
  if (npc <= m0 || nf < 1) return 0;
  if (nf > XS_NF) return set_error(MLG_EPARAM, "radial contraction: at most three fields per launch");
  const int nrows = mode == 0 ? (nrc + 1) / 2 : G.nrh;
  const int kmax = mode == 0 ? G.nrh : (nrc + 1) / 2;
  const int ns = xs_cfg(kmax, nrc, plain);
  XsPlan plan;
  const bool few = (long long)(npc - m0) * cdiv(G.nzdim, 16) * nf <= 76;
  if (!ns || !xs_plan(ns, xs_rawk(nrc), plan, few)) return set_error(MLG_ESIZE, "radial contraction: too many radial points for exact slices");
  const int nmt = cdiv(nrows, 128), nkc = cdiv(kmax, XS_KC), nrp = nmt * 128;
  MLG_TRY(xs_prepare(mode, nrc, npc, plain));
  const XsImg& im = g_xs[mode][plain ? 0 : 1];
  XsArgs args;
  for (int f = 0; f < XS_NF; ++f) {
    const int g = f < nf ? f : 0;
    args.in[f] = in[g]; args.out[f] = out[g]; args.lnp[f] = lnp ? lnp[g] : nullptr;
  }
  args.nf = nf;
  args.img = im.p; args.aexp = im.aexp; args.lnx = G.lnx;
  args.status = (int*)(G.dscal + DS_FLAG + 1) + 1;
  args.add_ln = add_ln ? 1 : 0; args.nr = G.nr; args.nrh = G.nrh; args.nrdim = G.nrdim; args.npdim = G.npdim;
  args.nzdim = G.nzdim; args.nrc = nrc; args.m0 = m0; args.npc = npc; args.nmt = nmt; args.nkc = nkc; args.nrp = nrp;
  args.rawk = xs_rawk(nrc);
  args.aent = plan.aent;
  args.bst = plan.bst;
  args.nraw = plan.nraw;
  args.sent = plan.sent;
  args.again = im.again; args.ngrp = cdiv(nrows, 32); args.least = xs_least_sum(kmax);
  const bool nz16 = plan.nz == 16;
  const int nitems = (npc - m0) * cdiv(G.nzdim, plan.nz) * nf;
#define XS_CASE(NSV)                                                                                   \
  case NSV:                                                                                            \
    if (mode == 0) return nz16 ? xs_launch<0, NSV, 16>(args, nitems) : xs_launch<0, NSV, 8>(args, nitems); \
    return nz16 ? xs_launch<1, NSV, 16>(args, nitems) : xs_launch<1, NSV, 8>(args, nitems);
  switch (ns) {
    XS_CASE(6)
    XS_CASE(7)
    XS_CASE(8)
    XS_CASE(9)
    XS_CASE(10)
  }
#undef XS_CASE
  return set_error(MLG_EPARAM, "radial contraction: digit configuration");
}

int xs_rtrans(int mode, const cd* in, cd* out, int nrc, int npc, int m0, const double* lnp, bool add_ln, bool plain) {
  return xs_rtrans_multi(mode, &in, &out, 1, nrc, npc, m0, &lnp, add_ln, plain);
}

// The bounded-wait path of the tensor-core kernels on its own: one thread waits on an mbarrier of
// arrival count 1.  arrive = 0: nothing arrives, so the wait runs out after `limit` clocks and the
// kernel sets the timeout word exactly as k_xs_rtrans does; arrive = 1: the thread arrives first and
// the wait ends at once.  Nothing is in flight and no tensor memory is held when it returns.
__global__ void k_wait_selftest(int* __restrict__ status, long long limit, int arrive) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  fence_mbar_init();
  if (arrive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&bar)) : "memory");
  if (!mbar_wait_limit(&bar, 0, limit)) atomicExch(status, 2);
}

int wait_selftest(long long limit, int arrive) {
  if (limit < 0 || limit > 2000000000LL) return set_error(MLG_EPARAM, "wait self-test: limit must be 0 .. 2e9 clocks");
  k_wait_selftest<<<1, 32, 0, G.stream>>>((int*)(G.dscal + DS_FLAG + 1) + 1, limit, arrive ? 1 : 0);
  MLG_LAUNCH();
  return 0;
}

}  // namespace mlg
