// xs_vec2tp.cu — the projection contraction of vector_projection (mlegs_scalar_ops.f90:1402-1438, with
// the eomul / oemul folds :2067-2145) as exact-slice products on the 5th-generation tensor cores.
//
// For each m and row parity par, rows j = 2t + par, radial points i < nr/2, z columns n:
//   psi = (m V).(-i F_s(ur)) + D.(-F_o(up))
//   chi = k X - Y,   X = D.(i F_o(ur)) + (m V).F_s(up),   Y = T.F_s(uz)
// F_s / F_o fold u(i) with u(nr-1-i) by the row's own / the other parity's sign.
//
// All three sums run in the exact-slice scheme of xs_radial.cu.  psi and X each add two products in one
// set of digit-order accumulators, so the two products share their scales: one row scale per j over
// m V and D (kit init), one column scale per real column n over the two field components that land in
// it (Im ur with Re up for the real part of the output, Re ur with Im up for the imaginary part;
// the folds may double), and the digits of the folds are exact integer sums of the rounded samples.
// Y has its own row scale (T) and column scale (uz).  The orders of each sum are combined exactly in
// 64-bit integers and rounded once to FP64, on the integer pipe; chi = k X - Y is one FP64 fused
// multiply-add.  The row parity of a work item fixes the folds, so each item is one (m, parity,
// 128-row tile, NZ complex z columns).
//
// Digits: NS for psi and X, NT for Y, of w bits.
// Mixed form: NS = 5 (35 bits) and NT = 7 (49 bits; 6 and 8 of 6 bits beyond about 200 radial points); w and the digit
// counts keep every order's accumulator exact: (pairs of the order) x (nr/2) x 2^(2w) < 2^24, where psi's and X's orders
// hold two products per digit pair.  Y needs the extra digits: at k = 0 chi is -Y alone, and the inverse
// Laplacian that ends the projection magnifies its error in the weak low modes; with 42-bit Y the
// (m = 1, k = 0) column left the step's nonlinear term chi 9e-6 from FP64 at 192 x 128 x 128, with
// 49 bits 2e-7.
// Plain form: nine balanced digits of 7 bits (63 bits) for all three, up to 744 radial points.  An order of psi or X holds two
// products per digit pair and is exact up to 186 terms (xs_order_bound); beyond 372 radial points the accumulators are drained
// every 176 and the parts added in 64-bit integers.  The order sums are shifted by what they need (xs_radial.cu): cut at a fixed
// 2^-52, as 54-bit slices once were, chi = k X - Y is left 7e-9 from FP64.  Beside the digits the magnitudes are contracted
// (xs_least_sum): psi and chi of outputs whose terms are all small beside their row's and column's largest entries, and of
// columns with non-finite samples, are summed again in FP64 (k_xv_again).
//
// Engine: a persistent grid of one CTA per SM over work items (m, 8 complex z columns, 128-row tile, parity).
//   warp 0        the table entries (the digits, and in the plain form the magnitudes, of m V, D or T for a chunk of 16
//                 radial points), by bulk copy
//   warp 1        MMA issue: a table digit t meets every field digit s <= n-1-t of its operands in
//                 one MMA (M = 128, K = 16; the field digits side by side in shared memory, the orders side by
//                 side in tensor memory, psi's and X's alternating), two where that passes 256 columns
//   warps 2, 3    the items' column scales, up to four items ahead
//   warps 4..15   field digits, in two groups of six warps that take the chunks in turn (ur, up and uz at i and nr-1-i,
//                 fetched in FP64 a chunk ahead; one staging item per thread: field, z column, K pair)
//   warps 16..23  epilogue
// Every hand-off is an mbarrier and every wait is bounded.  psi's and X's accumulators are released before Y's are
// read.
// What bounds it (clock64 traces, 192 points): plain, the MMAs, 1 200 cycles an entry, three entries a chunk, and 4 000
// cycles more a unit while the epilogue drains tensor memory (its three sets of order sums fill it, so that units do
// not overlap there).  Mixed: the MMAs (600 an entry) and the digits (2 300 a chunk for each of two groups) alike.
// Per launch at 192 x 128 x 128 (ncu): plain 263 us and 36 for k_xv_again (221 without the magnitudes; FP64 DFMA 2 602), mixed
// 176 us (events: 199; 234 while one lane issued the MMAs from a branch; 264 when one CTA of 256 threads walked scales, chunks and
// epilogue in turn); 512 x 512 x 256 mixed 5.4 ms (6.7; 7.3).
#include "common.cuh"
#include "tc_common.cuh"
#include "xs_common.cuh"
#include <cstdint>

namespace mlg {

constexpr int XV_KC = 16;
constexpr int XV_SBO = XV_KC * 16;
constexpr int XV_LBO = 128;
__host__ __device__ constexpr int xv_off(int row, int k) {
  return (row >> 3) * XV_SBO + (k >> 3) * XV_LBO + (row & 7) * 16 + (k & 7) * 2;
}
constexpr int XV_ATILE = 128 * XV_KC * 2;    // 4 KiB

__device__ __forceinline__ bool xs_wait(uint64_t* bar, uint32_t phase, bool& ok) {
  if (!ok) return false;
  ok = mbar_wait(bar, phase);
  return ok;
}
// the same for a whole warp, whose lanes share the outcome
__device__ __forceinline__ bool xs_wait_w(uint64_t* bar, uint32_t phase, bool& ok) {
  xs_wait(bar, phase, ok);
  ok = __all_sync(0xFFFFFFFFu, ok);
  return ok;
}

// ------------------------------------------------------------------------------------------------
// kit-time: row scales rexp[(m * 2 + par) * ntr + t] over (m V, D) and texp over T (-2000: zero row)
__global__ void k_xv_rexp(const double* __restrict__ tV, const double* __restrict__ tD, const double* __restrict__ tT,
                          int* __restrict__ rexp, int* __restrict__ texp, int nrh, int ne, int nrc, int ntr, int bal) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int mp = blockIdx.y, m = mp >> 1, par = mp & 1;
  if (t >= ntr) return;
  const int j = 2 * t + par, nn = max(min(nrc, nrc - m), 0);
  unsigned long long mv = 0, mt = 0;
  if (j < nn)
    for (int i = 0; i < nrh; ++i) {
      const size_t o = i + (size_t)nrh * (j + (size_t)ne * m);
      unsigned long long a = (unsigned long long)__double_as_longlong((double)m * tV[o]) & 0x7FFFFFFFFFFFFFFFull;
      unsigned long long b = (unsigned long long)__double_as_longlong(tD[o]) & 0x7FFFFFFFFFFFFFFFull;
      unsigned long long c = (unsigned long long)__double_as_longlong(tT[o]) & 0x7FFFFFFFFFFFFFFFull;
      mv = a > mv ? a : mv;
      mv = b > mv ? b : mv;
      mt = c > mt ? c : mt;
    }
  auto bound = [&](unsigned long long v) { return !v ? -2000 : bal ? xs_ebound_bal((unsigned)(v >> 32)) : xs_ebound(v); };
  rexp[(size_t)mp * ntr + t] = bound(mv);
  texp[(size_t)mp * ntr + t] = bound(mt);
}

// digit configurations: the plain form's nine balanced digits, else two's complement
template <int NS> __host__ __device__ constexpr bool xv_bal() { return NS == 9; }
template <int NS, int W> __host__ __device__ constexpr int xv_nb(int n) { return xv_bal<NS>() ? 63 : W * n; }
// the plain form's digits carry a magnitude tile beside them (xs_least_sum)
template <int NS> __host__ __device__ constexpr int xv_mag() { return xv_bal<NS>() ? 1 : 0; }
// tiles of a chunk's three table entries
template <int NS, int NT> __host__ __device__ constexpr int xv_tiles() { return 2 * NS + NT + 3 * xv_mag<NS>(); }

// tiles per (m, par, row tile mt, chunk kc): [m V digits NS | D digits NS | T digits NT], each with its magnitude tile behind it
template <int NS, int NT, int W>
__global__ void k_xv_table(const double* __restrict__ tV, const double* __restrict__ tD, const double* __restrict__ tT,
                           const int* __restrict__ rexp, const int* __restrict__ texp, uint16_t* __restrict__ img,
                           int nrh, int ne, int nrc, int nmt, int nkc, int ntr) {
  constexpr bool BAL = xv_bal<NS>();
  const size_t blk = blockIdx.x;   // ((m * 2 + par) * nmt + mt) * nkc + kc
  const int kc = (int)(blk % nkc), mt = (int)((blk / nkc) % nmt), mp = (int)(blk / ((size_t)nkc * nmt));
  const int m = mp >> 1, par = mp & 1;
  const int nn = max(min(nrc, nrc - m), 0);
  constexpr int MG = xv_mag<NS>();
  uint8_t* base = (uint8_t*)img + blk * (size_t)(xv_tiles<NS, NT>() * XV_ATILE);
  for (int idx = threadIdx.x; idx < 128 * XV_KC; idx += blockDim.x) {
    const int k = idx % XV_KC, r = idx / XV_KC;
    const int t = mt * 128 + r, j = 2 * t + par, i = kc * XV_KC + k;
    double v = 0.0, d = 0.0, tt = 0.0;
    int er = -2000, et = -2000;
    if (t < ntr && j < nn && i < nrh) {
      const size_t o = i + (size_t)nrh * (j + (size_t)ne * m);
      v = (double)m * tV[o]; d = tD[o]; tt = tT[o];
      er = rexp[(size_t)mp * ntr + t]; et = texp[(size_t)mp * ntr + t];
    }
    const int off = xv_off(r, k);
    constexpr unsigned long long bs = BAL ? xs_bias<NS, W>() : 0ull, bt = BAL ? xs_bias<NT, W>() : 0ull;
    const long long iv = xs_fix(v, er, xv_nb<NS, W>(NS)), id = xs_fix(d, er, xv_nb<NS, W>(NS)), it = xs_fix(tt, et, xv_nb<NS, W>(NT));
    const unsigned long long xv = (unsigned long long)iv + bs, xd = (unsigned long long)id + bs, xt = (unsigned long long)it + bt;
    xs_static_for<NS>([&](auto sc) {
      constexpr int q = decltype(sc)::value;
      *(uint16_t*)(base + q * XV_ATILE + off) = (uint16_t)xs_digit2<NS, W, BAL, q>(xv, xv);
      *(uint16_t*)(base + (NS + MG + q) * XV_ATILE + off) = (uint16_t)xs_digit2<NS, W, BAL, q>(xd, xd);
    });
    xs_static_for<NT>([&](auto sc) {
      constexpr int q = decltype(sc)::value;
      *(uint16_t*)(base + (2 * (NS + MG) + q) * XV_ATILE + off) = (uint16_t)xs_digit2<NT, W, BAL, q>(xt, xt);
    });
    if (MG) {
      *(uint16_t*)(base + NS * XV_ATILE + off) = (uint16_t)xs_mag2(iv, iv);
      *(uint16_t*)(base + (2 * NS + 1) * XV_ATILE + off) = (uint16_t)xs_mag2(id, id);
      *(uint16_t*)(base + (2 * (NS + 1) + NT) * XV_ATILE + off) = (uint16_t)xs_mag2(it, it);
    }
  }
}

// ------------------------------------------------------------------------------------------------
struct XvArgs {
  const double2 *ur, *up, *uz;
  double2 *psi, *chi;
  const uint16_t* img;
  const int *rexp, *texp;
  const double* ak;
  int* status;
  int nr, nrh, nrdim, npdim, nzdim, nrc, nzc, nzcu, nmt, nkc, ntr, m0, npc;
  int aent;           // table entries of the ring
  unsigned* again;    // plain form: the outputs to be summed again, a word of 32 rows (xv_word)
  int again_m, again_zl, again_zu;   // of them those of m < again_m and of z + 1 <= again_zl or >= again_zu
  int ngrp;
  float least;        // xs_least_sum
  int esh_s, esh_t;   // two's complement digits: right shifts that keep the 64-bit order sums of psi / X and of Y below 2^62
};

// the word of the rows t = 32 g .. 32 g + 31 of parity par of column (m, z)
__device__ __forceinline__ size_t xv_word(const XvArgs& a, int m, int par, int g, int z) {
  return (((size_t)m * 2 + par) * a.ngrp + g) * a.nzdim + z;
}

constexpr int XV_PART = 11;   // chunks between drains where one set of accumulators does not take all radial points
static_assert(xs_order_bound(9, 7, 2, XV_PART * XV_KC) <= XS_EXACT, "the orders of a part stay exact");
constexpr int XV_NZ = 8, XV_N = 2 * XV_NZ;   // complex z columns per item, real columns
constexpr int XV_NSW = 2, XV_GW = 6, XV_NEW = 8;   // scale warps, warps of a digit group (two groups), epilogue warps
constexpr int XV_THREADS = (2 + XV_NSW + 2 * XV_GW + XV_NEW) * 32;
constexpr int XV_CXS = 4, XV_AEMAX = 6, XV_SB = 2;   // column-scale slots, table entries (at most), digit stages
constexpr int XV_BTILE = XV_N * XV_KC * 2;
static_assert(3 * XV_NZ * 8 == XV_GW * 32, "one staging item per digit thread");
template <int NS, int NT> __host__ __device__ constexpr int xv_aent_bytes() { return ((NS > NT ? NS : NT) + xv_mag<NS>()) * XV_ATILE; }
template <int NS, int NT> __host__ __device__ constexpr int xv_bstage_bytes() { return (4 * NS + NT + 5 * xv_mag<NS>()) * XV_BTILE; }

// order sums of eight columns, two's complement digits: T[c] = sum_d G_d 2^(w (n-1-d) - esh), order d at tcol + d step
template <int NO, int W> __device__ __forceinline__ void xv_sums(uint32_t tcol, uint32_t step, int esh, long long* T) {
#pragma unroll
  for (int c = 0; c < 8; ++c) T[c] = 0;
  xs_static_for<(NO + 1) / 2>([&](auto dc) {
    constexpr int D = 2 * decltype(dc)::value, D2 = D + 1 < NO ? D + 1 : D;
    uint32_t g[8], h[8];
    tmem_ld8_nw(tcol + D * step, g);
    if constexpr (D2 != D) tmem_ld8_nw(tcol + D2 * step, h);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      T[c] += xs_shl((long long)xs_f2i(__uint_as_float(g[c])), W * (NO - 1 - D) - esh);
      if constexpr (D2 != D) T[c] += xs_shl((long long)xs_f2i(__uint_as_float(h[c])), W * (NO - 1 - D2) - esh);
    }
  });
}
// Balanced digits (xs_radial.cu): L = sum_{d>=2} G_d 2^(w (NO-1-d) - 3) and C = G_0 2^w + G_1; with K <= 372 and two products
// |G_2| <= 2 K (2^(2w-2) + 2 2^(w+6)), so |L| < 2^62.9, |L| 2^-cb < 2^17 and |C| < 2^31.  mag: the magnitude sums' columns.
constexpr int XV_LOW = 3;
template <int NO, int W> constexpr int xv_cb() { return W * (NO - 2) - XV_LOW; }
struct XvSum { long long L[8]; int C[8]; float S[8]; };
template <int NO, int W> __device__ __forceinline__ void xv_drain(uint32_t tcol, uint32_t step, uint32_t mag, XvSum& q, bool first) {
  if (first) {
#pragma unroll
    for (int c = 0; c < 8; ++c) { q.L[c] = 0; q.C[c] = 0; q.S[c] = 0.f; }
  }
  auto acc = [&](auto dc, uint32_t g, int c) {
    constexpr int SH = W * (NO - 1 - decltype(dc)::value) - XV_LOW;
    const int v = xs_f2i(__uint_as_float(g));
    if constexpr (SH > 30) q.L[c] += (long long)v << SH;
    else if constexpr (SH >= 0) q.L[c] += (long long)v * (long long)(1 << SH);
    else q.L[c] += (long long)(v >> -SH);
  };
  xs_static_for<(NO - 1) / 2>([&](auto dc) {
    constexpr int D = 2 * decltype(dc)::value + 2, D2 = D + 1 < NO ? D + 1 : D;
    uint32_t g[8], h[8];
    tmem_ld8_nw(tcol + D * step, g);
    if constexpr (D2 != D) tmem_ld8_nw(tcol + D2 * step, h);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      acc(std::integral_constant<int, D>(), g[c], c);
      if constexpr (D2 != D) acc(std::integral_constant<int, D2>(), h[c], c);
    }
  });
  uint32_t g[8], h[8];
  tmem_ld8_nw(tcol, g);
  tmem_ld8_nw(tcol + step, h);
  tmem_wait_ld();
#pragma unroll
  for (int c = 0; c < 8; ++c) q.C[c] += xs_f2i(__uint_as_float(g[c])) * (1 << W) + xs_f2i(__uint_as_float(h[c]));
  tmem_ld8_nw(mag, g);
  tmem_wait_ld();
#pragma unroll
  for (int c = 0; c < 8; ++c) q.S[c] += __uint_as_float(g[c]);
}
// column c's sum in FP64, times 2^e: T = C 2^(cb - es) + (L >> es) below 2^62, es the shift that this sum needs
template <int NO, int W> __device__ __forceinline__ double xv_value(const XvSum& q, int c, int e) {
  const int es = max(32 - __clz(abs(q.C[c]) + 131072) + xv_cb<NO, W>() - 62, 0);
  return xs_i64_to_double(((long long)q.C[c] << (xv_cb<NO, W>() - es)) + (q.L[c] >> es), e + es + XV_LOW);
}

// PARTS: more radial points than one set of accumulators takes exactly (xv_exact), drained every XV_PART chunks
template <int NS, int NT, int W, bool PARTS>
__global__ void __launch_bounds__(XV_THREADS, 1) k_xv_contract(XvArgs a) {
  constexpr bool BAL = xv_bal<NS>();
  constexpr int NZ = XV_NZ, N = XV_N;
  constexpr int nbs = xv_nb<NS, W>(NS), nbt = xv_nb<NS, W>(NT);
  constexpr int MG = xv_mag<NS>();
  constexpr int AENT = xv_aent_bytes<NS, NT>(), BSTAGE = xv_bstage_bytes<NS, NT>();
  constexpr int COLS = xv_tiles<NS, NT>() * N;
  constexpr int TCOLS = COLS <= 256 ? 256 : 512;
  constexpr uint32_t TY = 2 * NS * N;             // Y's accumulators, after psi's and X's
  constexpr uint32_t TM = TY + NT * N;            // the magnitude sums of psi, X and Y
  static_assert(COLS <= 512, "accumulators exceed tensor memory");
  extern __shared__ __align__(1024) uint8_t xv_smem_raw[];
  uint8_t* sbase = (uint8_t*)(((uintptr_t)xv_smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t AE = (uint32_t)a.aent;
  uint8_t* sA = sbase;                            // [AE][AENT]
  uint8_t* sB = sA + AE * AENT;                   // [XV_SB][BSTAGE]
  int* cxs = (int*)(sB + XV_SB * BSTAGE);         // [XV_CXS][2 N]: by item, ur/up columns then uz columns
  uint64_t* bars = (uint64_t*)(cxs + XV_CXS * 2 * N);
  uint64_t* bar_af = bars;                        // [AE] table entry landed
  uint64_t* bar_ae = bar_af + XV_AEMAX;           // [AE] table entry consumed (MMA commit)
  uint64_t* bar_bf = bar_ae + XV_AEMAX;           // [XV_SB] digit stage written (the group's digit threads)
  uint64_t* bar_be = bar_bf + XV_SB;              // [XV_SB] digit stage consumed (MMA commit)
  uint64_t* bar_tf = bar_be + XV_SB;              // accumulators complete (MMA commit)
  uint64_t* bar_te = bar_tf + 1;                  // [2] psi's and X's, Y's accumulators read (epilogue threads)
  uint64_t* bar_cx = bar_te + 2;                  // [XV_CXS] column scales written (scale threads)
  uint64_t* bar_ce = bar_cx + XV_CXS;             // [XV_CXS] column scales read (epilogue threads: the item's last readers)
  uint32_t* tslot = (uint32_t*)(bar_ce + XV_CXS);

  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;   // warp: uniform
  if (tid == 0) {
    for (int i = 0; i < XV_AEMAX; ++i) {
      mbar_init(bar_af + i, 1);
      mbar_init(bar_ae + i, 1);
    }
    for (int i = 0; i < XV_SB; ++i) {
      mbar_init(bar_bf + i, XV_GW * 32);
      mbar_init(bar_be + i, 1);
    }
    mbar_init(bar_tf, 1);
    mbar_init(bar_te, XV_NEW * 32);
    mbar_init(bar_te + 1, XV_NEW * 32);
    for (int i = 0; i < XV_CXS; ++i) {
      mbar_init(bar_cx + i, XV_NSW * 32);
      mbar_init(bar_ce + i, XV_NEW * 32);
    }
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

  // the CTA's items ((m, z tile), row tile, parity), those without rows skipped; every role walks the same sequence
  const int nzt = (a.nzdim + NZ - 1) / NZ, nv = 2 * a.nmt;
  const int nitems = (a.npc - a.m0) * nzt * nv;
  auto item_m = [&](int it) { return a.m0 + it / (nzt * nv); };
  auto item_z0 = [&](int it) { return (it / nv) % nzt * NZ; };
  auto item_mt = [&](int it) { return (it % nv) >> 1; };
  auto item_par = [&](int it) { return it & 1; };
  auto live = [&](int it) {
    const int m = item_m(it), nn = max(min(a.nrc, a.nrc - m), 0);
    return 2 * (item_mt(it) * 128) + item_par(it) < nn;
  };
  auto next_item = [&](int it) {
    for (it += gridDim.x; it < nitems && !live(it); it += gridDim.x) {}
    return it;
  };
  int first = blockIdx.x;
  if (first < nitems && !live(first)) first = next_item(first);
  const int nkc = a.nkc, npart = PARTS ? XV_PART : nkc;   // chunks between drains

  if (warp == 0) {
    // ---- the table entries
    if (lane == 0) {
      uint32_t c = 0, s = 0, ph = 0;
      for (int it = first; it < nitems && ok; it = next_item(it)) {
        const uint8_t* img = (const uint8_t*)a.img +
                             (((size_t)(item_m(it) * 2 + item_par(it)) * a.nmt + item_mt(it)) * nkc) * (size_t)(xv_tiles<NS, NT>() * XV_ATILE);
        for (int kc = 0; kc < nkc && ok; ++kc)
          for (int q = 0; q < 3; ++q, ++c) {
            if (c >= AE && !xs_wait(&bar_ae[s], ph ^ 1u, ok)) break;
            const uint32_t bytes = (uint32_t)((q < 2 ? NS : NT) + MG) * XV_ATILE;
            mbar_expect_tx(&bar_af[s], bytes);
            bulk_g2s(sA + s * AENT, img, bytes, &bar_af[s]);
            img += bytes;
            if (++s == AE) { s = 0; ph ^= 1u; }
          }
      }
      // the copies issued complete on their own: wait (bounded) for the last of them, so that no copy
      // is in flight when the CTA's shared memory goes away (at once in a run without a timeout)
      for (uint32_t j = c > AE ? c - AE : 0; j < c; ++j) {
        bool ok2 = true;
        xs_wait(&bar_af[j % AE], (j / AE) & 1, ok2);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issue (the whole warp, one elected lane issuing)
    const uint32_t el = elect_lane();
    uint32_t sa = 0, pa = 0, sb = 0, pb = 0, u = 0, last = 0, plast = 0;
    bool any = false;
    // the MMAs of one table entry: digit t against the B tiles [b, b + (n - t) cols), cols tiles per digit, onto the
    // accumulators from tc on; then the magnitudes, against the tiles at bm onto tm
    auto entry = [&](auto nc, auto colsc, uint32_t b, uint32_t tc, uint32_t bm, uint32_t tm, bool add) {
      constexpr int n = decltype(nc)::value, cols = decltype(colsc)::value;
      if (!xs_wait_w(&bar_af[sa], pa, ok)) return;
      tc_fence_after();
      const uint32_t a0 = smem_u32(sA) + sa * AENT;
#pragma unroll
      for (int t = 0; t < n; ++t) {
        const uint64_t ad = sdesc(a0 + t * XV_ATILE, XV_LBO, XV_SBO);
        const int tiles = (n - t) * cols, t1 = tiles * N > 256 ? 256 / N : tiles;
        umma_bf16(tmem + tc + (uint32_t)(t * cols * N), ad, sdesc(b, XV_LBO, XV_SBO), idesc_bf16(128, t1 * N),
                  (add || t > 0) ? 1u : 0u, el);
        if (tiles > t1)
          umma_bf16(tmem + tc + (uint32_t)((t * cols + t1) * N), ad, sdesc(b + t1 * XV_BTILE, XV_LBO, XV_SBO),
                    idesc_bf16(128, (tiles - t1) * N), (add || t > 0) ? 1u : 0u, el);
      }
      if constexpr (MG != 0)
        umma_bf16(tmem + tm, sdesc(a0 + n * XV_ATILE, XV_LBO, XV_SBO), sdesc(bm, XV_LBO, XV_SBO), idesc_bf16(128, cols * N), add ? 1u : 0u, el);
      umma_commit(&bar_ae[sa], el);
      last = sa; plast = pa; any = true;
      if (++sa == AE) { sa = 0; pa ^= 1u; }
    };
    for (int it = first; it < nitems && ok; it = next_item(it))
      for (int k0 = 0; k0 < nkc && ok; k0 += npart, ++u) {
        // psi's and X's accumulators, once the epilogue has read what they held before
        if (u > 0 && !xs_wait_w(&bar_te[0], (u - 1) & 1, ok)) break;
        for (int kc = k0; kc < min(k0 + npart, nkc) && ok; ++kc) {
          if (!xs_wait_w(&bar_bf[sb], pb, ok)) break;
          const uint32_t b0 = smem_u32(sB) + sb * BSTAGE, bm = b0 + (4 * NS + NT) * XV_BTILE;
          // psi and X alternate by order (psi_d at 2d N, X_d at (2d+1) N) and their field digits alternate the same way
          // ([psi_ur_s, X_up_s] against m V, [psi_up_s, X_ur_s] against D), so one MMA covers both sums
          entry(std::integral_constant<int, NS>(), std::integral_constant<int, 2>(), b0, 0, bm, TM, kc > k0);
          if (ok) entry(std::integral_constant<int, NS>(), std::integral_constant<int, 2>(), b0 + 2 * NS * XV_BTILE, 0, bm + 2 * XV_BTILE, TM, true);
          if (kc == k0 && u > 0) xs_wait_w(&bar_te[1], (u - 1) & 1, ok);
          if (ok)
            entry(std::integral_constant<int, NT>(), std::integral_constant<int, 1>(), b0 + 4 * NS * XV_BTILE, TY, bm + 4 * XV_BTILE,
                  TM + 2 * N, kc > k0);
          if (!ok) break;
          umma_commit(&bar_be[sb], el);
          if (++sb == XV_SB) { sb = 0; pb ^= 1u; }
        }
        if (ok) umma_commit(bar_tf, el);
      }
    if (any) {   // the MMAs issued have finished (bounded) before tensor memory is freed
      bool ok2 = true;
      xs_wait_w(&bar_ae[last], plast, ok2);
    }
  } else if (warp < 2 + XV_NSW) {
    // ---- column scales: cexp(2zz) over (Im ur, Re up), cexp(2zz+1) over (Re ur, Im up); fexp over uz.  Four z columns
    // per warp, eight lanes each, over the magnitudes' high words; |x| < 2^(exponent field - 1022), +1 because the folds
    // may double.
    int ii = 0;
    for (int it = first; it < nitems && ok; it = next_item(it), ++ii) {
      const int slot = ii % XV_CXS;
      if (ii >= XV_CXS && !xs_wait_w(&bar_ce[slot], (ii / XV_CXS - 1) & 1, ok)) break;
      const int zz = (warp - 2) * 4 + (lane >> 3), z = item_z0(it) + zz;
      unsigned e0 = 0, e1 = 0, u0 = 0, u1 = 0;
      if (z < a.nzdim) {
        const size_t cb = (size_t)a.nrdim * (item_m(it) + (size_t)a.npdim * z);
        const unsigned* pr = (const unsigned*)(a.ur + cb);   // (re lo, re hi, im lo, im hi)
        const unsigned* pp = (const unsigned*)(a.up + cb);
        const unsigned* pz = (const unsigned*)(a.uz + cb);
#pragma unroll 4
        for (int i = lane & 7; i < a.nr; i += 8) {
          const unsigned rr = __ldcg(pr + 4 * i + 1), ri = __ldcg(pr + 4 * i + 3), qr = __ldcg(pp + 4 * i + 1),
                         qi = __ldcg(pp + 4 * i + 3), wr = __ldcg(pz + 4 * i + 1), wi = __ldcg(pz + 4 * i + 3);
          e0 = max(e0, max(ri & 0x7FFFFFFFu, qr & 0x7FFFFFFFu));
          e1 = max(e1, max(rr & 0x7FFFFFFFu, qi & 0x7FFFFFFFu));
          u0 = max(u0, wr & 0x7FFFFFFFu);
          u1 = max(u1, wi & 0x7FFFFFFFu);
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        e0 = max(e0, __shfl_xor_sync(0xFFFFFFFFu, e0, o));
        e1 = max(e1, __shfl_xor_sync(0xFFFFFFFFu, e1, o));
        u0 = max(u0, __shfl_xor_sync(0xFFFFFFFFu, u0, o));
        u1 = max(u1, __shfl_xor_sync(0xFFFFFFFFu, u1, o));
      }
      if ((lane & 7) == 0) {
        // an all-subnormal column counts as zero
        auto bound = [](unsigned h) {
          if (BAL && xs_nonfin(h)) return XS_NONFIN;
          return !(h >> 20) ? -2000 : (BAL ? xs_ebound_bal(h) : (int)(h >> 20) - 1022) + 1;
        };
        int* cx = cxs + slot * 2 * N;
        cx[2 * zz] = bound(e0);
        cx[2 * zz + 1] = bound(e1);
        cx[N + 2 * zz] = bound(u0);
        cx[N + 2 * zz + 1] = bound(u1);
      }
      mbar_arrive(&bar_cx[slot]);
    }
  } else if (warp < 2 + XV_NSW + 2 * XV_GW) {
    // ---- field digits: the group's chunks c = grp, grp + 2, ... of the CTA's sequence (item c / nkc, chunk c % nkc), a
    // thread's two K of its field at i and nr-1-i fetched a chunk ahead
    const int dt0 = tid - (2 + XV_NSW) * 32, grp = dt0 / (XV_GW * 32), dt = dt0 % (XV_GW * 32);
    const int f = dt / (NZ * 8), kp = dt % 8, zz = (dt / 8) % NZ;   // eight K pairs of a column in consecutive lanes
    const double2* src = f == 0 ? a.ur : (f == 1 ? a.up : a.uz);
    const int off = xv_off(2 * zz, 2 * kp), off1 = xv_off(2 * zz + 1, 2 * kp);
    double2 va[2], vb[2];
    auto fetch = [&](int it, int kc) {
      const int z = item_z0(it) + zz;
      const bool zok = z < a.nzdim;
      const size_t cbase = (size_t)a.nrdim * (item_m(it) + (size_t)a.npdim * (zok ? z : 0));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = kc * XV_KC + 2 * kp + u;
        const bool okk = zok && i < a.nrh;
        va[u] = okk ? src[cbase + i] : make_double2(0.0, 0.0);
        vb[u] = okk ? src[cbase + a.nr - 1 - i] : make_double2(0.0, 0.0);
      }
    };
    int it = first, kc = grp, ii = 0;
    auto settle = [&]() {   // chunk counts past an item's end run into the next items
      while (it < nitems && kc >= nkc) { kc -= nkc; it = next_item(it); ++ii; }
    };
    settle();
    if (it < nitems) fetch(it, kc);
    int seen = -1, base0 = 0, base1 = 0;   // the item whose column scales are in base0 (re) and base1 (im)
    for (uint32_t c = grp; it < nitems; c += 2) {
      if (ii != seen) {
        if (!xs_wait_w(&bar_cx[ii % XV_CXS], (ii / XV_CXS) & 1, ok)) break;
        const int* cx = cxs + (ii % XV_CXS) * 2 * N + (f == 2 ? N : 0);
        // Re ur lands in column 2zz+1 and Im ur in 2zz; Re up (and Re uz) in 2zz and Im up in 2zz+1
        const int er = cx[2 * zz + (f == 0 ? 1 : 0)], ei = cx[2 * zz + (f == 0 ? 0 : 1)];
        base0 = xs_fix_base(er, f == 2 ? nbt : nbs, true);
        base1 = xs_fix_base(ei, f == 2 ? nbt : nbs, true);
        seen = ii;
      }
      const uint32_t s = c % XV_SB;
      if (c >= XV_SB && !xs_wait_w(&bar_be[s], (c / XV_SB - 1) & 1, ok)) break;
      uint8_t* bst = sB + s * BSTAGE;
      const bool odd = item_par(it);   // own-parity fold sign
      // integer folds of the two components with the column scales of the columns they land in
      long long sre[2], sim[2], ore[2], oim[2];   // F_s and F_o
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const long long ar = xs_fixs(va[u].x, base0), br0 = xs_fixs(vb[u].x, base0), br = odd ? -br0 : br0;
        const long long ai = xs_fixs(va[u].y, base1), bi0 = xs_fixs(vb[u].y, base1), bi = odd ? -bi0 : bi0;
        sre[u] = ar + br; sim[u] = ai + bi;
        ore[u] = ar - br; oim[u] = ai - bi;
      }
      if (f < 2) {
        // f = 0: psi_ur = -i F_s(ur) = (Im, -Re), X_ur = i F_o(ur) = (-Im, Re)
        // f = 1: psi_up = -F_o(up) = (-Re, -Im),  X_up = F_s(up) = (Re, Im)
        // B tiles: [psi_ur_s, X_up_s] at 2s, 2s+1; [psi_up_s, X_ur_s] at 2 NS + 2s, 2 NS + 2s + 1; their magnitudes in the same
        // order behind all digits
        constexpr unsigned long long bias = BAL ? xs_bias<NS, W>() : 0ull;
        const int tp = f == 0 ? 0 : 2 * NS, tx = f == 0 ? 2 * NS + 1 : 1, mp = f == 0 ? 0 : 2, mx = f == 0 ? 3 : 1;
        auto put = [&](int tile, int mag, int o, long long p, long long q) {
          if constexpr (MG != 0) *(uint32_t*)(bst + (4 * NS + NT + mag) * XV_BTILE + o) = xs_mag2(p, q);
          const unsigned long long x0 = (unsigned long long)p + bias, x1 = (unsigned long long)q + bias;
          xs_static_for<NS>([&](auto sc) {
            constexpr int g = decltype(sc)::value;
            *(uint32_t*)(bst + (tile + 2 * g) * XV_BTILE + o) = xs_digit2<NS, W, BAL, g>(x0, x1);
          });
        };
        put(tp, mp, off, f == 0 ? sim[0] : -ore[0], f == 0 ? sim[1] : -ore[1]);
        put(tp, mp, off1, f == 0 ? -sre[0] : -oim[0], f == 0 ? -sre[1] : -oim[1]);
        put(tx, mx, off, f == 0 ? -oim[0] : sre[0], f == 0 ? -oim[1] : sre[1]);
        put(tx, mx, off1, f == 0 ? ore[0] : sim[0], f == 0 ? ore[1] : sim[1]);
      } else {
        // Y: F_s(uz) with the uz column scales
        constexpr unsigned long long bias = BAL ? xs_bias<NT, W>() : 0ull;
        xs_static_for<NT>([&](auto sc) {
          constexpr int g = decltype(sc)::value;
          *(uint32_t*)(bst + (4 * NS + g) * XV_BTILE + off) =
              xs_digit2<NT, W, BAL, g>((unsigned long long)sre[0] + bias, (unsigned long long)sre[1] + bias);
          *(uint32_t*)(bst + (4 * NS + g) * XV_BTILE + off1) =
              xs_digit2<NT, W, BAL, g>((unsigned long long)sim[0] + bias, (unsigned long long)sim[1] + bias);
        });
        if constexpr (MG != 0) {
          *(uint32_t*)(bst + (4 * NS + NT + 4) * XV_BTILE + off) = xs_mag2(sre[0], sre[1]);
          *(uint32_t*)(bst + (4 * NS + NT + 4) * XV_BTILE + off1) = xs_mag2(sim[0], sim[1]);
        }
      }
      fence_async_smem();
      mbar_arrive(&bar_bf[s]);
      kc += 2;
      settle();
      if (it < nitems) fetch(it, kc);
    }
  } else {
    // ---- epilogue: warp e reads TMEM lanes 32 (e % 4) .. (rows t) and the 8-column block e / 4
    const int lq = warp & 3, cb = (warp - 2 - XV_NSW - 2 * XV_GW) >> 2;
    const uint32_t tcol = tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(cb * 8);
    uint32_t u = 0, ii = 0;   // drains, items
    for (int it = first; it < nitems; it = next_item(it), ++u, ++ii) {
      const int m = item_m(it), mt = item_mt(it), par = item_par(it), z0 = item_z0(it);
      const int nn = max(min(a.nrc, a.nrc - m), 0);
      const int t = mt * 128 + lq * 32 + lane, j = 2 * t + par;
      const bool rok = j < nn && t < a.ntr, wlive = mt * 128 + lq * 32 < a.ntr;
      // the row exponents, loaded before the wait so that their latency hides behind it
      const int er = rok ? a.rexp[(size_t)(m * 2 + par) * a.ntr + t] : -2000;
      const int et = rok ? a.texp[(size_t)(m * 2 + par) * a.ntr + t] : -2000;
      if (!xs_wait_w(bar_tf, u & 1, ok)) break;
      tc_fence_after();
      const uint32_t slot = ii % XV_CXS;
      const int* cx = cxs + slot * 2 * N + cb * 8;   // written before the item's digits were cut, and so before its accumulators
      // the products carry 2^(-2 nb), the orders' unit is 2^(w (n-1))
      constexpr int os = W * (NS - 1) - 2 * nbs, ot = W * (NT - 1) - 2 * nbt;
      auto kept = [&](int c) {   // column c's z
        const int zc = z0 + (cb * 8 + c) / 2, kk = zc + 1;
        return zc < a.nzdim && (kk <= a.nzc || kk >= a.nzcu);
      };
      auto put = [&](int c, const double* pv, const double* xv, const double* yv) {
        const int zc = z0 + (cb * 8 + c) / 2;
        const double kz = a.ak[zc];
        const size_t o = j + (size_t)a.nrdim * (m + (size_t)a.npdim * zc);
        a.psi[o] = make_double2(pv[0], pv[1]);
        a.chi[o] = make_double2(fma(kz, xv[0], -yv[0]), fma(kz, xv[1], -yv[1]));
      };
      if constexpr (!BAL) {
        long long tp[8], tx[8], ty[8];
        if (wlive) {
          xv_sums<NS, W>(tcol, 2 * N, a.esh_s, tp);
          xv_sums<NS, W>(tcol + N, 2 * N, a.esh_s, tx);
        }
        tc_fence_before();
        mbar_arrive(&bar_te[0]);
        if (wlive) xv_sums<NT, W>(tcol + TY, N, a.esh_t, ty);
        tc_fence_before();
        mbar_arrive(&bar_te[1]);
        if (!xs_wait_w(&bar_cx[slot], (ii / XV_CXS) & 1, ok)) break;   // long since complete
        if (rok && wlive) {
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            if (!kept(c)) continue;
            double pv[2], xv[2], yv[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int E = cx[c + h], F = cx[N + c + h];
              const bool ox = er > -2000 && E > -2000, oy = et > -2000 && F > -2000;
              pv[h] = ox ? xs_i64_to_double(tp[c + h], er + E + a.esh_s + os) : 0.0;
              xv[h] = ox ? xs_i64_to_double(tx[c + h], er + E + a.esh_s + os) : 0.0;
              yv[h] = oy ? xs_i64_to_double(ty[c + h], et + F + a.esh_t + ot) : 0.0;
            }
            put(c, pv, xv, yv);
          }
        }
      } else {
        if (!xs_wait_w(&bar_cx[slot], (ii / XV_CXS) & 1, ok)) break;   // long since complete
        XvSum q;   // Y's sums in the end
        double pv[8], xv[8];
        float sx[8];
        uint32_t few = 0;   // columns whose psi has only small terms
        auto take_psi = [&](const XvSum& v) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const bool on = er > -2000 && cx[c] > -2000;
            pv[c] = on ? xv_value<NS, W>(v, c, er + cx[c] + os) : 0.0;
            few |= on && v.S[c] < a.least ? 1u << c : 0u;
          }
        };
        auto take_x = [&](const XvSum& v) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            xv[c] = er > -2000 && cx[c] > -2000 ? xv_value<NS, W>(v, c, er + cx[c] + os) : 0.0;
            sx[c] = v.S[c];
          }
        };
        auto release = [&](int which) {
          tc_fence_before();
          mbar_arrive(&bar_te[which]);
        };
        if constexpr (!PARTS) {
          if (wlive) {
            xv_drain<NS, W>(tcol, 2 * N, tcol + TM, q, true);
            take_psi(q);
            xv_drain<NS, W>(tcol + N, 2 * N, tcol + TM + N, q, true);
            take_x(q);
          }
          release(0);
          if (wlive) xv_drain<NT, W>(tcol + TY, N, tcol + TM + 2 * N, q, true);
          release(1);
        } else {
          XvSum qp, qx;
          for (int k0 = 0; k0 < nkc; k0 += npart) {
            if (k0 > 0) {
              ++u;
              if (!xs_wait_w(bar_tf, u & 1, ok)) break;
              tc_fence_after();
            }
            if (wlive) {
              xv_drain<NS, W>(tcol, 2 * N, tcol + TM, qp, k0 == 0);
              xv_drain<NS, W>(tcol + N, 2 * N, tcol + TM + N, qx, k0 == 0);
            }
            release(0);
            if (wlive) xv_drain<NT, W>(tcol + TY, N, tcol + TM + 2 * N, q, k0 == 0);
            release(1);
          }
          if (!ok) break;
          if (wlive) {
            take_psi(qp);
            take_x(qx);
          }
        }
        if (wlive) {
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            if (!kept(c)) continue;
            const int zc = z0 + (cb * 8 + c) / 2;
            const float kz = fabsf((float)a.ak[zc]);
            double yv[2];
            bool again = (few >> c) & 3u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int E = cx[c + h], F = cx[N + c + h];
              const bool ox = er > -2000 && E > -2000 && kz > 0.f, oy = et > -2000 && F > -2000;
              yv[h] = oy ? xv_value<NT, W>(q, c + h, et + F + ot) : 0.0;
              // chi = k X - Y: the terms of both against the unit of the larger; k X's in units of Y's
              const float one = oy ? 1.f : 0.f;
              const float rel = !ox ? 0.f : oy ? kz * __int_as_float((127 + min(max(er + E - et - F, -100), 100)) << 23) : 1.f;
              again = again || E == XS_NONFIN || F == XS_NONFIN || (ox || oy) && rel * sx[c + h] + one * q.S[c + h] < a.least * (rel + one);
            }
            if (rok) put(c, pv + c, xv + c, yv);
            const unsigned word = __ballot_sync(0xFFFFFFFFu, rok && again);
            if (lane == 0) a.again[xv_word(a, m, par, mt * 4 + lq, zc)] = word;
          }
        }
      }
      mbar_arrive(&bar_ce[slot]);
    }
  }
  if (!ok) atomicExch(a.status, 2);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TCOLS);
}

// The marked outputs (k_xs_again), summed in FP64: a marked row after the other, the lanes over the radial points, each lane's
// shares of the five sums combined before they are added over the warp.
__global__ void __launch_bounds__(XS_AGAIN_T) k_xv_again(XvArgs a, const double* __restrict__ tV, const double* __restrict__ tD,
                                                  const double* __restrict__ tT, int ne, size_t nwords) {
  const int lane = threadIdx.x & 31;
  const size_t nw = XS_AGAIN, wid = (size_t)blockIdx.x * (XS_AGAIN_T / 32) + (threadIdx.x >> 5);
  if (wid >= nw) return;
  int m, par, g, z;
  auto place = [&](size_t idx) {
    z = (int)(idx % a.nzdim); idx /= a.nzdim;
    g = (int)(idx % a.ngrp); idx /= a.ngrp;
    par = (int)(idx & 1);
    m = (int)(idx >> 1);
  };
  for (size_t base = wid; base < nwords; base += 32 * nw) {
    const size_t mine = base + nw * lane;
    unsigned word = 0;
    if (mine < nwords) {
      place(mine);
      const int nn = max(min(a.nrc, a.nrc - m), 0);
      // (words of other rows and columns are not written)
      if (m >= a.m0 && m < a.again_m && 2 * (g * 32) + par < nn && (z + 1 <= a.nzc || z + 1 >= a.nzcu) &&
          (z + 1 <= a.again_zl || z + 1 >= a.again_zu))
        word = a.again[mine];
    }
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, word != 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const unsigned rows = __shfl_sync(0xFFFFFFFFu, word, src);
      place(base + nw * src);
      const size_t off = (size_t)a.nrdim * (m + (size_t)a.npdim * z);
      const double2 *ur = a.ur + off, *up = a.up + off, *uz = a.uz + off;
      const double ss = par ? -1.0 : 1.0, mv = (double)m, kv = a.ak[z];
      for (unsigned left = rows; left; left &= left - 1) {
        const int j = 2 * (g * 32 + __ffs(left) - 1) + par;
        if (j >= min(a.nrc, a.nrc - m)) break;   // (words that a contraction which ran out of time left unwritten)
        const size_t row = (size_t)a.nrh * (j + (size_t)ne * m);
        double v[10];   // V.F_s(ur), D.F_o(up), D.F_o(ur), V.F_s(up), T.F_s(uz)
#pragma unroll
        for (int q = 0; q < 10; ++q) v[q] = 0.0;
        for (int i = lane; i < a.nrh; i += 32) {
          const double V = __ldg(tV + row + i), D = __ldg(tD + row + i), T = __ldg(tT + row + i);
          double2 p = __ldg(ur + i), q = __ldg(ur + a.nr - 1 - i);
          v[0] = fma(V, p.x + ss * q.x, v[0]); v[1] = fma(V, p.y + ss * q.y, v[1]);
          v[4] = fma(D, p.x - ss * q.x, v[4]); v[5] = fma(D, p.y - ss * q.y, v[5]);
          p = __ldg(up + i); q = __ldg(up + a.nr - 1 - i);
          v[6] = fma(V, p.x + ss * q.x, v[6]); v[7] = fma(V, p.y + ss * q.y, v[7]);
          v[2] = fma(D, p.x - ss * q.x, v[2]); v[3] = fma(D, p.y - ss * q.y, v[3]);
          p = __ldg(uz + i); q = __ldg(uz + a.nr - 1 - i);
          v[8] = fma(T, p.x + ss * q.x, v[8]); v[9] = fma(T, p.y + ss * q.y, v[9]);
        }
        double o[4] = {mv * v[1] - v[2], -mv * v[0] - v[3], -kv * v[5] + mv * kv * v[6] - v[8], kv * v[4] + mv * kv * v[7] - v[9]};
#pragma unroll
        for (int d = 16; d; d >>= 1)
#pragma unroll
          for (int q = 0; q < 4; ++q) o[q] += __shfl_xor_sync(0xFFFFFFFFu, o[q], d);
        if (lane == 0) {
          a.psi[off + j] = make_double2(o[0], o[1]);
          a.chi[off + j] = make_double2(o[2], o[3]);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
struct XvImg {
  uint16_t* p = nullptr;
  int *rexp = nullptr, *texp = nullptr;
  unsigned* again = nullptr;
  size_t bytes = 0, ebytes = 0, gbytes = 0;
  int nrc = -1, npc = -1, ns = 0;
};
static XvImg g_xvs[2];   // plain, mixed

static void xv_drop(XvImg& im) {
  if (im.p) dfree(im.p, im.bytes);
  if (im.rexp) dfree(im.rexp, im.ebytes);
  if (im.texp) dfree(im.texp, im.ebytes);
  if (im.again) dfree(im.again, im.gbytes);
  im = XvImg();
}
void xv_free() {
  for (XvImg& im : g_xvs) xv_drop(im);
}

// digit counts of psi / X and of Y and their width; ns = 0 where no configuration is exact
struct XvCfg { int ns, nt, w; };
static XvCfg xv_cfg(int k, bool plain) {
  if (plain) return k <= 372 ? XvCfg{9, 9, 7} : XvCfg{0, 0, 0};
  const double lim = 16777216.0;
  auto fits = [&](int ns, int nt, int w) {
    const double d = (double)(1 << w) * (1 << w);   // largest digit product (two's-complement digits)
    return 2.0 * ns * k * d < lim && (double)nt * k * d < lim;
  };
  if (fits(5, 7, 7)) return {5, 7, 7};
  if (fits(6, 8, 6)) return {6, 8, 6};
  return {0, 0, 0};
}

bool xv_supported(bool plain) { return xv_cfg(G.nrh, plain).ns > 0; }

template <int NS, int NT, int W>
static int xv_image(const XvArgs& args, XvImg& im, int npc, bool plain) {
  if (im.nrc != args.nrc || im.npc != npc || !im.p || im.ns != NS) {
    xv_drop(im);
    im.bytes = (size_t)npc * 2 * args.nmt * args.nkc * xv_tiles<NS, NT>() * XV_ATILE;
    im.ebytes = (size_t)npc * 2 * args.ntr * sizeof(int);
    im.gbytes = xv_mag<NS>() ? (size_t)npc * 2 * cdiv(args.ntr, 32) * G.nzdim * sizeof(unsigned) : 0;
    if (int rc = dmalloc_all({{(void**)&im.p, im.bytes}, {(void**)&im.rexp, im.ebytes}, {(void**)&im.texp, im.ebytes},
                              {(void**)&im.again, im.gbytes}}))
      return rc;
    k_xv_rexp<<<dim3(cdiv(args.ntr, 128), npc * 2), 128, 0, G.stream>>>(G.tV, G.tD, G.tT, im.rexp, im.texp, G.nrh, G.ne, args.nrc,
                                                                        args.ntr, plain ? 1 : 0);
    MLG_LAUNCH();
    k_xv_table<NS, NT, W><<<npc * 2 * args.nmt * args.nkc, 256, 0, G.stream>>>(
        G.tV, G.tD, G.tT, im.rexp, im.texp, im.p, G.nrh, G.ne, args.nrc, args.nmt, args.nkc, args.ntr);
    MLG_LAUNCH();
    im.nrc = args.nrc; im.npc = npc; im.ns = NS;
  }
  return 0;
}
template <int NS, int NT, int W, bool PARTS = false>
static int xv_run(XvArgs args, const XvImg& im, int npc) {
  args.img = im.p; args.rexp = im.rexp; args.texp = im.texp;
  args.again = im.again; args.ngrp = cdiv(args.ntr, 32); args.least = xs_least_sum(2 * G.nrh);   // psi's and X's sums of two products
  const size_t fixed = 1024 + XV_SB * (size_t)xv_bstage_bytes<NS, NT>() + XV_CXS * 2 * XV_N * sizeof(int) + 512;
  args.aent = (int)std::min<size_t>(XV_AEMAX, (227 * 1024 - fixed) / xv_aent_bytes<NS, NT>());
  const size_t sm = fixed + (size_t)args.aent * xv_aent_bytes<NS, NT>();
  auto kern = k_xv_contract<NS, NT, W, PARTS>;
  MLG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  const int nitems = (npc - args.m0) * 2 * args.nmt * cdiv(G.nzdim, XV_NZ);
  kern<<<std::min(nitems, 152), XV_THREADS, sm, G.stream>>>(args);
  MLG_LAUNCH();
  if (xv_mag<NS>()) {
    k_xv_again<<<cdiv(XS_AGAIN, XS_AGAIN_T / 32), XS_AGAIN_T, 0, G.stream>>>(args, G.tV, G.tD, G.tT, G.ne, (size_t)npc * 2 * args.ngrp * G.nzdim);
    MLG_LAUNCH();
  }
  return 0;
}

// the table images, as xs_prepare
static void xv_extent(XvArgs& args, int nrc) {
  args.nrc = nrc;
  args.ntr = (nrc + 1) / 2;
  args.nmt = cdiv(args.ntr, 128); args.nkc = cdiv(G.nrh, XV_KC);
}
int xv_prepare(int nrc, int npc, bool plain) {
  XvArgs args{};
  xv_extent(args, nrc);
  XvImg& im = g_xvs[plain ? 0 : 1];
  switch (xv_cfg(G.nrh, plain).ns) {
    case 9: return xv_image<9, 9, 7>(args, im, npc, plain);
    case 5: return xv_image<5, 7, 7>(args, im, npc, plain);
    default: return xv_image<6, 8, 6>(args, im, npc, plain);
  }
}

// psi, chi: the rows of m0 <= m < npc written (zeroed elsewhere by the caller).  dealias_next: outputs that the caller's dealias
// mask zeroes are not summed again (many of the marked ones are high modes: 41 -> 19 us in the nonlinear term at 256 x 128 x 128)
int xv_contract(const cd* ur, const cd* up, const cd* uz, cd* psi, cd* chi, int nrc, int npc, int m0, bool plain, bool dealias_next) {
  if (npc <= m0) return 0;
  const XvCfg cfg = xv_cfg(G.nrh, plain);
  if (!cfg.ns) return set_error(MLG_ESIZE, "vec2tp: too many radial points for exact slices");
  XvArgs args{};
  args.ur = ur; args.up = up; args.uz = uz; args.psi = psi; args.chi = chi;
  args.ak = G.ak; args.status = (int*)(G.dscal + DS_FLAG + 1) + 1;
  args.nr = G.nr; args.nrh = G.nrh; args.nrdim = G.nrdim; args.npdim = G.npdim; args.nzdim = G.nzdim;
  const bool dp = dealias_next && G.np > 1, dz = dealias_next && G.nz > 1;
  args.again_m = dp ? std::min(npc, dealias_pcut()) : npc;
  args.again_zl = dz ? dealias_zcut() : G.nzdim;
  args.again_zu = dz ? G.nz - dealias_zcut() + 2 : 1;
  args.nzc = G.chopzl; args.nzcu = G.chopzu; args.m0 = m0; args.npc = npc;
  xv_extent(args, nrc);
  {
    // the 64-bit order sums stay below 2^62: |G_d| <= K (pairs of order d) 2^(2w), with two products
    // per digit pair for psi and X
    auto esh = [&](int n, int pairs) {
      const double mx = (double)G.nrh * pairs * (1 << cfg.w) * (1 << cfg.w);
      return std::max(0, (int)std::ceil(std::log2(mx) + 0.05) + cfg.w * (n - 1) - 62);
    };
    args.esh_s = esh(cfg.ns, 2 * cfg.ns);
    args.esh_t = esh(cfg.nt, cfg.nt);
  }
  MLG_TRY(xv_prepare(nrc, npc, plain));
  const XvImg& im = g_xvs[plain ? 0 : 1];
  if (cfg.ns == 9) return xs_order_bound(9, 7, 2, G.nrh) <= XS_EXACT ? xv_run<9, 9, 7>(args, im, npc) : xv_run<9, 9, 7, true>(args, im, npc);
  if (cfg.ns == 5) return xv_run<5, 7, 7>(args, im, npc);
  return xv_run<6, 8, 6>(args, im, npc);
}

}  // namespace mlg
