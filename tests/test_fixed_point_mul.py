"""The rounding of the fixed-point multiplications of the plain form's FFTs (fft_fixed.cuh), on the host: against the exact
128-bit product the error of q_mul is centred and bounded, for twiddles of either sign (a
conjugated twiddle has both parts of its imaginary component negated; the constants of sixteenths, either component)."""
import subprocess

import pytest

from mlegs_gb300.build import ARCH, CSRC, nvcc

SRC = r"""
#include "fft_fixed.cuh"
#include <cstdio>
#include <random>
using namespace mlg;
typedef __int128 big;
int main() {
  std::mt19937_64 g(7);
  const long long one = 1ll << 61;
  for (int neg = 0; neg < 4; ++neg)         // bit 0: real part negative, bit 1: imaginary part
    for (int rep = 0; rep < 64; ++rep) {
      const long long wx = (long long)(g() % (one - 1)), wy = (long long)(g() % (one - 1));
      int4 w = make_int4((int)(wx >> 31), (int)(wy >> 31), (int)(wx & 0x7FFFFFFF), (int)(wy & 0x7FFFFFFF));
      if (neg & 1) { w.x = -w.x; w.z = -w.z; }
      if (neg & 2) { w.y = -w.y; w.w = -w.w; }
      const big re = neg & 1 ? -wx : wx, im = neg & 2 ? -wy : wy;
      double mr = 0, mi = 0, top = 0;
      const int n = 4000;
      for (int i = 0; i < n; ++i) {
        const qc v = {(long long)g() >> 4, (long long)g() >> 4};   // |v| < 2^59.5
        const qc r = q_mul(v, w);
        auto err = [](long long got, big want) {   // got - want 2^-61
          return (double)((big)got * ((big)1 << 61) - want) / 2305843009213693952.0;
        };
        const double er = err(r.x, v.x * re - v.y * im), ei = err(r.y, v.x * im + v.y * re);
        mr += er; mi += ei;
        top = std::max(top, std::max(std::fabs(er), std::fabs(ei)));
      }
      printf("%d %.6f %.6f %.6f\n", neg, mr / n, mi / n, top);
    }
}
"""


def test_q_mul_is_centred(tmp_path):
    src, exe = tmp_path / "q.cu", tmp_path / "q"
    src.write_text(SRC)
    subprocess.run([nvcc(), *ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [[float(x) for x in line.split()] for line in out.splitlines()]
    assert len(rows) == 256
    for neg, mean_re, mean_im, top in rows:
        # a component drops two products of low parts, each in [0, 2) units and replaced by its mean (within one unit of it,
        # spread 0.58 at most), and rounds once to a unit: 2.5 units at most (and the means' own last bits, 2^-29), spread
        # 0.87, so the mean of 4 000 is within 0.1 (seven of its own spreads) of zero
        assert abs(mean_re) < 0.1 and abs(mean_im) < 0.1, (neg, mean_re, mean_im)
        assert top < 2.5 + 2.0 ** -28, (neg, top)
