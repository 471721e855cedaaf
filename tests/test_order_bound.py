"""The bound by which the balanced digits' orders are held exact in FP32 accumulators (xs_order_bound), on the host, against the
digits' extremes, and the radial points that it allows."""
import subprocess

import numpy as np

from mlegs_gb300.build import ARCH, CSRC, nvcc

SRC = r"""
#include "xs_common.cuh"
#include <cstdio>
int main() {
  for (int ns = 8; ns <= 9; ++ns)
    for (int products = 1; products <= 2; ++products)
      for (int K = 1; K <= 400; ++K)
        printf("%d %d %d %.0f %d\n", ns, products, K, mlg::xs_order_bound(ns, ns == 8 ? 8 : 7, products, K),
               mlg::xs_order_bound(ns, ns == 8 ? 8 : 7, products, K) <= mlg::XS_EXACT);
}
"""


def largest(ns, w):
    """The largest |order sum| of one term: every digit at the end of its range that makes its products positive and large."""
    top = np.array([128.0] + [2.0 ** (w - 1)] * (ns - 1))   # -128, -2^(w-1): the larger ends
    return max(float((top[:d + 1] * top[d::-1]).sum()) for d in range(ns))


def test_bound(tmp_path):
    src, exe = tmp_path / "b.cu", tmp_path / "b"
    src.write_text(SRC)
    subprocess.run([nvcc(), *ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    most = {}
    for line in out.splitlines():
        ns, products, K, bound, fits = (int(v) for v in line.split())
        want = largest(ns, 8 if ns == 8 else 7) * products * K
        assert bound == want
        assert fits == (want <= 2 ** 24)
        if fits:
            most[ns, products] = K
    assert most == {(8, 1): 128, (8, 2): 64, (9, 1): 372, (9, 2): 186}
