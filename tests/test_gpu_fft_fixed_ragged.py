"""The plain form's fixed-point FFTs of lengths that are no power of two, as test_gpu_fft_fixed.py has the powers: every
pair of passes' radices, white and one-mode lines, rows over the exponent range, and lines outside the fixed-point range."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params
from test_gpu_fft_fixed import check, rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [18, 20, 24, 27, 30, 36, 40, 45, 48, 50, 54, 60, 72, 75, 80, 81, 90, 96, 100, 108, 120, 135, 144,
                               150, 160, 180, 192, 225, 240])
@pytest.mark.parametrize("peak", [False, True])
def test_fixed_point_ragged(n, peak):
    from mlegs_gb300.kit import Kit
    rng = np.random.default_rng(n)
    nz = n if n % 2 == 0 else 6
    k = Kit(make_params(nr=20, np=2 * n, nz=nz, nrchop=20, npchop=4, nzchop=nz // 2 + 1))
    try:
        d = k.dims
        s = k.scalar()
        if nz == n:
            e = rows(rng, d, 2 if peak else None)
            s.set(e, 0.0, "FFF")
            k.trans(s, "FFP")
            check(s.e, np.fft.ifft(e.astype(np.clongdouble), axis=2) * n, 2, "z backward")
            s.set(e, 0.0, "FFP")
            k.trans(s, "FFF")
            check(s.e, np.fft.fft(e.astype(np.clongdouble), axis=2) / n, 2, "z forward")
        e = rows(rng, d, 1 if peak else None)
        s.set(e, 0.0, "PFP")
        k.trans(s, "PPP")
        g = s.e
        half = e.astype(np.clongdouble)
        half[:, 0].imag = 0
        half[:, n].imag = 0
        f = np.empty((d[0], 2 * n, d[2]))
        f[:, 0::2], f[:, 1::2] = g[:, :n].real, g[:, :n].imag
        check(f, np.fft.irfft(half, n=2 * n, axis=1) * (2 * n), 1, "phi backward")
        assert np.array_equal(g[:, n], e[:, n] * (2 * n))
        s.set(e, 0.0, "PPP")
        k.trans(s, "PFP")
        x = np.empty((d[0], 2 * n, d[2]), np.longdouble)
        x[:, 0::2], x[:, 1::2] = e[:, :n].real, e[:, :n].imag
        check(s.e, np.fft.rfft(x, axis=1) / (2 * n), 1, "phi forward")
    finally:
        k.close()


@pytest.mark.parametrize("n", [36, 90, 240])
@pytest.mark.parametrize("value", [np.inf, np.nan, 1e306, 1e-300])
def test_out_of_range_lines_ragged(n, value):
    """A line with such a sample takes the FP64 transform and the lines beside it stay right (all of a block's lines do)."""
    from mlegs_gb300.kit import Kit
    rng = np.random.default_rng(n)
    k = Kit(make_params(nr=20, np=2 * n, nz=n, nrchop=20, npchop=4, nzchop=n // 2 + 1))
    try:
        d = k.dims
        e = rng.standard_normal(d) + 1j * rng.standard_normal(d)
        if value == 1e-300:
            e[5] *= value
        else:
            e[5, :2, :2] = value
        s = k.scalar()
        rest = np.arange(d[0]) != 5
        small = value == 1e-300
        for sp, to, ref, ax in (("FFF", "FFP", lambda a: np.fft.ifft(a, axis=2) * n, 2),
                                ("FFP", "FFF", lambda a: np.fft.fft(a, axis=2) / n, 2)):
            s.set(e, 0.0, sp)
            k.trans(s, to)
            g = s.e
            want = ref(e[rest].astype(np.clongdouble))
            check(g[rest], want, ax, to)
            if small:
                check(g[5:6] * 2.0**900, ref((e[5:6] * 2.0**900).astype(np.clongdouble)), ax, to)
            elif not np.isfinite(value):
                assert not np.any(np.isfinite(g[5, :2]).all(axis=-1))
        s.set(e, 0.0, "PPP")
        k.trans(s, "PFP")
        x = np.empty((d[0], 2 * n, d[2]), np.longdouble)
        x[:, 0::2], x[:, 1::2] = e[:, :n].real, e[:, :n].imag
        check(s.e[rest], np.fft.rfft(x[rest], axis=1) / (2 * n), 1, "phi forward")
        if small:
            check(s.e[5:6] * 2.0**900, np.fft.rfft(x[5:6] * 2.0**900, axis=1) / (2 * n), 1, "phi forward")
        s.set(e, 0.0, "PFP")
        k.trans(s, "PPP")
        g = s.e
        half = e[rest].astype(np.clongdouble)
        half[:, 0].imag = 0
        half[:, n].imag = 0
        f = np.empty((rest.sum(), 2 * n, d[2]))
        f[:, 0::2], f[:, 1::2] = g[rest][:, :n].real, g[rest][:, :n].imag
        check(f, np.fft.irfft(half, n=2 * n, axis=1) * (2 * n), 1, "phi backward")
    finally:
        k.close()
