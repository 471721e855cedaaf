"""The plain form's fixed-point FFTs (power-of-two lengths 16..256) against NumPy's FFT in extended precision: every
length, white and one-mode lines, rows scaled over the exponent range, zero lines, and the lines that the kernels hand to
the FP64 transform (non-finite, huge and tiny samples)."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu

# relative L2 over a line: a few units in the last place of FP64 (the FP64 transforms themselves reach 3 x 2^-53)
TOL = 4 * 2.0 ** -53


def check(got, want, axis, what):
    num = np.sqrt((np.abs(got - want) ** 2).sum(axis=axis))
    den = np.sqrt((np.abs(want) ** 2).sum(axis=axis))
    bad = num > TOL * den
    assert not np.any(bad), (what, float((num / np.where(den == 0, 1, den)).max()))


def rows(rng, d, peak):
    """White rows, or rows of one large coefficient over small ones; row i times 2^(40 i - 400); row 3 zero."""
    e = rng.standard_normal(d) + 1j * rng.standard_normal(d)
    if peak is not None:
        e *= 1e-6
        e[(slice(None),) * peak + (0,)] = 1.0
    e *= np.ldexp(1.0, 40 * np.arange(d[0]) - 400)[:, None, None]
    e[3] = 0
    return np.asfortranarray(e)


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("peak", [False, True])
def test_fixed_point_transforms(n, peak):
    from mlegs_gb300.kit import Kit
    rng = np.random.default_rng(n)
    k = Kit(make_params(nr=20, np=2 * n, nz=n, nrchop=20, npchop=4, nzchop=n // 2 + 1))
    try:
        d = k.dims
        s = k.scalar()
        # z
        e = rows(rng, d, 2 if peak else None)
        s.set(e, 0.0, "FFF")
        k.trans(s, "FFP")
        check(s.e, np.fft.ifft(e.astype(np.clongdouble), axis=2) * n, 2, "z backward")
        s.set(e, 0.0, "FFP")
        k.trans(s, "FFF")
        check(s.e, np.fft.fft(e.astype(np.clongdouble), axis=2) / n, 2, "z forward")
        # phi
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


def test_lines_outside_the_fixed_point_range():
    from mlegs_gb300.kit import Kit
    rng = np.random.default_rng(1)
    n = 32
    k = Kit(make_params(nr=20, np=2 * n, nz=n, nrchop=20, npchop=4, nzchop=n // 2 + 1))
    try:
        d = k.dims
        e = np.asfortranarray(rng.standard_normal(d) + 1j * rng.standard_normal(d))
        e[0] *= 1e304                   # huge
        e[1] *= 1e-290                  # tiny
        e[2, 5, 7] = np.nan
        e[4, 6, 9] = np.inf
        s = k.scalar()
        for space, to, axis, fn in (("FFF", "FFP", 2, lambda a: np.fft.ifft(a, axis=2) * n),
                                    ("FFP", "FFF", 2, lambda a: np.fft.fft(a, axis=2) / n)):
            s.set(e, 0.0, space)
            k.trans(s, to)
            g, want = s.e, fn(e.astype(np.clongdouble))
            fine = np.isfinite(want.astype(complex)).all(axis=axis)
            assert np.array_equal(np.isfinite(g).all(axis=axis), fine)
            check(np.where(fine[..., None], g, 0), np.where(fine[..., None], want, 0), axis, to)
        s.set(e, 0.0, "PPP")
        k.trans(s, "PFP")
        g = s.e
        x = np.empty((d[0], 2 * n, d[2]), np.longdouble)
        x[:, 0::2], x[:, 1::2] = e[:, :n].real, e[:, :n].imag
        want = np.fft.rfft(x, axis=1) / (2 * n)
        fine = np.isfinite(want.astype(complex)).all(axis=1)
        assert np.array_equal(np.isfinite(g).all(axis=1), fine)
        check(np.where(fine[:, None], g, 0), np.where(fine[:, None], want, 0), 1, "PFP")
    finally:
        k.close()
