"""z and phi transforms of lengths that are no power of two in 16..256: one and several register passes, both forms.

Tolerance, per line in the 2-norm: a stage of the transform (a twiddle from a rounded table, a sum of at most five terms)
changes a line by at most 10 u relative, and the phi transforms' split and the conversions count as two stages more, so
10 (stages + 2) u; u = 2^-53, or 2^-24 where the mixed form runs in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stages(n):
    s = 0
    while n > 1:
        n //= next(p for p in (4, 2, 3, 5) if n % p == 0)
        s += 1
    return s


def close(got, want, axis, u, n):
    e = np.sqrt((np.abs(got - want) ** 2).sum(axis))
    v = np.sqrt((np.abs(want) ** 2).sum(axis))
    assert np.all(e <= 10 * (stages(n) + 2) * u * v), float((e / v).max() / u)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [6, 8, 12, 20, 30, 36, 54, 60, 80, 90, 96, 100, 162, 250, 320, 486, 512])
def test_z(n, mixed):
    from mlegs_gb300.kit import MIXED, PLAIN_FP64, Kit
    from mlegs_gb300.params import make_params

    k = Kit(make_params(nr=20, np=16, nz=n, nrchop=20, npchop=9, nzchop=n // 2 + 1), precision=MIXED if mixed else PLAIN_FP64)
    try:
        rng = np.random.default_rng(n)
        e = rng.standard_normal(k.dims) + 1j * rng.standard_normal(k.dims)
        s = k.scalar(e, 0, "FFF")
        k.trans(s, "FFP")
        back = s.e
        s.set(e, 0, "FFP")
        k.trans(s, "FFF")
        fwd = s.e
        s.free()
        for got, want in ((back, np.fft.ifft(e, axis=2) * n), (fwd, np.fft.fft(e, axis=2) / n)):
            close(got[:, :1], want[:, :1], 2, 2.0**-53, n)
            close(got[:, 1:], want[:, 1:], 2, 2.0**-24 if mixed else 2.0**-53, n)
    finally:
        k.close()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 12, 15, 25, 27, 45, 60, 75, 96, 125, 160, 243, 512])
def test_phi(n, mixed):
    from mlegs_gb300.kit import MIXED, PLAIN_FP64, Kit
    from mlegs_gb300.params import make_params

    k = Kit(make_params(nr=20, np=2 * n, nz=4, nrchop=20, npchop=min(9, n + 1), nzchop=3), precision=MIXED if mixed else PLAIN_FP64)
    try:
        rng = np.random.default_rng(n)
        d, u = k.dims, 2.0**-24 if mixed else 2.0**-53
        e = rng.standard_normal(d) + 1j * rng.standard_normal(d)
        s = k.scalar(e, 0, "PFP")
        k.trans(s, "PPP")
        g = s.e
        got = np.empty((d[0], 2 * n, d[2]))
        got[:, 0::2], got[:, 1::2] = g[:, :n].real, g[:, :n].imag
        h = e[:, : n + 1].copy()
        h[:, 0].imag = 0
        h[:, n].imag = 0
        close(got, np.fft.irfft(h, n=2 * n, axis=1) * 2 * n, 1, u, n)
        np.testing.assert_allclose(g[:, n], e[:, n] * 2 * n, rtol=2.0**-52)
        s.set(e, 0, "PPP")
        k.trans(s, "PFP")
        x = np.empty((d[0], 2 * n, d[2]))
        x[:, 0::2], x[:, 1::2] = e[:, :n].real, e[:, :n].imag
        close(s.e[:, : n + 1], np.fft.rfft(x, axis=1) / (2 * n), 1, u, n)
        s.free()
    finally:
        k.close()
