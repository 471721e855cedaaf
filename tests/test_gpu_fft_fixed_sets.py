"""The fixed-point FFTs of lengths that are no power of two on sets with points enough for them (4e4 a transform; smaller
sets run in FP64): every pair of passes' radices along phi and z, and lines outside the fixed-point range."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params
from test_gpu_fft_fixed import check, rows

pytestmark = pytest.mark.gpu

ENOUGH = 40000
LENGTHS = [18, 20, 24, 27, 30, 36, 40, 45, 48, 50, 54, 60, 72, 75, 80, 81, 90, 96, 100, 108, 120, 135, 144, 150, 160, 180,
           192, 225, 240]


def fft_length(least):
    n = max(least + least % 2, 2)
    while True:
        r = n
        for f in (2, 3, 5):
            while r % f == 0:
                r //= f
        if r == 1:
            return n
        n += 2


def phi_kit(n):
    from mlegs_gb300.kit import Kit
    nz = fft_length(max(6, -(-ENOUGH // (23 * n))))
    k = Kit(make_params(nr=20, np=2 * n, nz=nz, nrchop=20, npchop=4, nzchop=nz // 2 + 1))
    assert k.dims[0] * k.dims[2] * n >= ENOUGH
    return k


def z_kit(n):
    from mlegs_gb300.kit import Kit
    np_ = fft_length(max(8, 2 * -(-ENOUGH // (23 * n))))
    k = Kit(make_params(nr=20, np=np_, nz=n, nrchop=20, npchop=4, nzchop=n // 2 + 1))
    assert k.dims[0] * k.dims[1] * n >= ENOUGH
    return k


def real_lines(e, n):
    x = np.empty((e.shape[0], 2 * n, e.shape[2]), np.longdouble)
    x[:, 0::2], x[:, 1::2] = e[:, :n].real, e[:, :n].imag
    return x


def phi_both(k, s, e, n, lines):
    s.set(e, 0.0, "PFP")
    k.trans(s, "PPP")
    g = s.e[lines]
    half = e[lines].astype(np.clongdouble)
    half[:, 0].imag = 0
    half[:, n].imag = 0
    check(real_lines(g, n), np.fft.irfft(half, n=2 * n, axis=1) * (2 * n), 1, "phi backward")
    s.set(e, 0.0, "PPP")
    k.trans(s, "PFP")
    check(s.e[lines], np.fft.rfft(real_lines(e[lines], n), axis=1) / (2 * n), 1, "phi forward")


def z_both(k, s, e, n, lines):
    s.set(e, 0.0, "FFF")
    k.trans(s, "FFP")
    check(s.e[lines], np.fft.ifft(e[lines].astype(np.clongdouble), axis=2) * n, 2, "z backward")
    s.set(e, 0.0, "FFP")
    k.trans(s, "FFF")
    check(s.e[lines], np.fft.fft(e[lines].astype(np.clongdouble), axis=2) / n, 2, "z forward")


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("peak", [False, True])
def test_phi(n, peak):
    k = phi_kit(n)
    try:
        phi_both(k, k.scalar(), rows(np.random.default_rng(n), k.dims, 1 if peak else None), n, slice(None))
    finally:
        k.close()


@pytest.mark.parametrize("n", [n for n in LENGTHS if n % 2 == 0])
@pytest.mark.parametrize("peak", [False, True])
def test_z(n, peak):
    k = z_kit(n)
    try:
        z_both(k, k.scalar(), rows(np.random.default_rng(n), k.dims, 2 if peak else None), n, slice(None))
    finally:
        k.close()


@pytest.mark.parametrize("n", [18, 36, 60])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e306, 1e-300])
def test_out_of_range_lines(n, value):
    for make, both in ((phi_kit, phi_both), (z_kit, z_both)):
        k = make(n)
        try:
            rng = np.random.default_rng(n)
            e = rng.standard_normal(k.dims) + 1j * rng.standard_normal(k.dims)
            if value == 1e-300:
                e[5] *= value
            else:
                e[5, :2, :2] = value
            both(k, k.scalar(), np.asfortranarray(e), n, np.arange(k.dims[0]) != 5)
        finally:
            k.close()
