"""The plain form's projection entry by entry: psi is as near to the exact sum as an FP64 sum of the same terms, also where
a row's large table entries meet a field that is small there."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def check_psi(nr, m):
    """psi of a radial velocity g(r) cos(m phi) in the core: -i m V F_s(r v_r).  To the sum's own bound (psi's 2 K terms share
    their sums) come the rounding of the table's and the transform's entries, eight units of 2^-53 at most."""
    from mlegs_gb300.kit import Kit
    p = make_params(nr=nr, np=64, nz=2, nrchop=nr, npchop=33, nzchop=2, ell=4.0)
    k = Kit(p)
    try:
        h = nr // 2
        pf, x, w = (k.kit_get(n) for n in ("pf", "x", "w"))
        r = k.kit_get("r").astype(np.longdouble)
        phi = 2 * np.pi / 64 * np.arange(64)
        v = np.exp(-6 * r.astype(float)[:nr, None] ** 2) * np.cos(m * phi)[None]
        e = np.zeros(k.dims, complex, order="F")
        e[:nr, :32, :] = (v[:, 0::2] + 1j * v[:, 1::2])[:, :, None]
        vr, vp, vz = k.scalar(e, 0.0, "PPP"), k.scalar(0 * e, 0.0, "PPP"), k.scalar(0 * e, 0.0, "PPP")
        psi, chi = k.scalar(0 * e, 0.0, "FFF"), k.scalar(0 * e, 0.0, "FFF")
        k.vec2tp(vr, vp, vz, psi, chi)
        got = psi.e
        ang = 2 * np.longdouble(np.pi) / 64 * (m * np.arange(64) % 64)
        ur = r[:nr] * (v.astype(np.longdouble) @ np.cos(ang)) / 64
        nn = nr - m
        n = m + np.arange(nn)
        V = (m * (pf[:, :nn, m].T / n[:, None] / (n[:, None] + 1) / ((1 - x[:h] ** 2) / w[:h]))).astype(np.longdouble)
        for par in (0, 1):
            a, b = V[par::2], ur[:h] + (1 - 2 * par) * ur[h:][::-1]
            ref, s = -(a @ b), np.abs(a) @ np.abs(b)
            err = np.abs(got[par:nn:2, m, 0].imag - ref)
            bad = err > (3 * np.sqrt(2 * h) + 8) * U * s
            assert not bad.any(), (par, float((err / s).max() / U), int(bad.sum()))
        for q in (vr, vp, vz, psi, chi):
            q.free()
    finally:
        k.close()


@pytest.mark.parametrize("nr", [64, 192, 256, 370])
@pytest.mark.parametrize("m", [12, 31])
def test_projection_entries(nr, m):
    check_psi(nr, m)
