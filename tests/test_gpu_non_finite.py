"""A non-finite sample reaches the outputs of the plain form's contractions that it enters, and no others."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [62, 250, 288, 512])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_radial(nr, value):
    from mlegs_gb300.kit import Kit
    nz = 18
    k = Kit(make_params(nr=nr, np=16, nz=nz, nrchop=nr, npchop=9, nzchop=10, ell=4.0))
    try:
        rng = np.random.default_rng(nr)
        for space, to, rows, out in (("FFP", "PFP", lambda m: nr - m, lambda m: nr), ("PFP", "FFP", lambda m: nr, lambda m: nr - m)):
            e = np.zeros(k.dims, complex, order="F")
            for m in range(9):
                e[:rows(m), m] = rng.standard_normal((rows(m), nz)) + 1j * rng.standard_normal((rows(m), nz))
            s = k.scalar(e, 0.0, space)
            k.trans(s, to)
            clean = s.e.copy()
            bad = e.copy()
            bad[7, 3, 2] = complex(value, bad[7, 3, 2].imag)
            bad[nr // 2, 5, 17] = complex(bad[nr // 2, 5, 17].real, value)
            s.set(bad, 0.0, space)
            k.trans(s, to)
            got = s.e
            assert not np.isfinite(got[:out(3), 3, 2].real).any()
            assert not np.isfinite(got[:out(5), 5, 17].imag).any()
            rest = np.ones(k.dims, bool)
            rest[:, 3, 2] = rest[:, 5, 17] = False
            assert np.array_equal(got[rest], clean[rest])
            s.free()
    finally:
        k.close()


@pytest.mark.parametrize("nr", [64, 256, 400])
@pytest.mark.parametrize("where", [0, 1, 2])
def test_non_finite_velocity(nr, where):
    """A NaN in one sample of a velocity component is a NaN in every coefficient of the projection that it enters."""
    from mlegs_gb300.kit import Kit
    k = Kit(make_params(nr=nr, np=16, nz=6, nrchop=nr, npchop=9, nzchop=4, ell=4.0))
    try:
        rng = np.random.default_rng(nr)
        v = []
        for q in range(3):
            e = np.zeros(k.dims, complex, order="F")
            e[:nr, :8] = rng.standard_normal((nr, 8, 6)) + 1j * rng.standard_normal((nr, 8, 6))
            if q == where:
                e[9, 3, 2] = np.nan
            v.append(k.scalar(e, 0.0, "PPP"))
        psi, chi = (k.scalar(np.zeros(k.dims, complex, order="F"), 0.0, "FFF") for _ in range(2))
        k.vec2tp(*v, psi, chi)
        if where < 2:   # v_z enters chi alone
            g = psi.e
            for m in range(1, 9):
                assert not np.isfinite(g[:nr - m, m]).any(), ("psi", m)
        g = chi.e
        for m in range(1, 9):
            kz = slice(None) if where == 2 else slice(1, None)   # chi of v_r and v_phi carries a factor k
            assert not np.isfinite(g[:nr - m, m, kz]).any(), ("chi", m)
    finally:
        k.close()
