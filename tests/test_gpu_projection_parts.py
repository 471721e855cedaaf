"""The projection beyond 372 radial points, whose accumulators are drained in parts: entry by entry, and the whole of psi and
chi against the oracle (the bars of test_gpu_slices.py; the (m, k) = (0, 0) column of chi on its own path)."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params
from test_gpu_projection_entries import check_psi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [374, 512, 744])
@pytest.mark.parametrize("m", [12, 31])
def test_entries(nr, m):
    check_psi(nr, m)


@pytest.mark.parametrize("nr,nrchop,nz", [(374, 374, 4), (512, 500, 18), (744, 744, 2)])
def test_against_the_oracle(nr, nrchop, nz):
    from mlegs_gb300 import fields
    from mlegs_gb300.kit import Kit
    from oracle.oracle import Oracle
    p = make_params(nr=nr, np=8, nz=nz, nrchop=nrchop, npchop=5, nzchop=nz // 2 + 1, ell=4.0)
    o, k = Oracle(p), Kit(p)
    try:
        a = [o.scalar(fields.spectral_noise(p, k.dims, 5 + i, amp=1.0, decay=0.3), 0.0, "FFF") for i in range(2)]
        v = [o.scalar(np.zeros(k.dims, complex), 0.0, "PPP") for _ in range(3)]
        o.tp2vec(*a, *v)
        o.vec2tp(*v, *a)
        g = [k.scalar(np.zeros(k.dims, complex, order="F"), 0.0, "FFF") for _ in range(2)]
        k.vec2tp(*[k.scalar(s.e, 0.0, "PPP") for s in v], *g)
        for i, tol in ((0, 1e-12), (1, 1e-11)):
            got, want = g[i].e.copy(), a[i].e.copy()
            got[:, 0, 0] = want[:, 0, 0] = 0
            err = np.linalg.norm(got - want) / np.linalg.norm(want)
            assert err <= tol, (i, err)
    finally:
        k.close()
        o.close()
