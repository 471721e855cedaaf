"""The nonlinear term leaves marked outputs of the projection alone where its dealias mask zeroes them: the same bits as the
operations one by one, whose projection sums every marked output again."""
import numpy as np
import pytest

from mlegs_gb300 import fields
from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,np_,nz", [(64, 64, 16), (96, 60, 30), (64, 64, 2), (40, 16, 1)])
def test_advection_equals_its_operations(nr, np_, nz):
    from mlegs_gb300.kit import Kit
    k = Kit(make_params(nr=nr, np=np_, nz=nz, nrchop=nr, npchop=np_ // 2 + 1, nzchop=nz // 2 + 1 if nz > 1 else 1, ell=4.0))
    try:
        zero = np.zeros(k.dims, complex, order="F")
        e = [fields.spectral_noise(k.params, k.dims, 21 + i, amp=1.0, decay=0.5) for i in range(2)]
        psi, chi = (k.scalar(v, 0.1, "FFF") for v in e)
        nl = [k.scalar(zero, 0.0, "FFF") for _ in range(2)]
        k.advection_rhs(psi, chi, *nl, k.scalar(zero, 0.0, "PPP"))
        psi, chi = (k.scalar(v, 0.1, "FFF") for v in e)
        k.dealias(psi)
        k.dealias(chi)
        v, w = ([k.scalar(zero, 0.0, "PPP") for _ in range(3)] for _ in range(2))
        k.tp2vec(psi, chi, *v)
        k.tp2curlvec(psi, chi, *w)
        k.vecprod(*v, *w)
        one = [k.scalar(zero, 0.0, "FFF") for _ in range(2)]
        k.vec2tp(*v, *one)
        for a, b in zip(nl, one):
            k.dealias(b)
            assert np.any(b.e != 0)
            assert np.array_equal(a.e, b.e)
    finally:
        k.close()
