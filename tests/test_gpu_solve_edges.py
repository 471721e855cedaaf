"""The banded substitution at the edges of its row batches (8 rows, 4 where rows are exchanged) and of its 16-system warps,
against the oracle.  Tolerance: that of the solves elsewhere in the suite, 1e-10 of the field's norm, and 1e-9 without a
dominant alpha (condition number about 1e4)."""
import numpy as np
import pytest

from helpers import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrchop", [3, 7, 8, 9, 12, 15, 16, 17, 24, 31, 32, 33, 47, 48])
@pytest.mark.parametrize("alpha,tol", [(-3.5e3, 1e-10), (-0.5, 1e-9)])
def test_ihelm_rows(nrchop, alpha, tol):
    from mlegs_gb300.kit import Kit
    from mlegs_gb300.params import make_params
    from oracle.oracle import Oracle

    p = make_params(nr=48, np=8, nz=6, nrchop=nrchop, npchop=3, nzchop=4)
    k, o = Kit(p), Oracle(p)
    try:
        rng = np.random.default_rng(nrchop)
        e = np.zeros(k.dims, complex, order="F")
        for m in range(3):
            n = max(nrchop - m, 0)
            e[:n, m] = rng.standard_normal((n, k.dims[2])) + 1j * rng.standard_normal((n, k.dims[2]))
        g, r = k.scalar(e, 0.3, "FFF"), o.scalar(e, 0.3, "FFF")
        k.ihelm(g, alpha)
        o.ihelm(r, alpha)
        compare(g, r, tol, what=f"{nrchop} rows, alpha {alpha}")
    finally:
        k.close()
        o.close()
