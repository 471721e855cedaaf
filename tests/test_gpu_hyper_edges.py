"""The powered Helmholtz solve at the edges of its row batches (four or two rows) and its bands, two calls in a row (factored,
then from the kept factors), against the oracle to 1e-10 of the field's norm, the tolerance of the solves with a dominant
diagonal elsewhere in the suite."""
import numpy as np
import pytest

from helpers import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [4, 6, 8])
@pytest.mark.parametrize("nrchop", [3, 5, 8, 9, 10, 12, 13, 16, 17, 24])
def test_ihelmp_rows(nrchop, power):
    from mlegs_gb300.kit import Kit
    from mlegs_gb300.params import make_params
    from oracle.oracle import Oracle

    p = make_params(nr=24, np=8, nz=6, nrchop=nrchop, npchop=3, nzchop=4, visc=1e-3, hyperpow=power, hypervisc=1e-6)
    k, o = Kit(p), Oracle(p)
    try:
        rng = np.random.default_rng(nrchop)
        e = np.zeros(k.dims, complex, order="F")
        for m in range(3):
            n = max(nrchop - m, 0)
            e[:n, m] = rng.standard_normal((n, k.dims[2])) + 1j * rng.standard_normal((n, k.dims[2]))
        sign = 1.0 if power == 6 else -1.0     # of alpha, that of D^(power/2)'s dominant part
        for call in range(2):
            g, r = k.scalar(e, 0.3, "FFF"), o.scalar(e, 0.3, "FFF")
            alpha, beta = -sign * 1e12, 10.0
            k.ihelmp(g, power, alpha, beta)
            o.ihelmp(r, power, alpha, beta)
            compare(g, r, 1e-10, what=f"{nrchop} rows, power {power}, call {call}")
            g.free()
    finally:
        k.close()
        o.close()
