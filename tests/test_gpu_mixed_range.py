"""The range of the mixed form's radial slices."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params
from test_gpu_radial_entries import near, parts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nrchop", [(742, 742), (800, 800), (894, 300)])
def test_mixed_form_beyond_its_slices(nr, nrchop):
    """Past 740 radial points (892 with six digits, up to 340 rows) the mixed form's backward sums are FP64."""
    from mlegs_gb300.kit import Kit, MIXED
    m, nn = 2, nrchop - 2
    k = Kit(make_params(nr=nr, np=8, nz=2, nrchop=nrchop, npchop=3, nzchop=2, ell=4.0), precision=MIXED)
    try:
        pf = k.kit_get("pf").astype(np.longdouble)
        rng = np.random.default_rng(8)
        c = np.zeros(k.dims, complex, order="F")
        c[:nn, m] = rng.standard_normal((nn, 2)) + 1j * rng.standard_normal((nn, 2))
        s = k.scalar(c, 0.0, "FFP")
        k.trans(s, "PFP")
        a = np.concatenate([np.concatenate([pf[:, 0:nn:2, m], sg * pf[:, 1:nn:2, m]], axis=1) for sg in (1, -1)])
        b = np.concatenate([c[0:nn:2, m], c[1:nn:2, m]])
        near(parts(np.concatenate([s.e[:nr // 2, m], s.e[nr // 2:nr, m][::-1]])), (a, parts(b)), nr)
    finally:
        k.close()
