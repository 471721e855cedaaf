"""The plain form where the device has no room for the slices' tables: its FP64 kernels take the contractions, as they do for
grids that the slices do not cover."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu

LEFT = 256 << 20   # bytes left on the device; the tables of this grid's projection take 400 MB


def velocities(k):
    rng = np.random.default_rng(3)
    out = []
    for _ in range(3):
        e = np.zeros(k.dims, complex, order="F")
        e[:512, :32] = rng.standard_normal((512, 32, 4)) + 1j * rng.standard_normal((512, 32, 4))
        out.append(k.scalar(e, 0.0, "PPP"))
    return out


def test_without_room_for_the_tables():
    torch = pytest.importorskip("torch")
    from mlegs_gb300.kit import Kit
    p = make_params(nr=512, np=64, nz=4, nrchop=512, npchop=33, nzchop=3, ell=4.0)

    def projected(fill):
        k = Kit(p)
        held = None
        try:
            v = velocities(k)
            psi, chi = (k.scalar(np.zeros(k.dims, complex, order="F"), 0.0, "FFF") for _ in range(2))
            before = k.mem_bytes()
            if fill:
                free, _ = torch.cuda.mem_get_info()
                held = torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")
            k.vec2tp(*v, psi, chi)
            k.sync()
            return psi.e.copy(), k.mem_bytes() - before
        finally:
            del held
            torch.cuda.empty_cache()
            k.close()

    want, roomy = projected(False)
    got, tight = projected(True)
    assert roomy > LEFT > tight            # the tables were made, and could not be
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err < 1e-12, err                # the drop-in's bar
