"""The plain form's radial transforms entry by entry, at sizes beyond 284 points: every output is as near to the exact sum as an
FP64 sum of the same terms, also where a row's large table entries meet small coefficients (points near the axis and far out,
where the functions of high m vanish)."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def near(got, terms, what):
    """got (real) against sum(terms, axis 0) in extended precision.  The K additions of an FP64 sum round by 2^-53 / sqrt(3) of S =
    sum |terms| each in the root mean square at most; five times their sum over the entries: 3 sqrt(K) 2^-53 S."""
    a, b = terms          # (rows, K) table and (K, columns) data
    ref, s = a @ b, np.abs(a) @ np.abs(b)
    err = np.abs(got.astype(np.longdouble) - ref)
    bad = err > 3 * np.sqrt(a.shape[1]) * U * s
    assert not bad.any(), (what, float((err / np.where(s > 0, s, 1)).max() / U), int(bad.sum()))


def parts(z):
    return np.concatenate([np.asarray(z).real, np.asarray(z).imag], axis=-1).astype(np.longdouble)


@pytest.mark.parametrize("nr,nrchop", [(288, 288), (320, 200), (512, 512), (744, 600)])
@pytest.mark.parametrize("kind", ["steep", "mild", "spike", "white"])
def test_radial_entries(nr, nrchop, kind):
    from mlegs_gb300.kit import Kit
    mc, nz = 41, 2
    k = Kit(make_params(nr=nr, np=80, nz=nz, nrchop=nrchop, npchop=mc, nzchop=2, ell=4.0))
    try:
        pf, w, r = k.kit_get("pf").astype(np.longdouble), k.kit_get("w").astype(np.longdouble), k.kit_get("r")
        h = nr // 2
        rng = np.random.default_rng(nr + len(kind))
        some = (1, 2, 4, 13, 27, 40)
        c = np.zeros(k.dims, complex, order="F")
        f = np.zeros(k.dims, complex, order="F")
        for m in some:
            nn = nrchop - m
            n = np.arange(nn)
            ph = np.exp(2j * np.pi * rng.random((nn, nz)))
            size = {"steep": np.exp(-1.0 * n), "mild": np.exp(-0.05 * n), "spike": np.where(n == 3, 1.0, 1e-9), "white": 1.0 + 0 * n}
            c[:nn, m] = size[kind][:, None] * ph
            size = {"steep": np.exp(-r[:nr] ** 2), "mild": (r[:nr] / (1 + r[:nr])) ** m, "spike": np.where(np.arange(nr) == 5, 1.0, 1e-9),
                    "white": 1.0 + 0 * r[:nr]}
            f[:nr, m] = size[kind][:, None] * np.exp(2j * np.pi * rng.random((nr, nz)))
        s = k.scalar(c, 0.0, "FFP")
        k.trans(s, "PFP")
        got = s.e
        for m in some:
            nn = nrchop - m
            a = np.concatenate([np.concatenate([pf[:, 0:nn:2, m], sg * pf[:, 1:nn:2, m]], axis=1) for sg in (1, -1)])
            b = np.concatenate([c[0:nn:2, m], c[1:nn:2, m]])
            near(parts(np.concatenate([got[:h, m], got[h:nr, m][::-1]])), (a, parts(b)), (kind, "backward", m))
        s.set(f, 0.0, "PFP")
        k.trans(s, "FFP")
        got = s.e
        for m in some:
            nn = nrchop - m
            for par in (0, 1):
                a = pf[:, par:nn:2, m].T * w[:h]
                b = parts(f[:h, m]) + (1 - 2 * par) * parts(f[h:nr, m][::-1])
                near(parts(got[par:nn:2, m]), (a, b), (kind, "forward", m, par))
        s.free()
    finally:
        k.close()
