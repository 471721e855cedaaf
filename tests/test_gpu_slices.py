"""The plain form's radial contractions at the edges of the exact-slice kernel: digit counts (8 digits up to 128 terms,
9 up to 372, FP64 beyond), row tiles, ragged z tiles and column values at the edge of the fixed-point scale, against the
same sums over the kit's own table in extended precision."""
import numpy as np
import pytest

from mlegs_gb300.params import make_params

pytestmark = pytest.mark.gpu

# The drop-in's bar (relative L2): far above the kernel's truncation (2^-61 of the largest table entry times the
# largest value of a column) and far below any lost digit (2^-49 or more).
TOL = 1e-12


def edge_values(rng, shape):
    """+-(2 - 2^-u), u = 1..52: magnitudes with long runs of ones below the leading bit."""
    return (2.0 - 2.0 ** -rng.integers(1, 53, shape)) * rng.choice([-1.0, 1.0], shape)


@pytest.mark.parametrize("nr,nrchop,nz", [(30, 30, 1), (62, 60, 18), (192, 192, 8), (254, 254, 18), (256, 256, 16),
                                          (258, 258, 18), (320, 200, 10), (512, 512, 18), (744, 744, 2), (746, 746, 2)])
def test_radial_contractions_at_the_digit_edges(nr, nrchop, nz):
    from mlegs_gb300.kit import Kit
    p = make_params(nr=nr, np=8, nz=nz, nrchop=nrchop, npchop=5, nzchop=nz // 2 + 1 if nz > 1 else 1, ell=4.0)
    k = Kit(p)
    try:
        pf = k.kit_get("pf").astype(np.longdouble)          # (nr/2, rows, m)
        w = k.kit_get("w").astype(np.longdouble)
        h = nr // 2
        rng = np.random.default_rng(nr + nz)
        for kind in ("normal", "edge", "graded"):
            def values(shape):
                if kind == "edge":
                    return edge_values(rng, shape) + 1j * edge_values(rng, shape)
                v = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
                return v * np.exp(-0.2 * np.arange(shape[0]))[:, None, None] if kind == "graded" else v

            # backward: FFP -> PFP
            c = np.zeros(k.dims, complex, order="F")
            c[:nrchop, :5] = values((nrchop, 5, k.dims[2]))
            for m in range(5):
                c[max(nrchop - m, 0):, m] = 0
            s = k.scalar(c, 0.0, "FFP")
            k.trans(s, "PFP")
            got = s.e
            ref = np.zeros(k.dims, np.clongdouble)
            for m in range(5):
                nn = nrchop - m
                e, o = (pf[:, q:nn:2, m] @ c[q:nn:2, m].astype(np.clongdouble) for q in (0, 1))
                ref[:h, m], ref[h:nr, m] = e + o, (e - o)[::-1]
            for m in range(5):
                err = np.linalg.norm((got[:, m] - ref[:, m]).astype(complex)) / np.linalg.norm(ref[:, m].astype(complex))
                assert err <= TOL, (kind, "backward", m, err)
            assert np.all(got[nr:] == 0)
            # forward: PFP -> FFP
            f = np.zeros(k.dims, complex, order="F")
            f[:nr, :5] = values((nr, 5, k.dims[2]))
            s.set(f, 0.0, "PFP")
            k.trans(s, "FFP")
            got = s.e
            for m in range(5):
                nn = nrchop - m
                a, b = f[:h, m].astype(np.clongdouble), f[h:nr, m][::-1].astype(np.clongdouble)
                want = np.zeros((nn, k.dims[2]), np.clongdouble)
                want[0::2] = (pf[:, 0:nn:2, m] * w[:h, None]).T @ (a + b)
                want[1::2] = (pf[:, 1:nn:2, m] * w[:h, None]).T @ (a - b)
                err = np.linalg.norm((got[:nn, m] - want).astype(complex)) / np.linalg.norm(want.astype(complex))
                assert err <= TOL, (kind, "forward", m, err)
                assert np.all(got[nn:, m] == 0)
            s.free()
    finally:
        k.close()


@pytest.mark.parametrize("nr,nrchop,nz", [(30, 30, 2), (126, 120, 18), (250, 250, 8), (258, 254, 6), (376, 376, 4)])
def test_plain_projection_at_the_tile_edges(nr, nrchop, nz):
    """vec2tp in the plain form (nine balanced digits; two row tiles past 253 rows; ragged z tiles) against the oracle.
    psi: the drop-in's bar.  chi ends in the inverse Laplacian, whose condition (about 1e4 here, for the columns other
    than (m, k) = (0, 0)) multiplies the last bit: 1e-11; the (0, 0) column, which runs in FP64 on its own path, is
    conditioned worse and is left to the kits of the parity tests."""
    from mlegs_gb300 import fields
    from mlegs_gb300.kit import Kit
    from oracle.oracle import Oracle
    p = make_params(nr=nr, np=8, nz=nz, nrchop=nrchop, npchop=5, nzchop=nz // 2 + 1, ell=4.0)
    o, k = Oracle(p), Kit(p)
    try:
        pair = []
        for kit in (k, o):
            psi = kit.scalar(fields.spectral_noise(p, k.dims, 5, amp=1.0, decay=0.3), 0.0, "FFF")
            chi = kit.scalar(fields.spectral_noise(p, k.dims, 6, amp=1.0, decay=0.3), 0.0, "FFF")
            if kit is k:   # one velocity for both: the oracle's
                pair.append((psi, chi))
                continue
            v = [kit.scalar(np.zeros(k.dims, complex), 0.0, "PPP") for _ in range(3)]
            kit.tp2vec(psi, chi, *v)
            kit.vec2tp(*v, psi, chi)
            pair.append((psi, chi))
        gv = [k.scalar(s.e, 0.0, "PPP") for s in v]
        k.vec2tp(*gv, *pair[0])
        for i, tol in ((0, TOL), (1, 10 * TOL)):
            g, c = pair[0][i].e, pair[1][i].e
            if i == 1:
                g, c = g.copy(), c.copy()
                g[:, 0, 0] = c[:, 0, 0] = 0
            err = np.linalg.norm(g - c) / np.linalg.norm(c)
            assert err <= tol, (i, err)
    finally:
        k.close()
        o.close()
