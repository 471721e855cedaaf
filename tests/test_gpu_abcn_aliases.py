"""abcn with one field in two of its places: the assignments at its end come in the reference's order, s_p = s and then
nl_p = nl (mlegs_scalar_ops.f90:1200-1262), and a call that is refused for its alpha leaves nl_p as it was."""
import numpy as np
import pytest

from mlegs_gb300 import fields
from helpers import params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kit():
    from mlegs_gb300.kit import Kit
    k = Kit(params("odd"))
    yield k
    k.close()


def four(k):
    """s, s_p, nl, nl_p with their own values and log terms."""
    return [k.scalar(fields.spectral_noise(k.params, k.dims, 11 + i, amp=1.0, decay=0.1), 0.1 * (i + 1), "FFF") for i in range(4)]


def value(s):
    e, ln, _, _ = s.get()
    return e.copy(), ln


def same(s, want):
    e, ln = value(s)
    assert np.array_equal(e, want[0]) and ln == want[1]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("who", ["s_p is nl_p", "s_p is nl", "nl is nl_p", "s_p is s", "nl is s", "nl_p is s"])
def test_a_field_in_two_places(kit, mixed, who):
    from mlegs_gb300.kit import MIXED, PLAIN_FP64
    kit.set_precision(MIXED if mixed else PLAIN_FP64)
    names = ("s", "s_p", "nl", "nl_p")
    one, other = who.split(" is ")
    dt = 1e-3
    # four fields of their own, with the values that the aliased call sees
    f = dict(zip(names, four(kit)))
    f[one].copy_from(f[other])
    kit.abcn(*(f[n] for n in names), dt)
    s = value(f["s"])
    g = dict(zip(names, four(kit)))
    g[one] = g[other]
    before = {n: value(v) for n, v in g.items()}
    kit.abcn(*(g[n] for n in names), dt)
    # the reference's order of assignments on the aliased fields
    slot = {n: (other if n == one else n) for n in names}
    val = {slot[n]: before[n] for n in names}
    val[slot["s"]] = s
    val[slot["s_p"]] = val[slot["s"]]
    val[slot["nl_p"]] = val[slot["nl"]]
    for n in names:
        same(g[n], val[slot[n]])
    kit.set_precision(PLAIN_FP64)


def test_refused_alpha_leaves_nl_p(kit):
    from mlegs_gb300.kit import MlgError
    s, s_p, nl, nl_p = four(kit)
    before = value(nl_p), value(s_p)
    with pytest.raises(MlgError, match="alpha equals to zero"):
        kit.abcn(s, s_p, nl, nl_p, 1e20)
    same(nl_p, before[0])
    same(s_p, before[1])
