"""The workloads whose speed is followed from commit to commit.

Each case is one piece of work that a program built on this library has it do, through the public Python
front end (mlegs_gb300.kit), with fields that live on the GPU:

  transform   a spectral field to physical space and that field back again (trans, FFF -> PPP -> FFF)
  diffuse     steps of the advection-diffusion stepper of one scalar (abcn; with hyperviscosity where
              hyperpow is set)
  fields      velocity and vorticity of a toroidal/poloidal pair in physical space (tp2vec, tp2curlvec)
  advect      the nonlinear term of the vortex equations (advection_rhs)
  run         steps of the vortex equations (vortex_run)
  adjoint     a cost and its gradient over a horizon of steps (adjoint_run)

`exact` restates the same operations in 64 bits with torch alone, on dense matrices where the library
uses bands and slices.
"""
import math

import numpy as np
import torch

from mlegs_gb300.kit import Kit, MIXED, PLAIN_FP64, load
from mlegs_gb300.params import dims_of, make_params

PREC = {"plain": PLAIN_FP64, "mixed": MIXED}
KIT_KEYS = ("nr", "np", "nz", "nrchop", "npchop", "nzchop", "ell", "visc", "hyperpow", "hypervisc", "is_svv")


def _case(op, precision, shape, chops=None, **kw):
    nr, np_, nz = shape
    a, b, c = chops or (nr, np_ // 2 + 1, nz // 2 + 1 if nz > 1 else 1)
    d = dict(op=op, precision=precision, nr=nr, np=np_, nz=nz, nrchop=a, npchop=b, nzchop=c, ell=4.0, visc=1.0e-3,
             hyperpow=0, hypervisc=0.0, is_svv=0, steps=1, dt=1.0e-3)
    d.update(kw)
    return d


def listed():
    return [
        # the two-dimensional tutorial kit: the smallest transform pair, all of it latency
        dict(_case("transform", "plain", (32, 48, 1), ell=1.0), name="transform_2d"),
        # the small three-dimensional grid of the tests: scalar diffusion steps
        dict(_case("diffuse", "plain", (32, 32, 32), steps=4), name="diffuse_32"),
        # factors of 3 and 5 in both FFTs and truncations short of the full ones
        dict(_case("transform", "plain", (160, 120, 96), (144, 41, 33), ell=2.0), name="transform_ragged"),
        # the cube on which transforms are compared, in both precision forms
        dict(_case("transform", "plain", (256, 256, 256)), name="transform_256"),
        dict(_case("transform", "mixed", (256, 256, 256)), name="transform_256_mixed"),
        # the default grid: one nonlinear term
        dict(_case("advect", "plain", (256, 128, 128)), name="advect_256x128x128"),
        # a small ragged vortex run in the mixed form
        dict(_case("run", "mixed", (96, 120, 90), (96, 41, 31), steps=10, dt=2.0e-4, is_svv=1), name="run_ragged_mixed"),
        # the vortex run that the library is quoted on, in both precision forms
        dict(_case("run", "mixed", (192, 128, 128), steps=10, dt=2.0e-4, visc=1.0e-4, is_svv=1), name="run_192_mixed"),
        dict(_case("run", "plain", (192, 128, 128), steps=4, dt=2.0e-4, visc=1.0e-4, is_svv=1), name="run_192"),
        # gradient of the perturbation energy over a horizon
        dict(_case("adjoint", "plain", (40, 64, 64), steps=10, dt=2.0e-3, ckpt=5), name="adjoint_40"),
        # the large grid: physical fields of a state, as written out or fed to diagnostics, in the plain form, and
        # steps in the mixed form
        dict(_case("fields", "plain", (512, 512, 256), ell=6.0, visc=5.0e-5), name="fields_512"),
        dict(_case("run", "mixed", (512, 512, 256), ell=6.0, steps=2, dt=2.0e-4, visc=5.0e-5, is_svv=1), name="run_512_mixed"),
    ]


def _size(rng, lo, hi, ok):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while not ok(v):
        v = v + 1 if v < hi else lo
    return v


def _fft_size(v):
    if v % 2:
        return False
    for p in (2, 3, 5):
        while v % p == 0:
            v //= p
    return v == 1


# points of the grid times steps that keep a drawn case within the largest listed one, by operation and form
MOST = {("transform", "plain"): 67e6, ("transform", "mixed"): 67e6, ("diffuse", "plain"): 67e6, ("diffuse", "mixed"): 67e6,
        ("fields", "plain"): 33e6, ("fields", "mixed"): 67e6, ("advect", "plain"): 17e6, ("advect", "mixed"): 33e6,
        ("run", "plain"): 20e6, ("run", "mixed"): 60e6, ("adjoint", "plain"): 5e6, ("adjoint", "mixed"): 5e6}
# radial points up to which nonlinear terms and gradients are drawn: beyond, the inverse Laplacian of the (m, k) =
# (0, 0) column (and its transpose, in the gradient) magnifies the last bit of 64-bit arithmetic a millionfold and
# more, and two right answers differ visibly there; gradients in the plain form for the same reason
MOST_NR = {"advect": 256, "run": 256, "adjoint": 48}


def draw(rng):
    """One more case of the listed ranges: grids of 24 to 512 radial points (see MOST_NR), powers of two and products of 2, 3
    and 5 along the periodic directions, full and short truncations, both forms."""
    op = rng.choice(("transform", "transform", "diffuse", "fields", "advect", "run", "run", "adjoint"))
    precision = rng.choice(("plain", "mixed")) if op != "adjoint" else "plain"
    steps = {"run": rng.randint(2, 10), "diffuse": rng.randint(1, 4), "adjoint": rng.choice((4, 8))}.get(op, 1)
    flat = op in ("transform", "diffuse") and rng.random() < 0.2
    pow2 = rng.random() < 0.5
    fft_ok = (lambda v: v >= 4 and v & (v - 1) == 0) if pow2 else _fft_size
    while True:
        nr = _size(rng, 24, MOST_NR.get(op, 512), lambda v: v % 2 == 0)
        np_ = _size(rng, 16, 512, fft_ok)
        nz = 1 if flat else _size(rng, 12, 256, fft_ok)
        if nr * np_ * nz * steps <= MOST[op, precision]:
            break
    chops = None
    if rng.random() < 0.4:
        chops = (nr - 2 * rng.randint(0, nr // 8), max(4, np_ // 3 + 1), max(2, nz // 3 + 1) if nz > 1 else 1)
    kw = {}
    if op == "run":
        kw = dict(dt=2.0e-4, is_svv=rng.randint(0, 1))
    elif op == "adjoint":
        kw = dict(dt=1.0e-3, ckpt=steps // 2)
    elif op == "diffuse" and rng.random() < 0.3:
        kw = dict(hyperpow=4, hypervisc=1.0e-6)
    return _case(op, precision, (nr, np_, nz), chops, ell=rng.choice((1.0, 2.0, 4.0, 6.0)), steps=steps, **kw)


# ---------------------------------------------------------------------------------------------------
# inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _params(c):
    return make_params(**{k: c[k] for k in KIT_KEYS})


def _nodes(c):
    x, w = np.polynomial.legendre.leggauss(c["nr"])
    return x, w, c["ell"] * np.sqrt((1.0 + x) / (1.0 - x))


def _active(c, offset=0):
    """The coefficients (k, m, n) that the truncation keeps, as a mask in a field's own order."""
    nrdim, npdim, nzdim = dims_of(_params(c))
    dev = _device()
    k, m, n = (torch.arange(s, device=dev) for s in (nzdim, npdim, nrdim))
    m, n = m[:, None], n[None, :]
    rows = (n < c["nrchop"] + offset - m) & (m < c["npchop"])
    kept = (k + 1 <= c["nzchop"]) | (k + 1 >= c["nz"] - c["nzchop"] + 2)
    return kept[:, None, None] & rows[None]


def _noise(c, seed, amp, decay, m_max=None, k_max=None):
    """Seeded coefficients amp exp(-decay (n + |m| + |k|)) with random phases on the kept modes, of a real field."""
    nrdim, npdim, nzdim = dims_of(_params(c))
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) % (1 << 62))
    k = torch.arange(nzdim, device=dev, dtype=torch.float64)
    k = torch.minimum(k, nzdim - k)[:, None, None]
    m = torch.arange(npdim, device=dev, dtype=torch.float64)[None, :, None]
    n = torch.arange(nrdim, device=dev, dtype=torch.float64)[None, None, :]
    ph = torch.rand((nzdim, npdim, nrdim), generator=g, device=dev, dtype=torch.float64) * (2 * math.pi)
    e = torch.polar((amp * torch.exp(-decay * (n + m + k))), ph)
    keep = _active(c)
    if m_max is not None:
        keep = keep & (m <= m_max) & (k <= k_max)
    e = torch.where(keep, e, torch.zeros((), dtype=e.dtype, device=dev))
    for mm in (0, npdim - 1):   # conjugate symmetric in k: the field is real
        p = e[:, mm]
        e[:, mm] = 0.5 * (p + torch.roll(p.flip(0), 1, 0).conj())
    return e


def _axis_column(c, source):
    """The (m, k) = (0, 0) column and the log term of the field whose horizontal Laplacian times (1 - x)^2 is
    `source` at the radial points: Legendre analysis, inversion of n (n + 1), and zero at infinity."""
    x, w, _ = _nodes(c)
    nn = c["nrchop"]

    def table(at):
        p = np.zeros((nn, len(at)))
        p[0] = math.sqrt(0.5)
        if nn > 1:
            p[1] = math.sqrt(1.5) * at
        for n in range(2, nn):
            a, b = math.sqrt((4.0 * n * n - 1) / (n * n)), math.sqrt((4.0 * (n - 1) ** 2 - 1) / ((n - 1) ** 2))
            p[n] = a * (at * p[n - 1] - p[n - 2] / b)
        return p

    col = table(x) @ (w * source)
    n = np.arange(nn)
    ln = col[0] * c["ell"] ** 2 * math.sqrt(0.5)
    col[1:] = -col[1:] / n[1:] / (n[1:] + 1) * c["ell"] ** 2
    col[0] = 0.0
    at1 = table(np.array([1.0 - 1.0e-15]))[:, 0]
    col[0] -= (col @ at1) / at1[0]
    return col, float(ln)


def _vortex(c, seed):
    """psi, chi and their log terms: a Batchelor vortex on the axis and a seeded perturbation."""
    x, _, r = _nodes(c)
    out = []
    for i, f in enumerate((2.0, 0.25)):
        col, ln = _axis_column(c, -f * np.exp(-r ** 2) / (1.0 - x) ** 2)
        e = _noise(c, 2 * seed + i, 1.0e-2, 1.0, 4, 8)
        e[0, 0, : len(col)] += torch.from_numpy(col).to(e.device)
        out.append((e, ln))
    return out


def _inputs(c, seed):
    """The fields of a case by name: (coefficients, log term)."""
    if c["op"] == "transform":
        return {"spectral": (_noise(c, seed, 1.0, 0.05), 0.0)}
    if c["op"] == "diffuse":
        return {n: (_noise(c, 4 * seed + i, a, 0.1), 0.0)
                for i, (n, a) in enumerate((("s", 1.0), ("s_p", 1.0), ("nl", 0.1), ("nl_p", 0.1)))}
    psi, chi = _vortex(c, seed)
    d = {"psi": psi, "chi": chi}
    if c["op"] == "run":
        for i, n in enumerate(("nlpsi", "nlchi", "nlpsi_p", "nlchi_p")):
            d[n] = (_noise(c, 7 * seed + 3 + i, 1.0e-2, 1.0, 4, 8), 0.0)
        d["psi_p"], d["chi_p"] = psi, chi
    return d


# ---------------------------------------------------------------------------------------------------
# the programs
_kit = {"key": None, "kit": None}


def _get_kit(c):
    """The process's one transform kit, made again when another grid is asked for."""
    key = tuple(c[k] for k in KIT_KEYS)
    if _kit["key"] != key:
        if _kit["kit"] is not None:
            _kit["kit"].close()
        _kit["key"], _kit["kit"] = key, Kit(_params(c))
    _kit["kit"].set_precision(PREC[c["precision"]])
    return _kit["kit"]


class _DeviceArray:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<c16", "version": 3}


class Program:
    """The library's fields of one case, as a program keeps them."""

    def __init__(self, c):
        self.c, self.kit, self.fields, self.views = c, _get_kit(c), {}, {}

    def add(self, name, e=None, ln=0.0, space="FFF"):
        s = self.fields[name] = self.kit.scalar()
        if e is None:
            load().mlg_scalar_set_space(s.h, space.encode())
        else:
            load().mlg_scalar_upload_device(s.h, e.data_ptr(), float(ln), space.encode())
            torch.cuda.current_stream().synchronize()   # e may go when this returns
        return s

    def out(self, *names):
        """The named fields' device memory as tensors (k, m, n); a field's buffer may change from call to call."""
        got = []
        for n in names:
            ptr = self.fields[n].device_ptr()
            if ptr not in self.views:
                self.views[ptr] = torch.as_tensor(_DeviceArray(ptr, self.kit.dims[::-1]), device="cuda")
            got.append(self.views[ptr])
        return got

    def __del__(self):
        if _kit["kit"] is self.kit:   # fields of a kit that is closed went with it
            for s in self.fields.values():
                s.free()


RUN_FIELDS = ("psi", "chi", "nlpsi", "nlchi", "psi_p", "chi_p", "nlpsi_p", "nlchi_p")
VECTORS = ("vr", "vp", "vz", "wr", "wp", "wz")


def prepare(case, seed):
    p = Program(dict(case))
    for n, (e, ln) in _inputs(p.c, int(seed)).items():
        p.add(n, e, ln)
    op = p.c["op"]
    if op == "transform":
        p.add("physical")
        p.add("back")
    elif op == "fields":
        for n in VECTORS:
            p.add(n, space="PPP")
    elif op == "advect":
        p.add("nlpsi")
        p.add("nlchi")
    elif op == "adjoint":
        p.add("grad_psi")
        p.add("grad_chi")
    if op in ("advect", "run", "adjoint"):
        p.add("uz", space="PPP")
    p.gains = [0.0, 0.0]
    return p


def run(p):
    c, k, f = p.c, p.kit, p.fields
    k.set_precision(PREC[c["precision"]])
    if c["op"] == "transform":
        f["physical"].copy_from(f["spectral"])
        k.trans(f["physical"], "PPP")
        f["back"].copy_from(f["physical"])
        k.trans(f["back"], "FFF")
        return p.out("physical", "back")
    if c["op"] == "diffuse":
        for _ in range(c["steps"]):
            k.abcn(f["s"], f["s_p"], f["nl"], f["nl_p"], c["dt"])
        return p.out("s", "s_p", "nl_p")
    if c["op"] == "fields":
        k.tp2vec(f["psi"], f["chi"], *(f[n] for n in VECTORS[:3]))
        k.tp2curlvec(f["psi"], f["chi"], *(f[n] for n in VECTORS[3:]))
        return p.out(*VECTORS)
    if c["op"] == "advect":
        k.advection_rhs(f["psi"], f["chi"], f["nlpsi"], f["nlchi"], f["uz"])
        return p.out("nlpsi", "nlchi")
    if c["op"] == "run":
        k.vortex_run(*(f[n] for n in RUN_FIELDS), f["uz"], c["dt"], c["steps"], p.gains)
        return p.out(*RUN_FIELDS), list(p.gains)
    cost = k.adjoint_run(f["psi"], f["chi"], f["uz"], c["dt"], c["steps"], c["ckpt"], f["grad_psi"], f["grad_chi"])
    return p.out("grad_psi", "grad_chi"), cost


def work(case):
    """Bytes: each field of a pass read once and written once (of a run or a horizon, once for each step: the
    fields of a step pass through memory).  Flops: the radial contractions over the kept rows and the FFTs."""
    c = dict(case)
    nrdim, npdim, nzdim = dims_of(_params(c))
    field = 16.0 * nrdim * npdim * nzdim
    rows = sum(max(c["nrchop"] - m, 0) for m in range(c["npchop"]))
    radial = 4.0 * rows * (c["nr"] // 2) * nzdim
    fft = 5.0 * nrdim * (npdim * nzdim * math.log2(max(nzdim, 2)) + nzdim * (npdim - 1) * math.log2(max(c["np"], 2)))
    band = 60.0 * nrdim * npdim * nzdim
    nl = 13 * radial + 11 * fft + 4 * band
    fields, flops = {
        "transform": (3, 2 * (radial + fft)),
        "diffuse": (7 * c["steps"], 2 * band * c["steps"]),
        "fields": (8, 6 * (radial + fft) + 4 * band),
        "advect": (4, nl),
        "run": (10 * c["steps"], (nl + 4 * band) * c["steps"]),
        "adjoint": (24 * c["steps"], 4 * (nl + 4 * band) * c["steps"]),
    }[c["op"]]
    return {"bytes": fields * field, "flops": flops}


# ---------------------------------------------------------------------------------------------------
# the same operations in 64 bits, with torch alone
def _complex(v):
    return torch.complex(v[..., 0], v[..., 1])


class Exact:
    """Fields are (k, m, n) tensors with a log term beside them; the radial table is dense, the banded solves are
    dense LU factorisations."""

    def __init__(self, c):
        self.c, self.dev = c, _device()
        self.nrdim, self.npdim, self.nzdim = dims_of(_params(c))
        x, w, r = _nodes(c)
        self.x, self.w, self.r = (torch.from_numpy(v).to(self.dev) for v in (x, w, r))
        self.lnx = -torch.log(1.0 - self.x)
        self.rows = c["nrchop"] + 4
        ells = np.arange(self.nzdim)
        self.ak = torch.from_numpy(2 * math.pi / (2 * math.pi) * np.where(ells <= self.nzdim // 2, ells, ells - self.nzdim).astype(float)).to(self.dev)
        self.pf = self.table(self.x)                                   # (m, n, i)
        self.at1 = self.table(torch.tensor([1.0 - 1.0e-15], dtype=torch.float64, device=self.dev), 1)[0, : c["nrchop"], 0]
        m = np.arange(c["npchop"])[:, None].astype(float)
        n = m + np.arange(self.rows)[None, :]
        # log of the normalisation of row n: half of log (n + 1/2) + log (n - m)! - log (n + m)!
        lf = np.array([math.lgamma(v + 1.0) for v in range(int(n.max()) + c["npchop"] + 2)])
        norm = 0.5 * (np.log(n + 0.5) + lf[(n - m).astype(int)] - lf[(n + m).astype(int)])
        self.norm0 = np.exp(norm[0])

        def band(cols):
            b = np.zeros((c["npchop"], self.rows, len(cols)))
            h = len(cols) // 2
            for q, v in enumerate(cols):
                d = q - h
                lo, hi = max(0, -d), self.rows - max(0, d)
                b[:, lo:hi, q] = v[:, lo:hi] * np.exp(norm[:, lo + d:hi + d] - norm[:, lo:hi])
            return torch.from_numpy(b).to(self.dev)

        with np.errstate(divide="ignore", invalid="ignore"):
            self.bd2 = band([-(n - m - 1) * (n - m) * (n - 2) * (n - 1) / (2 * n - 3) / (2 * n - 1),
                             2 * n * (n - m) * (n - 1) / (2 * n - 1),
                             -2 * n * (n + 1) * (3 * n * n + 3 * n - m * m - 2) / (2 * n - 1) / (2 * n + 3),
                             2 * (n + 1) * (n + m + 1) * (n + 2) / (2 * n + 3),
                             -(n + m + 1) * (n + m + 2) * (n + 3) * (n + 2) / (2 * n + 3) / (2 * n + 5)]) / c["ell"] ** 2
            self.bxx = band([-(n - 1) * (n - m) / (2 * n - 1), 0 * n, (n + 2) * (n + m + 1) / (2 * n + 3)])
        self.lu = {}

    def table(self, x, modes=None):
        """Orthonormal associated Legendre functions (m, n - m, x), Condon-Shortley phase, by the stable recurrence."""
        modes = modes or self.c["npchop"]
        t = torch.zeros((modes, self.rows, len(x)), dtype=torch.float64, device=self.dev)
        m = torch.arange(modes, device=self.dev, dtype=torch.float64)[:, None]
        sec = torch.full((len(x),), math.sqrt(0.5), dtype=torch.float64, device=self.dev)
        for q in range(modes):
            t[q, 0] = sec
            sec = -sec * math.sqrt((2 * q + 3.0) / (2 * q + 2.0)) * torch.sqrt((1 - x) * (1 + x))
        for j in range(1, self.rows):
            n = m + j
            a = torch.sqrt((4 * n * n - 1) / (n * n - m * m))
            t[:, j] = a * x * t[:, j - 1]
            if j > 1:
                t[:, j] -= a / torch.sqrt((4 * (n - 1) ** 2 - 1) / ((n - 1) ** 2 - m * m)) * t[:, j - 2]
        return t

    def zeros(self):
        return torch.zeros((self.nzdim, self.npdim, self.nrdim), dtype=torch.complex128, device=self.dev)

    def nn(self, m, offset=0):
        return max(min(self.c["nrchop"] + offset - m, self.rows), 0)

    def kept(self):
        """Slots k in the order that the banded operators visit them, the shared Nyquist slot twice."""
        lo, hi = self.c["nzchop"], self.c["nz"] - self.c["nzchop"] + 2
        first = torch.arange(self.nzdim, device=self.dev)
        return first[first + 1 <= lo], first[first + 1 >= max(hi, 1)]

    # -- transforms
    def phi(self, e, sign):
        h = self.c["np"] // 2
        if sign < 0:
            f = torch.view_as_real(e[:, :h]).permute(0, 1, 3, 2).reshape(self.nzdim, 2 * h, self.nrdim)
            return torch.fft.rfft(f, dim=1) / (2 * h)
        a = e.clone()
        a[:, 0].imag.zero_()
        a[:, h].imag.zero_()
        f = torch.fft.irfft(a, n=2 * h, dim=1) * (2 * h)
        out = torch.empty_like(e)
        out[:, :h] = _complex(f.reshape(self.nzdim, h, 2, self.nrdim).permute(0, 1, 3, 2))
        out[:, h] = e[:, h] * (2 * h)
        return out

    def z(self, e, sign):
        if self.c["nz"] == 1:
            return e
        return torch.fft.fft(e, dim=0) / self.nzdim if sign < 0 else torch.fft.ifft(e, dim=0) * self.nzdim

    def radial(self, e, sign):
        out, nr = self.zeros(), self.c["nr"]
        for m in range(self.c["npchop"]):
            nn = self.nn(m)
            if nn < 1:
                continue
            t = self.pf[m, :nn]
            if sign < 0:
                f = torch.view_as_real(e[:, m, :nr] * self.w).permute(0, 2, 1)
                out[:, m, :nn] = _complex((f @ t.T).permute(0, 2, 1))
            else:
                f = torch.view_as_real(e[:, m, :nn].contiguous()).permute(0, 2, 1)
                out[:, m, :nr] = _complex((f @ t).permute(0, 2, 1))
        return out

    def to_ppp(self, e, ln):
        e = self.radial(self.z(e, 1), 1)
        e[:, 0, : self.c["nr"]] += ln * self.lnx
        return self.phi(e, 1)

    def to_fff(self, e, ln):
        e = self.phi(e, -1)
        e[:, 0, : self.c["nr"]] -= ln * self.lnx
        return self.z(self.radial(e, -1), -1)

    # -- masks
    def chop(self, e):
        return torch.where(_active(self.c), e, torch.zeros_like(e))

    def dealias(self, e):
        e = e.clone()
        e[:, self.c["np"] // 3 + 1:] = 0
        if self.c["nz"] > 1:
            zc = self.c["nz"] // 3 + 1
            e[zc: self.c["nz"] - zc + 1] = 0
        return e

    def zeroat1(self, e):
        e = e.clone()
        a = (e[:, 0, : self.c["nrchop"]] * self.at1).sum(-1)
        e[:, 0, 0] -= a / self.at1[0]
        return e

    def svv(self, e, gain):
        p = _params(self.c)
        n = torch.arange(self.nrdim, device=self.dev, dtype=torch.float64)
        m = torch.arange(self.npdim, device=self.dev, dtype=torch.float64)
        q = torch.maximum(torch.maximum((n / max(self.c["nrchop"] - 1, 1)).clamp(max=1)[None, None, :],
                                        (m / max(self.c["np"] // 2, 1)).clamp(max=1)[None, :, None]),
                          (self.ak.abs() / max(float(self.ak.abs().max()), 1.0)).clamp(max=1)[:, None, None])
        a = torch.view_as_real(e).square().sum(-1)
        total, tail = float(a.sum()), float(a[q >= p.svv_cutoff].sum())
        if total <= 2.3e-308:
            return e, gain
        fb = min(max(tail / total / p.svv_target - 1.0, 0.0), 1.0)
        gain = (1 - p.svv_relax) * gain + p.svv_relax * fb
        s = min(p.svv_strength * gain, 1.0)
        if s <= 0:
            return e, gain
        f = torch.exp(-s * ((q - p.svv_cutoff) / (1 - p.svv_cutoff)).clamp(min=0) ** 8)
        return e * f, gain

    # -- banded operators
    def log_terms(self, ln, op):
        e2 = self.c["ell"] ** 2
        if op == "xx":
            t = [ln / self.norm0[0], ln / self.norm0[1]]
        else:
            t = [4 / 3 / e2 / self.norm0[0] * ln, -2 / e2 / self.norm0[1] * ln, 2 / 3 / e2 / self.norm0[2] * ln]
        return torch.tensor(t, dtype=torch.complex128, device=self.dev)

    def band(self, e, ln, op, offset=0):
        """xxdx ("xx"), del2h ("h") or del2 ("2"); the log term becomes coefficients."""
        out = e.clone()
        b = self.bxx if op == "xx" else self.bd2
        half = b.shape[2] // 2
        for m in range(self.c["npchop"]):
            nn = self.nn(m, offset)
            if nn < 1:
                continue
            for slots in self.kept():
                v = torch.zeros((len(slots), nn + 2 * half), dtype=e.dtype, device=self.dev)
                v[:, half: half + nn] = out[slots, m, :nn]
                y = sum(b[m, :nn, q] * v[:, q: q + nn] for q in range(2 * half + 1))
                if op == "2":
                    y = y - self.ak[slots][:, None] ** 2 * v[:, half: half + nn]
                out[slots, m, :nn] = y
        t = self.log_terms(ln, op)
        out[0, 0, : len(t)] += t
        return out

    def dense(self, m, nn, slots):
        a = torch.zeros((nn, nn), dtype=torch.float64, device=self.dev)
        for q in range(5):
            d = q - 2
            if nn > abs(d):
                a.diagonal(d).copy_(self.bd2[m, max(0, -d): nn - max(0, d), q])
        return a[None] - torch.diag_embed((self.ak[slots] ** 2)[:, None].expand(-1, nn))

    def solve(self, e, key, matrix):
        """The banded systems of every kept column, factored once for each key."""
        out = e.clone()
        for m in range(self.c["npchop"]):
            nn = self.nn(m)
            if nn < 1:
                continue
            for i, slots in enumerate(self.kept()):
                if not len(slots):
                    continue
                if (key, m, i) not in self.lu:
                    self.lu[key, m, i] = torch.linalg.lu_factor(matrix(m, nn, slots))
                v = torch.view_as_real(out[slots, m, :nn].contiguous())
                out[slots, m, :nn] = _complex(torch.linalg.lu_solve(*self.lu[key, m, i], v))
        return out

    def ihelm(self, e, ln, alpha):
        e, ln = e.clone(), ln / alpha
        e[0, 0, :3] -= self.log_terms(ln, "2")
        eye = lambda nn: torch.eye(nn, dtype=torch.float64, device=self.dev)  # noqa: E731
        return self.solve(e, ("h", alpha), lambda m, nn, s: self.dense(m, nn, s) + alpha * eye(nn)), ln

    def ihelmp(self, e, ln, power, alpha, beta):
        e, ln = e.clone(), ln / alpha
        d = self.dense(0, self.c["nrchop"], torch.zeros(1, dtype=torch.long, device=self.dev))[0].to(e.dtype)
        low = torch.zeros(self.c["nrchop"], dtype=e.dtype, device=self.dev)
        low[:3] = self.log_terms(ln, "2")
        high = low
        for _ in range(power // 2 - 1):
            high = d @ high
        e[0, 0, : self.c["nrchop"]] -= high + beta * low

        def matrix(m, nn, slots):
            a = self.dense(m, nn, slots)
            return torch.linalg.matrix_power(a, power // 2) + beta * a + alpha * torch.eye(nn, dtype=a.dtype, device=self.dev)

        return self.solve(e, ("p", power, alpha, beta), matrix), ln

    def idel2(self, e):
        """The inverse Laplacian that also finds the log term (from the (0, 0) column's first row)."""
        def matrix(m, nn, slots):
            a = self.dense(m, nn, slots)
            if m == 0:
                a[slots == 0, :3, 0] += self.log_terms(self.norm0[0], "2").real
            return a
        out = self.solve(e, "poisson", matrix)
        return out, float(out[0, 0, 0].real) * self.norm0[0]

    def abcn(self, s, ln, nl, nlp, dt):
        c = self.c
        if c["hyperpow"] == 0:
            vis = c["visc"] * self.band(s, ln, "2")
            a = -2.0 / (dt * c["visc"])
        else:
            hv = c["hypervisc"] * (-1.0) ** (c["hyperpow"] // 2 + 1)
            two = self.band(s, ln, "2")
            top = two
            for _ in range(c["hyperpow"] // 2 - 1):
                top = self.band(top, 0.0, "2")
            vis = hv * (top + c["visc"] / hv * two)
            a = -2.0 / (dt * hv)
        e = a * (s + dt * (1.5 * nl - 0.5 * nlp) + dt / 2 * vis)
        if c["hyperpow"] == 0:
            return self.ihelm(e, a * ln, a)
        return self.ihelmp(e, a * ln, c["hyperpow"], a, c["visc"] / hv)

    # -- vector fields
    def tp2vec(self, psi, lnpsi, chi, lnchi):
        ur, up = self.band(chi, lnchi, "xx", 3), self.band(psi, lnpsi, "xx", 3)
        uz = -self.band(chi, lnchi, "h", 3)
        m = torch.arange(self.npdim, device=self.dev, dtype=torch.float64)[None, :, None]
        k = self.ak[:, None, None]
        on = _active(self.c, 3)
        ur, up = (torch.where(on, a, b) for a, b in ((1j * m * psi + 1j * k * ur, ur), (-up - m * k * chi, up)))
        out = []
        for i, e in enumerate((ur, up, uz)):
            e = self.to_ppp(self.chop(e), 0.0)
            if i < 2:
                e[..., : self.c["nr"]] /= self.r
            out.append(e)
        return out

    def curl(self, psi, lnpsi, chi, lnchi):
        return self.tp2vec(-self.band(chi, lnchi, "2"), 0.0, psi, lnpsi)

    def vec2tp(self, vr, vp, vz):
        c, nr, h = self.c, self.c["nr"], self.c["nr"] // 2
        ur, up, uz = vr.clone(), vp.clone(), vz.clone()
        ur[..., :nr] *= self.r
        up[..., :nr] *= self.r
        ur, uz = (self.z(self.phi(e, -1), -1) for e in (ur, uz))
        up = self.to_fff(up, 0.0)
        ln = -0.5 * float((up[0, 0, : c["nrchop"]] * self.at1).sum().real)
        up = self.radial(up, 1)
        up[0, 0, :nr] += ln * (1 + self.x)
        psi, chi = self.zeros(), self.zeros()
        x, w = self.x[:h], self.w[:h]
        fff = (1 - x ** 2) / w
        keep = torch.cat(self.kept())
        for m in range(c["npchop"]):
            nn = self.nn(m, 3)
            if nn < 1:
                continue
            n = torch.clamp(m + torch.arange(nn, device=self.dev, dtype=torch.float64), min=1)[:, None]
            p = self.pf[m, : nn + 1, :h]
            t = torch.zeros((nn + 1, nn + 1), dtype=torch.float64, device=self.dev)
            t.diagonal(-1).copy_(self.bxx[m, 1: nn + 1, 0])
            t.diagonal(1).copy_(self.bxx[m, :nn, 2])
            d = (t.T @ p)[:nn] / n / (n + 1) / fff
            v = p[:nn] / n / (n + 1) / fff
            even = (torch.arange(nn, device=self.dev) % 2 == 0)[None]

            def mul(a, u, own):
                f, g = u[keep, m, :h], u[keep, m, h:nr].flip(-1)
                a = a.to(u.dtype).T
                return torch.where(even == own, (f + g) @ a, (f - g) @ a)

            kv = self.ak[keep][:, None]
            psi[keep, m, :nn] = -1j * m * mul(v, ur, True) - mul(d, up, False)
            chi[keep, m, :nn] = 1j * kv * mul(d, ur, False) + m * kv * mul(v, up, True) - mul(p[:nn] * w, uz, True)
        chi, _ = self.idel2(chi)
        return self.zeroat1(self.chop(psi)), self.zeroat1(self.chop(chi))

    def advect(self, psi, lnpsi, chi, lnchi):
        psi, chi = self.dealias(psi), self.dealias(chi)
        v, w = self.tp2vec(psi, lnpsi, chi, lnchi), self.curl(psi, lnpsi, chi, lnchi)
        nr, h = self.c["nr"], self.c["np"] // 2

        def product(a, b, c, d):   # a b - c d of the two samples in each value
            a, b, c, d = (torch.view_as_real(u[:, :h, :nr].contiguous()) for u in (a, b, c, d))
            o = self.zeros()
            o[:, :h, :nr] = _complex(a * b - c * d)
            return o

        s = (product(v[1], w[2], v[2], w[1]), product(v[2], w[0], v[0], w[2]), product(v[0], w[1], v[1], w[0]))
        return tuple(self.dealias(e) for e in self.vec2tp(*s))


def exact(case, seed):
    c = dict(case)
    points = c["nr"] * c["np"] * c["nz"]
    # dense factorisations and one multiplication for each m: within about 20 seconds up to these sizes
    if c["op"] == "adjoint" or points > (18e6 if c["op"] in ("transform", "fields") else 3.3e6):
        return None
    if c["op"] == "advect" and c["nr"] > 256 or c["op"] in ("run", "diffuse") and c["nr"] > 256:
        return None
    x, f = Exact(c), _inputs(c, int(seed))
    if c["op"] == "transform":
        p = x.to_ppp(*f["spectral"])
        return [p, x.to_fff(p, 0.0)]
    if c["op"] == "diffuse":
        (s, ln), nl, nlp = f["s"], f["nl"][0], f["nl_p"][0]
        for _ in range(c["steps"]):
            s, ln = x.abcn(s, ln, nl, nlp, c["dt"])
            nlp = nl
        return [s, s, nlp]
    (psi, lnpsi), (chi, lnchi) = f["psi"], f["chi"]
    if c["op"] == "fields":
        return x.tp2vec(psi, lnpsi, chi, lnchi) + x.curl(psi, lnpsi, chi, lnchi)
    if c["op"] == "advect":
        return list(x.advect(psi, lnpsi, chi, lnchi))
    nl = [f["nlpsi"][0], f["nlchi"][0]]
    old = [f["nlpsi_p"][0], f["nlchi_p"][0]]
    state, ln, gains, prev = [psi, chi], [lnpsi, lnchi], [0.0, 0.0], None
    for _ in range(c["steps"]):
        for i in range(2):
            state[i], ln[i] = x.abcn(state[i], ln[i], nl[i], old[i], c["dt"])
        prev, old = list(state), list(nl)
        for i in range(2):
            state[i] = x.dealias(state[i])
            if c["is_svv"]:
                state[i], gains[i] = x.svv(state[i], gains[i])
            state[i] = x.zeroat1(state[i])
        nl = list(x.advect(state[0], ln[0], state[1], ln[1]))
    return [*state, *nl, *prev, *old], gains
