"""Workloads of the framework for timing, through its public entry points.

Each case is what a user's program has it do: RK3 steps of boxes of the sizes
and precisions of opentbl_b200/config.py and of the parameter sweep of
opentbl_b200/ensemble.py (``Box.advance``), the reference's own call sequence
on caller-owned arrays (``rhsp_arrays``, ``outflow_correction_arrays``,
``pois_arrays``), an ensemble advanced by one CUDA graph, sampling of the
one-point statistics, and the stand-alone transforms of ffts.f90 with the
transposes of change.f90.

``exact`` restates each of them in plain torch and numpy in 64 bits: the
compact operators as dense matrices, torch's FFTs, cosine transforms as
matrices. It takes the packed coefficients (include/otbl_layout.h) as the
input they are to a context; nothing of the library's arithmetic is used.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from opentbl_b200 import ensemble, native, synth
from opentbl_b200.box import Box
from opentbl_b200.config import BoxConfig

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest box (tests and smoke runs, first experiments): latency of one step
        dict(name="step-33x41x32", kind="step", nx=33, ny=41, nz=32, mode="fp64", steps=1),
        # the smallest boxes of the parameter sweep, in the serving loop's chunks of 4 steps
        dict(name="step-mixed-129x65x64", kind="step", nx=129, ny=65, nz=64, mode="mixed", steps=4),
        # the reference's validation-sized box
        dict(name="step-257x97x128", kind="step", nx=257, ny=97, nz=128, mode="fp64", steps=1),
        # the same with the REAL4 transposes of change.f90, for runs that are compared with the reference
        dict(name="step-real4-385x97x64", kind="step", nx=385, ny=97, nz=64, mode="real4", steps=1),
        # the drop-in surface: the host program's own arrays and call sequence,
        # a streamwise length that is no power of two and an even ny
        dict(name="arrays-241x74x128", kind="arrays", nx=241, ny=74, nz=128, mode="fp64"),
        # the largest boxes of the parameter sweep
        dict(name="step-mixed-513x129x256", kind="step", nx=513, ny=129, nz=256, mode="mixed", steps=1),
        # production: the headline box, in both precisions
        dict(name="step-1025x193x512", kind="step", nx=1025, ny=193, nz=512, mode="fp64", steps=1),
        dict(name="step-mixed-1025x193x512", kind="step", nx=1025, ny=193, nz=512, mode="mixed", steps=1),
        # boxes of the seeded sweep advanced by one graph launch
        dict(name="ensemble-12", kind="ensemble", boxes=12, sweep=2024),
        # statistics: samples of statsp, then the accumulators read back
        dict(name="stats-257x97x128", kind="stats", nx=257, ny=97, nz=128, mode="fp64", samples=4),
        # fourxz on every row of a box, both directions
        dict(name="fourxz-256", kind="fourxz", nx=513, ny=97, nz=256),
        # the pencil cosine transforms with their transposes, both directions
        dict(name="pencils-513x65x128", kind="pencils", nx=513, ny=65, nz=128, mode="fp64"),
    ]


# nx - 1 is a product of 2, 3 and 5; nz a power of two; ny any integer
_NX = (33, 41, 49, 65, 73, 81, 97, 109, 129, 145, 161, 181, 193, 217, 241, 257, 289, 321, 361, 385, 433, 481, 513,
       577, 641, 721, 769, 865, 961, 1025)
_NZ = (32, 64, 128, 256, 512)
_MOST = 1025 * 193 * 512


def draw(rng):
    kind = rng.choice(("step",) * 6 + ("arrays", "ensemble", "stats", "fourxz", "pencils"))
    if kind == "ensemble":
        return dict(kind=kind, boxes=rng.randint(3, 10), sweep=rng.randrange(1 << 20))
    most = _MOST if kind in ("step", "arrays") else _MOST // 8
    while True:
        nx, nz = rng.choice(_NX), rng.choice(_NZ)
        ny = round(41 * (193 / 41) ** rng.random())
        if nx * ny * nz <= most:
            break
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "step":
        case.update(mode=rng.choice(("fp64", "fp64", "mixed", "mixed", "real4")), steps=rng.choice((1, 1, 2)))
        if nx * ny * nz > _MOST // 2:
            case["steps"] = 1
    elif kind == "arrays":
        case.update(mode="fp64")
    elif kind == "stats":
        case.update(mode=rng.choice(("fp64", "mixed")), samples=rng.choice((1, 2, 4)))
    elif kind == "pencils":
        case.update(mode=rng.choice(("fp64", "real4")))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(nx, ny, nz, mode):
    """A box of this size: the domain grows with nx as config.py's boxes."""
    re_theta = 300.0 if nx * ny * nz < 4_000_000 else 1000.0
    return BoxConfig(nx=nx, ny=ny, nz=nz, lx=max(12.0, 80.0 * nx / 1025), ly=8.0, lz=8.0,
                     dy_wall=0.02 if ny < 57 else 0.002, re_theta=re_theta,
                     profile="blasius" if re_theta < 700.0 else "musker",
                     xpose_round=int(mode == "real4"), precision=int(mode == "mixed"))


@functools.lru_cache(maxsize=64)
def _plan(key):
    """Grid, Reynolds number, mean flow and coefficients of a box."""
    cfg = BoxConfig(**dict(key))
    nx, ny = cfg.nx, cfg.ny
    y = synth.y_grid(cfg)
    re = synth.reynolds_for(cfg, y)
    dx = cfg.ax * math.pi / (nx + 1)
    # a layer that grows like x^0.8, profiles interpolated between 17 thicknesses
    delta = (1.0 + np.arange(nx) * dx / 60.0) ** 0.8
    at = np.linspace(delta[0], delta[-1], 17)
    prof = np.stack([synth.mean_profile(cfg, y, d, re) for d in at])
    pos = (delta - at[0]) / (at[1] - at[0])
    lo = np.clip(pos.astype(int), 0, 15)
    U = prof[lo] + (pos - lo)[:, None] * (prof[lo + 1] - prof[lo])
    dy = np.diff(y)
    V = np.zeros((nx, ny))  # from the discrete continuity of pois.f90:41-54
    V[1:, 1:] = -np.cumsum(dy[1:ny] * (U[1:, 1:ny] - U[:-1, 1:ny]) / dx, axis=1)
    V[0] = V[1]
    U, V = (a.astype(np.float32).astype(np.float64) for a in (U, V))
    xout = cfg.resolved_xout()
    coef = native.coef_compute(cfg, re, xout, y, U[0].copy())
    return cfg, y, re, xout, U, V, coef


def _key(cfg):
    return tuple(sorted(vars(cfg).items()))


def _velocity(cfg, seed):
    """u, v, w (nx, rows, nz1) on the GPU: the mean flow and divergence-free
    fluctuations of 5% below y = 1.2, smooth in x, around kz = 2."""
    _, y, _, _, U, V, _ = _plan(_key(cfg))
    nx, ny, nk = cfg.nx, cfg.ny, cfg.nz1 // 2
    rng = np.random.default_rng(seed)
    dx = cfg.ax * math.pi / (nx + 1)
    kz = np.arange(nk) / cfg.az
    spec = np.exp(-0.5 * (kz - 2.0) ** 2)
    spec[0] = 0.0
    t = np.clip(y[1:ny + 1] / 1.2, 0.0, 1.0)
    win = torch.as_tensor((t * (1.0 - t)) ** 2 * 16.0, device=DEV)
    lam, ph = rng.uniform(3.0, 8.0, (2, nk, 4, 1)), rng.uniform(0.0, 2 * np.pi, (2, nk, 4, 1))
    ca = rng.normal(size=(2, nk, 4, 1)) + 1j * rng.normal(size=(2, nk, 4, 1))
    arg = 2 * np.pi * np.arange(nx + 1) * dx / lam + ph
    pot = torch.as_tensor((ca * np.cos(arg)).sum(axis=2) * spec[:, None], device=DEV)  # (2, nk, nx+1)
    dy = torch.as_tensor(np.diff(y), device=DEV)[1:ny]
    u = torch.zeros(nx, ny + 1, nk, dtype=torch.complex128, device=DEV)
    w = torch.zeros_like(u)
    psi = pot[0].T[:, None, :] * win[None, :, None]
    u[:, 1:ny] = (psi[1:, 1:] - psi[1:, :-1]) / dy[None, :, None]
    v = (psi[:-1] - psi[1:]) / dx
    phi = pot[1].T[1:, None, :] * win[None, :, None]
    v += 1j * torch.as_tensor(kz, device=DEV) * phi
    w[:, 1:ny] = -(phi[:, 1:] - phi[:, :-1]) / dy[None, :, None]
    peak = max(float(torch.view_as_real(f).abs().max()) for f in (u, v, w))
    out = []
    for f, mean in ((u, U), (v, V), (w, None)):
        f *= cfg.amp / peak
        f[0] = 0.0  # the inflow plane: mean only
        if mean is not None:
            f[:, :, 0] += torch.as_tensor(mean, device=DEV)
        # restart files are REAL4 (getstartzy-bg.F90:98,110,128)
        out.append(torch.view_as_real(f).reshape(nx, f.shape[1], -1).float().double())
    return out


def _pressure(cfg, seed):
    """A pressure field with the size and spectrum of the flow's."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nk = cfg.nz1 // 2
    p = torch.randn(cfg.nx, cfg.ny, nk, 2, generator=g, device=DEV, dtype=F64)
    p *= (1e-3 / (1.0 + torch.arange(nk, device=DEV)))[:, None]
    p[:, :, 0, 1] = 0.0
    return p.reshape(cfg.nx, cfg.ny, -1).float().double()


class _Raw:
    """One field of a box as something torch can view; the views keep the box."""

    def __init__(self, box, name):
        self.box = box
        self.__cuda_array_interface__ = dict(shape=tuple(box.shape(name)), typestr="<f8",
                                             data=(box.device_ptr(name), False), version=3)


def _fields(box):
    """{name: tensor} of the state fields the box holds in 64 bits."""
    names = ("u", "v", "w") if box.cfg.precision else native.FIELDS
    return {n: torch.as_tensor(_Raw(box, n), device=DEV) for n in names}


class _DeviceBox(Box):
    """A box whose velocity comes from tensors on the GPU."""

    def load(self, init):
        own = _fields(self)
        for n, t in init["fields"].items():
            if n in own:
                own[n].copy_(t)
            else:
                self.set_field(n, t.cpu().numpy())
        torch.cuda.synchronize()  # the box's streams do not wait for torch's
        inf = native.OtblInflow()
        self._check(self.L.otbl_set_inflow(self.h, native.dptr(init["u0"]), native.dptr(init["v0"]),
                                           native.dptr(init["um"]), inf), "otbl_set_inflow")


def _box(cfg, seed, pressure=False):
    _, y, re, xout, U, V, coef = _plan(_key(cfg))
    f = dict(zip("uvw", _velocity(cfg, seed)))
    um = f["u"][xout - 1, :, 0].cpu().numpy()
    if pressure:
        f["p"] = _pressure(cfg, seed)
    return _DeviceBox(cfg, dict(re=re, xout=xout, y=y, u0=U[0].copy(), v0=V[0].copy(), um=um, fields=f), coef)


def _case_config(case):
    return _config(case["nx"], case["ny"], case["nz"], case.get("mode", "fp64"))


def _sweep(case):
    return ensemble.ensemble_configs(case["boxes"], seed=case["sweep"])


def _phys(case, seed):
    """fourxz: rows of physical values, and rows of modes."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    cfg = _case_config(case)
    lines = cfg.nx * (cfg.ny + 1)
    phys = torch.randn(lines, cfg.nz + 2, generator=g, device=DEV, dtype=F64)
    phys[:, cfg.nz:] = 0.0
    fou = torch.randn(lines, cfg.nz1, generator=g, device=DEV, dtype=F64)
    fou[:, 1] = 0.0
    return cfg, lines, phys, fou


def _planes(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    cfg = _case_config(case)
    return cfg, [torch.randn(cfg.nx, cfg.ny, cfg.nz1, generator=g, device=DEV, dtype=F64) for _ in range(2)]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("step", "stats"):
        s["box"] = _box(_case_config(case), seed, pressure=kind == "stats")
        s["fields"] = _fields(s["box"])
    elif kind == "arrays":
        cfg = _case_config(case)
        s["box"] = b = _box(cfg, seed)
        s["own"] = {n: t.clone() for n, t in _fields(b).items()}
        s["ptr"] = {n: t.data_ptr() for n, t in s["own"].items()}
    elif kind == "ensemble":
        s["members"] = [_box(cfg, seed + k) for k, cfg in enumerate(_sweep(case))]
        s["fields"] = [_fields(b) for b in s["members"]]
        s["graph"] = ensemble.Graph(s["members"], 1)
    elif kind == "fourxz":
        cfg, s["lines"], s["phys"], s["fou"] = _phys(case, seed)
        s["fou_out"], s["phys_out"] = torch.zeros_like(s["fou"]), torch.zeros_like(s["phys"])
        s["box"] = _box(_config(33, 41, case["nz"], "fp64"), seed)
    elif kind == "pencils":
        cfg, (s["a"], s["b"]) = _planes(case, seed)
        s["pen"] = torch.zeros(cfg.nz1 * cfg.ny, cfg.nx, device=DEV, dtype=F64)
        s["a_out"], s["b_out"] = torch.zeros_like(s["a"]), torch.zeros_like(s["b"])
        s["box"] = _box(cfg, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "step":
        s["box"].advance(s["steps"])
        return s["fields"]
    if kind == "arrays":
        b, own = s["box"], s["ptr"]
        for m in (1, 2, 3):
            b.rhsp_arrays(own, m, m == 1)
            b.outflow_correction_arrays(own)
            b.pois_arrays(own, m)
        return s["own"]
    if kind == "ensemble":
        s["graph"].launch()
        return s["fields"]
    if kind == "stats":
        b = s["box"]
        b.reset_stats()
        for _ in range(s["samples"]):
            b.statsp()
        acc, n = b.stats()
        return dict(acc=acc, samples=n)
    if kind == "fourxz":
        b = s["box"]
        b.fourxz(s["fou_out"].data_ptr(), s["phys"].data_ptr(), -1, s["lines"])
        b.fourxz(s["fou"].data_ptr(), s["phys_out"].data_ptr(), 1, s["lines"])
        return s["fou_out"], s["phys_out"]
    # the transforms of pois.f90: planes to pencils, transform, back; then the inverse
    b, ny, lines, pen = s["box"], s["ny"], s["pen"].shape[0], s["pen"].data_ptr()
    for src, dst, iopt in (("a", "a_out", -1), ("b", "b_out", 1)):
        b.chp2x(pen, s[src].data_ptr(), ny)
        b.cosftx(pen, lines, iopt)
        b.chx2p(pen, s[dst].data_ptr(), ny)
    return s["a_out"], s["b_out"]


def _box_work(cfg):
    """One RK3 step: each substep couples every point with every other
    (Poisson), so the seven state fields are read and written by each."""
    nf = cfg.nx * (cfg.ny + 1) * cfg.nz1
    e = 4 if cfg.precision else 8
    nbytes = 3 * 2 * nf * (3 * 8 + 4 * e)
    rows, lz = cfg.nx * (cfg.ny + 1), math.log2(cfg.nz)
    fft = rows * 15 * 2.5 * cfg.nz * lz                              # nine c2r, six r2c
    dct = 2 * (cfg.ny * cfg.nz1 / 2) * 5 * cfg.nx * math.log2(cfg.nx)
    lines = nf * (9 * 8 + 9 * 8 + 60)                                # 18 compact operators, the rest per point
    return dict(bytes=nbytes, flops=3 * (fft + dct + lines))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        each = [_box_work(c) for c in _sweep(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    cfg = _case_config(case)
    nf = cfg.nx * (cfg.ny + 1) * cfg.nz1
    if kind in ("step", "arrays"):
        return {k: v * case.get("steps", 1) for k, v in _box_work(cfg).items()}
    if kind == "stats":  # u, v, w, p in; 40 sums per row updated
        e = 4 if cfg.precision else 8
        per = nf * (3 * 8 + e) + 2 * 40 * 8 * cfg.nx * cfg.ny
        flops = nf * (12 * 9 + 60) + cfg.nx * cfg.ny * 3 * 2.5 * cfg.nz * math.log2(cfg.nz)
        return dict(bytes=case["samples"] * per, flops=case["samples"] * flops)
    if kind == "fourxz":
        lines = cfg.nx * (cfg.ny + 1)
        return dict(bytes=2 * lines * 8 * (cfg.nz + cfg.nz1), flops=2 * lines * 2.5 * cfg.nz * math.log2(cfg.nz))
    nf = cfg.nx * cfg.ny * cfg.nz1  # three passes each way: transpose, transform, transpose
    return dict(bytes=2 * 3 * 2 * nf * 8, flops=2 * nf * 2.5 * math.log2(cfg.nx))


def tolerance(case):
    """Four times what the framework shows against `exact` over the ranges,
    worst output and first or second pass: FP64 2.4e-9 (the pressure of a
    first projection, which the near-wall second differences amplify), mixed
    2.4e-6, REAL4 5e-4 (ties of the REAL4 rounding that fall the other way,
    amplified like that), statistics 1.4e-15, transforms 8e-16."""
    kind = case["kind"]
    if kind == "fourxz":
        return {"rel": 1e-15, "max": 4e-14}
    if kind == "pencils":
        return {"rel": 1e-7, "max": 1e-6} if case["mode"] == "real4" else {"rel": 4e-15, "max": 2e-13}
    if kind == "stats":
        return {"rel": 1e-14, "max": 1e-12}
    if kind == "ensemble" or case["mode"] == "mixed":
        return {"rel": 1e-5, "max": 5e-4}
    if case["mode"] == "real4":
        return {"rel": 2e-3, "max": 0.2}
    return {"rel": 1e-8, "max": 1e-6}


# ---------------------------------------------------------------------------
# the same in plain torch and numpy, 64 bits
# ---------------------------------------------------------------------------
_SCAL = dict(RE=0, REX=1, IDX=7, IDXX=8, DXMIN=9, DTRET=11, UINF=13, RTHIN=14, DIN=15, YBLEND=16, DX1=6)
_LENGTHS = (  # include/otbl_layout.h, in order: name, rows (Fortran's first dimension), length over that
    ("SCAL", 1, "64"), ("Y", 1, "ny+2"), ("DY", 1, "ny+1"), ("IDY", 1, "ny+1"), ("IDYY", 1, "ny"), ("DYMIN", 1, "ny"),
    ("HY", 1, "ny+1"), ("XG", 1, "nx+2"), ("DX", 1, "nx+1"), ("KAZ", 1, "nk"), ("KAZ2", 1, "nk"), ("KVIS", 1, "nk"),
    ("KMOD", 1, "nx-1"), ("AYP", 3, "ny"), ("VMAGIC", 1, "nx"), ("INXU", 3, "nx"), ("INXV", 3, "nx"),
    ("COFIUX", 2, "nx"), ("COFIVX", 2, "nx"), ("INBX", 4, "4"), ("DCXU", 3, "nx"), ("DCXV", 3, "nx"),
    ("COFCXU", 2, "nx"), ("COFCXV", 2, "nx"), ("DCBX", 5, "4"), ("VIXU", 3, "nx"), ("VIXV", 3, "nx"),
    ("COFVXU", 3, "nx"), ("COFVXV", 3, "nx"), ("COFVBX", 4, "4"), ("INYU", 3, "ny"), ("INYV", 3, "ny"),
    ("COFIUY", 2, "ny"), ("COFIVY", 2, "ny"), ("INBY", 4, "4"), ("DCYU", 3, "ny+1"), ("DCYV", 3, "ny"),
    ("COFCYU", 2, "ny"), ("COFCYV", 2, "ny"), ("DCBY", 4, "4"), ("VIYU", 3, "ny+1"), ("VIYV", 3, "ny"),
    ("VYUI", 3, "ny+1"), ("VYVI", 3, "ny"), ("COFVYU", 3, "ny"), ("COFVYV", 3, "ny"), ("COFVBY", 4, "4"),
    ("CCON", 2, "4"), ("FD_DVDY", 8, "ny"), ("FD_DX", 8, "nx"), ("FD_IX", 8, "nx"), ("FD_IY", 8, "ny"),
    ("FD_IYP", 8, "ny"))


def _unpack(cfg, coef):
    """{name: (length,) or (length, rows)} numpy arrays."""
    nx, ny = cfg.nx, cfg.ny
    sizes = {"4": 4, "64": 64, "nk": cfg.nz1 // 2, "nx-1": nx - 1, "nx": nx, "nx+1": nx + 1, "nx+2": nx + 2,
             "ny": ny, "ny+1": ny + 1, "ny+2": ny + 2}
    out, at = {}, 0
    for name, rows, length in _LENGTHS:
        n = rows * sizes[length]
        a = coef[at:at + n]
        out[name] = a.reshape(-1, rows) if rows > 1 else a
        at += n
    if at != len(coef):
        raise ValueError("coefficient layout")
    return out


def _solved(lu, B):
    """A^-1 B for the factored tridiagonal A: lu rows are -l, 1/pivot, upper."""
    n = len(lu)
    L = np.eye(n)
    U = np.diag(1.0 / lu[:, 1])
    k = np.arange(n - 1)
    L[k + 1, k] = -lu[1:, 0]
    U[k, k + 1] = lu[:-1, 2]
    A = torch.as_tensor(L @ U, device=DEV)
    return torch.linalg.solve(A, torch.as_tensor(B, device=DEV))


def _stencil(rows, cols, inner, first, last, lo=1, hi=None):
    """Dense matrix: `inner` (offset, values by row) on rows lo..rows-2, the
    closures on the first row (from column 0 up) and the last (from the last
    column down)."""
    B = np.zeros((rows, cols))
    for off, val in inner:
        for j in range(lo, rows - 1):
            B[j, j + off] = val[j]
    B[0, :len(first)] = first
    B[rows - 1, cols - 1 - np.arange(len(last))] = last
    return B


class _Exact:
    """One box in 64 bits."""

    def __init__(self, cfg, seed, pressure=False):
        _, self.y, self.re, self.xout, U, V, coef = _plan(_key(cfg))
        self.cfg, self.c = cfg, _unpack(cfg, coef)
        self.S = self.c["SCAL"]
        self.u, self.v, self.w = _velocity(cfg, seed)
        self.p = _pressure(cfg, seed) if pressure else torch.zeros_like(self.v)
        self.um = self.u[self.xout - 1, :, 0].cpu().numpy().copy()
        self.u0, self.v0 = U[0], V[0]
        self.hu, self.hv, self.hw = (torch.zeros_like(f) for f in (self.u, self.v, self.w))
        self.tiempo = 0.0
        self.dt = 0.0

    def s(self, name):
        return float(self.S[_SCAL[name]])

    def r(self, f):  # the REAL4 rounding of the transposes
        return f.float().double() if self.cfg.xpose_round else f

    def dev(self, name):
        return torch.as_tensor(self.c[name], device=DEV)

    # ---- operators as matrices ----
    @functools.cached_property
    def mats(self):
        c, nx, ny = self.c, self.cfg.nx, self.cfg.ny
        m = {}
        for t, chi, ic, chv in (("U", 1, 2, 0), ("V", 0, 0, 1)):
            e = c["COFI%sX" % t]
            first = c["INBX"][:, 2 if t == "U" else 3]
            m["ix" + t] = _solved(c["INX" + t], _stencil(nx, nx, ((0, e[:, 0]), (1, e[:, 1])), first, c["INBX"][:, chi]))
            e = c["COFCX" + t]
            m["dx" + t] = _solved(c["DCX" + t], _stencil(nx, nx, ((-1, e[:, 0]), (0, e[:, 1])), c["DCBX"][:, chv],
                                                         c["DCBX"][:, chv + 2]))
            e = c["COFVX" + t]
            m["vx" + t] = _solved(c["VIX" + t], _stencil(nx, nx, ((1, e[:, 0]), (0, e[:, 1]), (-1, e[:, 2])),
                                                         c["COFVBX"][:, ic], c["COFVBX"][:, ic + 1]))
        e = c["COFIUY"]
        m["iyU"] = _solved(c["INYU"], _stencil(ny, ny + 1, ((0, e[:, 0]), (1, e[:, 1])), [], c["INBY"][:, 0]))
        e = c["COFIVY"]
        m["iyV"] = _solved(c["INYV"], _stencil(ny, ny, ((0, e[:, 1]), (-1, e[:, 0])), c["INBY"][:, 2], c["INBY"][:, 3]))
        e = c["COFCYU"]
        m["dyU"] = _solved(c["DCYU"], _stencil(ny + 1, ny, ((0, e[:, 1]), (-1, e[:, 0])), c["DCBY"][:, 2],
                                               c["DCBY"][:, 3]))
        e = c["COFCYV"]
        m["dyV"] = _solved(c["DCYV"], _stencil(ny, ny, ((1, e[:, 1]), (0, e[:, 0])), c["DCBY"][:, 0], c["DCBY"][:, 1]))
        for t, rows, ic in (("U", ny + 1, 2), ("V", ny, 0)):
            e = c["COFVY" + t]
            m["vy" + t] = _solved(c["VIY" + t], _stencil(rows, rows, ((1, e[:, 0]), (0, e[:, 1]), (-1, e[:, 2])),
                                                         c["COFVBY"][:, ic], c["COFVBY"][:, ic + 1]))
        return m

    def X(self, name, f):
        return (self.mats[name] @ f.reshape(f.shape[0], -1)).reshape(f.shape)

    def Y(self, name, f):
        return torch.matmul(self.mats[name], f)

    # ---- spanwise transforms ----
    def cx(self, f):
        return torch.view_as_complex(f.reshape(*f.shape[:-1], -1, 2))

    def re_(self, z):
        return torch.view_as_real(z.contiguous()).reshape(*z.shape[:-1], -1)

    def phys(self, f):
        z = self.cx(f).clone()
        z[..., 0].imag = 0.0
        return torch.fft.irfft(z, n=self.cfg.nz, dim=-1, norm="forward")

    def modes(self, q):
        return self.re_(torch.fft.rfft(q, dim=-1, norm="forward")[..., :self.cfg.nz1 // 2])

    def ikz(self, f):
        return self.re_(1j * self.dev("KAZ") * self.cx(f))

    # ---- genflu.F90:3-242 ----
    def genflu(self):
        c, ny, y = self.c, self.cfg.ny, self.y
        din, dy = self.s("DIN"), self.c["DY"]
        i = self.xout - 1
        pl = {n: getattr(self, n)[i].clone() for n in "uvw"}
        fb = torch.as_tensor(0.5 * (1 - np.tanh(y[1:ny + 2] - self.s("YBLEND"))), device=DEV)[:, None]
        for n in "uw":
            pl[n][:, 2:] *= fb
        tl = self.tiempo
        timec = 20.0 if tl < 20 else 100.0 if tl < 100 else tl
        a = self.dt / timec
        self.um = um = a * pl["u"][:, 0].cpu().numpy() + self.um * (1.0 - a)
        uinf = um[ny - 20:ny - 4].sum() / 16.0
        above = np.nonzero(um[:ny - 2] >= float(np.float32(0.99)) * uinf)[0]
        first = int(above[0]) + 1 if len(above) else ny - 1
        jtop = 0 if first == 1 else first
        q = um[1:jtop + 3]
        rthout = ((uinf - q) * q * dy[1:jtop + 3]).sum() * self.re / uinf
        g2 = self.s("RTHIN") / rthout
        g1 = g2 ** 0.125
        tabs = []
        for kk in (0, 1):
            ys = (0.5 * (y[1:ny + 1] + y[2:ny + 2]) if kk == 0 else y[1:ny + 1]) / din
            mid = 0.5 * (ys[1:] + ys[:-1])
            with np.errstate(over="ignore"):
                wt = np.where(mid >= 1.0, 1.0, 0.5 * (1.0 + np.tanh(4.0 * (mid - 0.2) / (0.6 * mid + 0.2)) / np.tanh(4.0)))
            ww = np.concatenate([[0.0], np.cumsum(wt * np.diff(ys))])
            www1 = float(np.float32(0.7895))
            for j in range(1, ny):
                if ys[j] >= 1.0 and ys[j - 1] < 1.0:
                    www1 = ww[j - 1] + (1.0 - ys[j - 1]) * wt[j - 1]
            wl = ys / g1 + (1.0 / g2 - 1.0 / g1) / www1 * ww
            kl, fs, ntop, kll = np.zeros(ny, int), np.zeros(ny), 0, 1
            for j in range(ny):
                if wl[j] <= ys[ny - 1]:
                    ntop, khh = j + 1, ny
                    while khh - kll > 1:
                        kx = (khh + kll) // 2
                        if ys[kx - 1] >= wl[j]:
                            khh = kx
                        else:
                            kll = kx
                    kl[j], fs[j] = kll, (wl[j] - ys[kll - 1]) / (ys[khh - 1] - ys[kll - 1])
            tabs.append((kl, fs, ntop))
        for n, kk, rows in (("u", 0, ny + 1), ("w", 0, ny + 1), ("v", 1, ny)):
            kl, fs, nt = tabs[kk]
            f = pl[n]
            k = torch.as_tensor(kl[:nt], device=DEV)
            t = torch.as_tensor(fs[:nt], device=DEV)[:, None]
            off = 1 if rows == ny + 1 else 0
            wk = torch.zeros(max(rows, nt + off), f.shape[1], device=DEV, dtype=F64)
            wk[off:nt + off] = f[k + off] * t + f[k + off - 1] * (1 - t)
            if off:
                wk[0] = -wk[1]
            wk[nt - 3:] = wk[nt - 4].clone()
            out = wk[:rows] / g1
            out[:, :2] = 0.0
            if n != "w":
                out[:, 0] = torch.as_tensor(self.u0 if n == "u" else self.v0, device=DEV)
            getattr(self, n)[0] = out

    # ---- rhsp.F90:22-489 ----
    def implicit(self, u, res, t, var1):
        icon, e = self.c["VY%sI" % t], self.c["COFVY" + t]
        jee = len(icon)
        n = jee - 2
        j = np.arange(1, jee - 1)
        a = icon[j] + var1 * e[j][:, ::-1]
        T = np.zeros((n, jee))
        Bm = np.zeros((n, jee))
        for q in range(3):
            T[np.arange(n), np.arange(n) + q] = a[:, q]
            Bm[np.arange(n), np.arange(n) + q] = icon[j, q]
        T, Bm = torch.as_tensor(T, device=DEV), torch.as_tensor(Bm, device=DEV)
        rhs = torch.matmul(Bm, res) - torch.matmul(T[:, [0, jee - 1]], u[:, [0, jee - 1]])
        inv = torch.linalg.inv(T[:, 1:-1])
        x = torch.matmul(inv, rhs)
        x += torch.matmul(inv, rhs - torch.matmul(T[:, 1:-1], x))  # one refinement
        u[:, 1:-1] = x

    def rhsp(self, m, setstep):
        c, cfg = self.c, self.cfg
        nx, ny = cfg.nx, cfg.ny
        u, v, w, p = self.u, self.v, self.w, self.p
        r = self.r
        pu, pv, pw = r(u), r(v), r(w)
        pux, puy = self.phys(u), self.phys(self.Y("iyU", u))
        q = self.phys(r(self.X("ixU", pu)))
        uu = self.modes(q * q)
        q = self.phys(r(self.X("ixV", pw)))
        wmax = float(q.abs().max())
        uw = self.modes(q * pux)
        umax = float(pux.abs().max())
        q = self.phys(r(self.X("ixV", pv)))
        vmax = q.abs().amax(dim=(0, 2)).cpu().numpy()
        uv = self.modes(q * puy)
        del q, pux, puy
        uinf, idx, rex = self.s("UINF"), self.s("IDX"), self.s("REX")

        def difvis(g, f, t):
            o = self.X("dx" + t, r(g))
            o[-1] = uinf * (f[-1] - f[-2]) * idx
            x = self.X("vx" + t, f)
            x[-1] = 0.0
            return r(o + rex * x)

        cu, rv, rw = difvis(uu, pu, "U"), difvis(uv, pv, "V"), difvis(uw, pw, "V")
        ru = self.Y("dyU", uv) + self.ikz(uw) + cu
        ru[-1] = cu[-1]
        del cu, uu, uw, uv, pu, pv, pw
        if setstep:
            dt = min(self.s("DXMIN") / max(1e-7, umax), self.s("DXMIN") / max(1e-7, wmax), self.s("DTRET"))
            self.dt = min(dt, float((c["DYMIN"] / np.maximum(1e-7, vmax)).min()))
        rk = {n: float(self.S[o + m - 1]) for n, o in (("c", 20), ("d", 23), ("cv", 26), ("dv", 29))}
        var1, var2 = self.dt * (rk["cv"] + rk["dv"]), self.dt * rex * rk["cv"]
        var3, var4 = self.dt * rk["c"], self.dt * rk["d"]
        old = [f.clone() for f in (u, v, w)]
        self.genflu()
        u[1:-1, 1:ny] -= var1 * self.s("IDXX") * (p[2:, 1:] - p[1:-1, 1:])
        v[1:, 1:ny - 1] -= var1 * self.dev("IDYY")[1:ny - 1, None] * (p[1:, 2:] - p[1:, 1:-1])
        w[1:, 1:ny] -= var1 * self.ikz(p[1:, 1:])
        kvis = self.dev("KVIS").repeat_interleave(2)
        I = slice(1, nx - 1)
        ru[I, 1:ny] -= old[0][I, 1:ny] * kvis
        rw[I, 1:ny] -= old[2][I, 1:ny] * kvis
        rv[I, 1:ny - 1] -= old[1][I, 1:ny - 1] * kvis
        vw = self.modes(self.phys(old[1][I]) * self.phys(self.Y("iyU", old[2][I])))
        rv[I] += self.ikz(vw)
        rw[I] += self.Y("dyU", vw)
        del vw
        q = self.phys(self.Y("iyV", old[1][I]))
        rv[I] += self.Y("dyV", self.modes(q * q))
        q = self.phys(old[2][I, :ny])
        rw[I, :ny] += self.ikz(self.modes(q * q))
        del q
        ib, cc = c["INBY"][:, 1], c["CCON"][:, 0]
        v[:, 0] = 0.0
        v[:, -1] = 0.0
        v[:, -1, 0] = self.dev("VMAGIC")
        for f in (u, w):
            f[:, 0] = -(ib[1] * f[:, 1] + ib[2] * f[:, 2] + ib[3] * f[:, 3]) / ib[0]
            f[:, ny] = -(cc[1] * f[:, ny - 1] + cc[2] * f[:, ny - 2] + cc[3] * f[:, ny - 3]) / cc[0]
        for f in (ru, rv, rw):
            f[0] = 0.0
        rv[:, 0] = 0.0
        rv[:, -1] = 0.0
        for f in (ru, rw):
            f[:, 0] = -(ib[1] * f[:, 1] + ib[2] * f[:, 2] + ib[3] * f[:, 3]) / ib[0]
            f[:, ny] = 0.0
        rkk = rex * self.dt * rk["dv"]
        for f, o, rh, h, t in ((u, old[0], ru, self.hu, "U"), (v, old[1], rv, self.hv, "V"), (w, old[2], rw, self.hw, "U")):
            vis = self.Y("vy" + t, o[1:])
            vis[-1] = 0.0
            res = f[1:] - (var3 * rh[1:] + var2 * vis + var4 * h[1:])
            self.implicit(f[1:], res, t, rkk)
        self.hu, self.hv, self.hw = ru, rv, rw

    # ---- boun.f90:63-93, pois.f90:11-239 ----
    def outflow(self):
        dy, ny = self.dev("DY"), self.cfg.ny
        total = self.v[1:, -1, 0].sum() * self.s("DX1")
        total = total + ((self.u[-1, 1:ny, 0] - self.u[0, 1:ny, 0]) * dy[1:ny]).sum()
        alpha = -total / float(self.y[ny] - self.y[1])
        self.u[-1, 1:ny, 0] += alpha
        self.hu[-1, 1:ny, 0] += alpha * self.s("IDX")

    def pois(self, m):
        c, cfg, ny = self.c, self.cfg, self.cfg.ny
        n, r = cfg.nx - 1, self.r
        u, v, w, p = self.u, self.v, self.w, self.p
        f = self.ikz(w[1:, 1:ny]) + (v[1:, 1:] - v[1:, :-1]) * self.dev("IDY")[1:ny, None]
        f = r(f + self.s("IDX") * (u[1:, 1:ny] - u[:-1, 1:ny]))
        C = _cosines(n)
        f = r((2.0 / n * (C @ f.reshape(n, -1))).reshape(f.shape))
        f[..., 1] = 0.0
        z = self.cx(f)
        ayp = c["AYP"]
        diag0 = -self.dev("KAZ2")[None, :] - self.dev("KMOD")[:, None]
        z[0, ny - 2, 0] = 0.0
        piv, low = [None] * (ny - 1), [None] * (ny - 1)
        for j in range(ny - 1):
            d = ayp[j, 1] + diag0
            if j == ny - 2:
                d[0, 0] = 2.0 * ayp[j, 1]
            if j:
                low[j] = -ayp[j, 0] * piv[j - 1]
                d = d + low[j] * ayp[j - 1, 2]
                z[:, j] += low[j] * z[:, j - 1]
            piv[j] = 1.0 / d
        z[:, ny - 2] *= piv[ny - 2]
        for j in range(ny - 3, -1, -1):
            z[:, j] = (z[:, j] - ayp[j, 2] * z[:, j + 1]) * piv[j]
        f = r(self.re_(z))
        half = torch.ones(n, 1, device=DEV, dtype=F64)
        half[0] = 0.5
        f = r((C.T @ (half * f.reshape(n, -1))).reshape(f.shape))
        varstep = 0.5 / self.dt / float(self.S[29 + m - 1])
        p[1:, 1:] += varstep * f
        w[1:, 1:ny] -= self.ikz(f)
        v[1:, 1:ny - 1] -= self.dev("IDYY")[1:ny - 1, None] * (f[:, 1:] - f[:, :-1])
        u[1:-1, 1:ny] -= self.s("IDXX") * (f[1:] - f[:-1])

    def advance(self, steps):
        for _ in range(steps):
            for m in (1, 2, 3):
                self.rhsp(m, m == 1)
                self.outflow()
                self.pois(m)
            self.tiempo += self.dt

    def fields(self):
        f = dict(u=self.u, v=self.v, w=self.w)
        if not self.cfg.precision:
            f.update(p=self.p, rhsupa=self.hu, rhsvpa=self.hv, rhswpa=self.hw)
        return f

    # ---- stotf.F90:51-291, rhsp.F90:70-92 ----
    def stats(self):
        c, cfg = self.c, self.cfg
        nx, ny, r = cfg.nx, cfg.ny, self.r

        def lu(a, first=1):
            t = np.stack([-a[:, 5], a[:, 6], a[:, 7]], axis=1)
            t[:first, 0] = 0.0
            return t

        def rows(shape, entries):
            B = np.zeros(shape)
            for j, at, val in entries:
                B[j, at:at + len(val)] = val
            return B

        a = c["FD_IX"]
        ix = _solved(lu(a), rows((nx, nx), [(0, 0, a[0, :4])] + [(i, i - 1, a[2, :4]) for i in range(1, nx - 2)] +
                                 [(nx - 2, nx - 4, a[nx - 2, :4]), (nx - 1, nx - 4, a[nx - 1, :4])]))
        a = c["FD_DX"]
        dx = _solved(lu(a), rows((nx, nx), [(0, 0, a[0, :5]), (1, 0, a[1, :5])] +
                                 [(i, i - 2, a[2, :5]) for i in range(2, nx - 2)] +
                                 [(nx - 2, nx - 5, a[nx - 2, :5]), (nx - 1, nx - 5, a[nx - 1, :5])]))

        def iy(a, tipo):
            k = 3 if tipo else 4
            ent = [] if tipo == 0 else [(0, 1, a[0, :4])]
            ent += [(1, 1, a[1, :5])] + [(j, j - 1, a[j, :4]) for j in range(2, ny - 2)]
            ent += [(ny - 2, ny - 3, a[ny - 2, :k]), (ny - 1, ny - 3, a[ny - 1, :k])]
            t = lu(a, first=2)
            t[0] = (0.0, 1.0, 0.0)
            return _solved(t, rows((ny, ny + 1 - tipo), ent))

        iyu, iyp = iy(c["FD_IY"], 0), iy(c["FD_IYP"], 1)
        a = c["FD_DVDY"]
        dy = _solved(lu(a), rows((ny, ny), [(0, 0, a[0, :4]), (1, 0, a[1, :4])] +
                                 [(j, j - 2, a[j, :5]) for j in range(2, ny - 2)] +
                                 [(ny - 2, ny - 4, a[ny - 2, :4]), (ny - 1, ny - 4, a[ny - 1, :4])]))

        def X(M, f):
            return (M @ f.reshape(nx, -1)).reshape(f.shape)

        pu, pv, pw = r(self.u), r(self.v), r(self.w)
        ux = X(ix, pu)
        ux[1:] = ux[:-1].clone()
        dudx, dvdx, dwdx = r(X(dx, ux)), r(X(dx, pv)), r(X(dx, pw))
        u, w = torch.matmul(iyu, r(ux)), torch.matmul(iyu, self.w)
        wx, ux_, p = torch.matmul(iyu, dwdx), torch.matmul(iyu, dudx), torch.matmul(iyp, self.p)
        uy, wy, vy = torch.matmul(dy, u), torch.matmul(dy, w), torch.matmul(dy, self.v)
        v, vx = self.v, dvdx
        uz, vz, wz = self.ikz(u), self.ikz(v), self.ikz(w)
        cte = torch.full((cfg.nz1,), 2.0, device=DEV, dtype=F64)
        cte[:2] = 1.0
        dot = lambda f, g: (cte * f * g).sum(-1)  # noqa: E731
        sq = lambda *fs: sum(dot(f, f) for f in fs)  # noqa: E731
        m0 = [f[..., 0] for f in (u, v, w, p, ux_, vx, wx, uy, vy, wy)]
        out = m0 + [wy[..., 0], -wx[..., 0], vx[..., 0] - uy[..., 0]]
        out += [sq(u), sq(v), sq(w), dot(u, v), dot(u, w), dot(v, w)]
        out += [dot(p, u), dot(p, v), sq(p), dot(p, ux_), dot(p, uy), dot(p, vx), dot(p, vy), dot(p, wz)]
        out += [sq(wy - vz), sq(uz - wx), sq(vx - uy)]
        out += [sq(ux_, uz, uy), sq(vx, vz, vy), sq(wz, wx, wy), dot(uz, vz) + dot(ux_, vx) + dot(uy, vy)]
        a, b, d = self.phys(u), self.phys(v), self.phys(w)
        out += [t.sum(-1) for t in (a ** 3, b ** 3, a * a * b, b * b * a, d * d * b, d * d * a)]
        return torch.stack(out)


@functools.lru_cache(maxsize=2)
def _cosines(n):
    k = torch.arange(n, device=DEV, dtype=torch.int64)
    arg = (k[:, None] * (2 * k[None, :] + 1)) % (4 * n)
    return torch.cos(arg.double() * (math.pi / (2 * n)))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "arrays"):
        e = _Exact(_case_config(case), seed)
        e.advance(case.get("steps", 1))
        return e.fields()
    if kind == "ensemble":
        out = []
        for k, cfg in enumerate(_sweep(case)):
            e = _Exact(cfg, seed + k)
            e.advance(1)
            out.append(e.fields())
        return out
    if kind == "stats":
        acc = _Exact(_case_config(case), seed, pressure=True).stats()
        return dict(acc=case["samples"] * acc, samples=None)
    if kind == "fourxz":
        cfg, _, phys, fou = _phys(case, seed)
        f = torch.fft.rfft(phys[:, :cfg.nz], norm="forward")[:, :cfg.nz1 // 2]
        q = torch.zeros_like(phys)
        q[:, :cfg.nz] = torch.fft.irfft(torch.view_as_complex(fou.reshape(len(fou), -1, 2)), n=cfg.nz, norm="forward")
        return torch.view_as_real(f.contiguous()).reshape(len(fou), -1), q
    cfg, (a, b) = _planes(case, seed)
    r = (lambda f: f.float().double()) if cfg.xpose_round else (lambda f: f)  # noqa: E731
    n = cfg.nx - 1
    C = _cosines(n)
    a, b = r(a), r(b)
    a[1:] = (2.0 / n * (C @ a[1:].reshape(n, -1))).reshape(n, *a.shape[1:])
    half = torch.ones(n, 1, device=DEV, dtype=F64)
    half[0] = 0.5
    b[1:] = (C.T @ (half * b[1:].reshape(n, -1))).reshape(n, *b.shape[1:])
    return r(a), r(b)
