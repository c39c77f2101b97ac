"""The chunked line solves at the edges of their chunks, against the oracle.

Chunk lengths change at nx = 160, 1152 and 2176 (5, 9, 17, 33 planes) and at
ny = 447 (7, 15 rows); a last chunk may hold a single plane or row, whose
boundary closures then reach into the chunk before it. Bounds: those of
test_gpu_parity.py and the mixed path's regression bound of test_gpu_mixed.py.
"""
import numpy as np
import pytest

from opentbl_b200 import Box, config, native
from opentbl_b200.config import replace

from helpers import oracle_box, rel_l2, setup, velocity_rel_l2

pytestmark = pytest.mark.gpu

STATE = ("u", "v", "w", "p", "rhsupa", "rhsvpa", "rhswpa")


@pytest.mark.parametrize("nx,ny,dy", [
    (151, 49, 0.02),    # 30 chunks of 5 and one plane; 7 x 7 rows and one (u, w)
    (161, 50, 0.02),    # 17 x 9 + 8 planes; 7 x 7 rows and one (v)
    (1153, 41, 0.02),   # chunks of 17 planes, coefficients from global memory
    (2305, 41, 0.02),   # chunks of 33 planes
    (33, 450, 0.005),   # chunks of 15 rows; 30 x 15 rows and one (u, w)
], ids=str)
def test_one_substep(nx, ny, dy):
    cfg = replace(config.TINY, nx=nx, ny=ny, lx=12.0 * nx / 33, dy_wall=dy, name=f"lines-{nx}x{ny}")
    init, coef = setup(cfg)
    g, o = Box(cfg, init, coef), oracle_box(cfg, init)
    g.rhsp(1, True)
    o.rhsp(1, 1)
    e = {n: rel_l2(g.field(n), o.field(n)) for n in STATE}
    assert max(e.values()) <= 1e-11, e
    # the projection of a box 838 delta0 long amplifies rounding: 1.7e-11 in v
    # at nx = 2305, with serial line solves too
    for b in (g, o):
        b.outflow_correction()
        b.pois(1)
    e = {n: rel_l2(g.field(n), o.field(n)) for n in STATE}
    assert max(e.values()) <= 1e-10, e


@pytest.mark.parametrize("nx,ny,nz", [(17, 50, 512), (65, 71, 256)], ids=str)
def test_wide_one_substep(nx, ny, nz):
    """Rows of several blocks of 128 columns: interpyy and the tail are streamed
    on small boxes too."""
    cfg = replace(config.TINY, nx=nx, ny=ny, nz=nz, lx=12.0 * max(nx, 33) / 33, name="lines-wide")
    init, coef = setup(cfg)
    g, o = Box(cfg, init, coef), oracle_box(cfg, init)
    g.substep(1, True)
    o.substep(1, 1)
    e = {n: rel_l2(g.field(n), o.field(n)) for n in STATE}
    assert max(e.values()) <= 1e-11, e


@pytest.mark.parametrize("nx,ny,nz", [(151, 50, 32), (17, 50, 512), (65, 50, 512)], ids=str)
def test_mixed_one_substep(nx, ny, nz):
    cfg = replace(config.TINY, nx=nx, ny=ny, nz=nz, lx=12.0 * max(nx, 33) / 33, precision=1, name="lines-mixed")
    init, coef = setup(cfg)
    g, o = Box(cfg, init, coef), oracle_box(replace(cfg, precision=0), init)
    g.substep(1, True)
    o.substep(1, 1)
    assert velocity_rel_l2(*({n: b.field(n) for n in "uvw"} for b in (g, o))) <= 1e-7


def _serial_interpyy(g, coef, cfg, which, T):
    """interpyy of the columns g (rows, columns) as one serial sweep up and one
    down, every multiply-add rounded once to T (T None: not rounded)."""
    ny, off, X = cfg.ny, native.coef_offsets(cfg), np.longdouble
    R = (lambda a: a) if T is None else (lambda a: np.asarray(a).astype(T).astype(X))

    def block(name, n, m):
        return R(coef[off[name]:off[name] + n * m].reshape(n, m).astype(X))

    lu, e = block("INYV" if which else "INYU", ny, 3), block("COFIVY" if which else "COFIUY", ny, 2)
    inby = block("INBY", 4, 4)
    g = R(g.astype(X))
    rows = len(g)
    b = np.zeros((ny, g.shape[1]), X)
    lo = -1 if which else 0
    for r in range(1, ny - 1):
        b[r] = R(e[r, 1] * g[r + lo + 1] + R(e[r, 0] * g[r + lo]))
    for m in range(4):
        if which:
            b[0] = R(b[0] + inby[m, 2] * g[m])
        b[ny - 1] = R(b[ny - 1] + inby[m, 3 if which else 0] * g[rows - 1 - m])
    for r in range(1, ny):
        b[r] = R(b[r] + lu[r, 0] * b[r - 1])
    b[ny - 1] = R(b[ny - 1] * lu[ny - 1, 1])
    for r in range(ny - 2, -1, -1):
        b[r] = R(R(b[r] - lu[r, 2] * b[r + 1]) * lu[r, 1])
    return b


@pytest.mark.parametrize("precision,ny", [(0, 57), (1, 57), (0, 450), (1, 450)], ids=str)
def test_solves_round_like_serial_sweeps(precision, ny):
    """The chunked solve is no further from the exact one than a serial sweep
    in the same precision: rms errors over 3 fields x 41 x 42 random smooth
    columns, whose means agree to 3% (sweeps that add the carry afterwards
    are 10-20% further off)."""
    cfg = replace(config.SMALL, nx=41, ny=ny, lx=24.0 * 41 / 65, dy_wall=0.006 if ny < 100 else 0.001,
                  precision=precision)
    init, coef = setup(cfg)
    rng = np.random.default_rng(5)
    fields = {}
    for n, rows in (("u", ny + 1), ("w", ny + 1), ("v", ny)):
        t, k = np.linspace(0.0, 1.0, rows)[:, None], rng.integers(0, 12, cfg.nx * cfg.nz1)
        a, c, p = (rng.uniform(lo, hi, len(k)) for lo, hi in ((0.2, 1.0), (0.0, 0.3), (0.0, 6.0)))
        f = a + c * np.sin(2 * np.pi * k * t + p)
        fields[n] = f
        init[n] = np.ascontiguousarray(f.reshape(rows, cfg.nx, cfg.nz1).transpose(1, 0, 2))
    b = Box(cfg, init, coef)
    got = dict(zip(("u", "w", "v"), b.interpyy()))
    T = np.float32 if precision else np.float64
    err = {"chunked": 0.0, "serial": 0.0}
    for n, f in fields.items():
        which = int(n == "v")
        ref = _serial_interpyy(f, coef, cfg, which, None)
        mine = got[n].transpose(1, 0, 2).reshape(ny, -1)
        for how, x in (("chunked", mine), ("serial", _serial_interpyy(f, coef, cfg, which, T))):
            err[how] += float(np.mean((x - ref) ** 2) / np.mean(ref ** 2))
    print({k: v ** 0.5 for k, v in err.items()})
    assert err["chunked"] ** 0.5 <= 1.03 * err["serial"] ** 0.5, err
