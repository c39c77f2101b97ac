"""The chunked line solves at the edges of their chunks, against the oracle.

Chunk lengths change at nx = 160, 1152 and 2176 (5, 9, 17, 33 planes) and at
ny = 447 (7, 15 rows); a last chunk may hold a single plane or row, whose
boundary closures then reach into the chunk before it. Bounds: those of
test_gpu_parity.py and the mixed path's regression bound of test_gpu_mixed.py.
"""
import pytest

from opentbl_b200 import Box, config
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


def test_wide_one_substep():
    """nz1 = 340 fills the streamed kernels' blocks of 128 columns: interpyy and
    the tail are streamed on a small box too."""
    cfg = replace(config.TINY, nx=17, ny=50, nz=512, name="lines-wide")
    init, coef = setup(cfg)
    g, o = Box(cfg, init, coef), oracle_box(cfg, init)
    g.substep(1, True)
    o.substep(1, 1)
    e = {n: rel_l2(g.field(n), o.field(n)) for n in STATE}
    assert max(e.values()) <= 1e-11, e


@pytest.mark.parametrize("nx,ny,nz", [(151, 50, 32), (17, 50, 512)], ids=str)
def test_mixed_one_substep(nx, ny, nz):
    cfg = replace(config.TINY, nx=nx, ny=ny, nz=nz, lx=12.0 * max(nx, 33) / 33, precision=1, name="lines-mixed")
    init, coef = setup(cfg)
    g, o = Box(cfg, init, coef), oracle_box(replace(cfg, precision=0), init)
    g.substep(1, True)
    o.substep(1, 1)
    assert velocity_rel_l2(*({n: b.field(n) for n in "uvw"} for b in (g, o))) <= 1e-7
