"""Entry points on boxes taller than the chunked line solves hold (3840 rows,
8448 for the statistics), against the oracle: pois, interpyy and statsp have no
limit on ny of their own (rhsp ends at genflu's 3227 rows)."""
import numpy as np
import pytest

from opentbl_b200 import Box, config
from opentbl_b200.config import replace

from helpers import oracle_box, rel_l2, setup
from test_gpu_stats import _errors
from test_gpu_ydense import _oracle_interpyy

pytestmark = pytest.mark.gpu


def _boxes(ny, **kw):
    cfg = replace(config.TINY, nx=9, ny=ny, nz=16, dy_wall=2.0 / ny, name=f"tall-{ny}")
    init, coef = setup(cfg)
    return cfg, Box(replace(cfg, **kw), init, coef), oracle_box(cfg, init)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ny", [3840, 3841, 3842, 4500])
def test_interpyy(ny, precision):
    cfg, g, o = _boxes(ny, precision=precision)
    got = g.interpyy()
    for f, which, out in (("u", 0, got[0]), ("w", 0, got[1]), ("v", 1, got[2])):
        # FP32: that of test_gpu_ydense.py for the banded solve
        ref = _oracle_interpyy(cfg, o, o.field(f), which)
        assert np.abs(out - ref).max() <= (2e-6 if precision else 1e-13) * np.abs(ref).max(), f


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ny", [3841, 3842, 4500])
def test_pois(ny, precision):
    """The velocity after the projection (the pressure takes a dt)."""
    cfg, g, o = _boxes(ny, precision=precision)
    for b in (g, o):
        b.pois(1)
    e = {n: rel_l2(g.field(n), o.field(n)) for n in "uvw"}
    print(ny, precision, e)
    assert max(e.values()) <= (1e-7 if precision else 1e-10), e


@pytest.mark.parametrize("ny", [8448, 8449, 9001])
def test_statsp(ny):
    cfg, g, o = _boxes(ny)
    g.statsp()
    e = _errors(g.stats()[0], o.statsp())
    print(ny, max(e, key=e.get), max(e.values()))
    assert max(e.values()) <= 1e-11, e
