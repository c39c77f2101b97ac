"""The CFL maxima of a step start from zero, also after a step whose products
ran and whose dt reduction did not (a launch between them that is refused)."""
import numpy as np
import pytest

from opentbl_b200 import Box, config, native
from opentbl_b200.config import replace

from helpers import setup

pytestmark = pytest.mark.gpu


def _rhsp_without_dt(b):
    """rhsp(1, setstep) as a graph in which k_dt is switched off, run once."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    s = drv.CUstream(b.stream)
    ok(drv.cuStreamBeginCapture(s, drv.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    b.rhsp(1, True)
    g = ok(drv.cuStreamEndCapture(s))
    n = ok(drv.cuGraphGetNodes(g))[1]
    nodes = ok(drv.cuGraphGetNodes(g, n))[0]
    exe = ok(drv.cuGraphInstantiate(g, 0))
    off = 0
    for node in nodes:
        if ok(drv.cuGraphNodeGetType(node)) != drv.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(drv.cuGraphKernelNodeGetParams(node))
        name = ok(drv.cuFuncGetName(p.func)) if int(p.func) else ok(drv.cuKernelGetName(p.kern))
        if b"4k_dt" in name:
            ok(drv.cuGraphNodeSetEnabled(exe, node, 0))
            off += 1
    assert off == 1
    ok(drv.cuGraphLaunch(exe, s))
    ok(drv.cuStreamSynchronize(s))
    ok(drv.cuGraphExecDestroy(exe))
    ok(drv.cuGraphDestroy(g))


@pytest.mark.parametrize("how", ["load", "rebind"])
@pytest.mark.parametrize("nz", [32, 512])  # nz = 512: the streamed kernels
def test_maxima_of_a_broken_step_do_not_last(nz, how):
    cfg = replace(config.TINY, nz=nz)
    init, coef = setup(cfg)
    ref, b = Box(cfg, init, coef), Box(cfg, init, coef)
    fast = dict(init, **{n: 3.0 * init[n] for n in "uvw"})
    b.load(fast)
    b.substep(1, True)  # a dt for the kernels after the products
    b.load(fast)
    _rhsp_without_dt(b)
    b.load(init) if how == "load" else b.rebind(cfg, init, coef)
    for x in (ref, b):
        x.rhsp(1, True)
    got, want = b.inflow()[1], ref.inflow()[1]
    for n in ("dt", "umax", "vmax", "wmax"):
        assert got[n] == want[n], n
    for n in native.FIELDS:
        np.testing.assert_array_equal(b.field(n), ref.field(n))
