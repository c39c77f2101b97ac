"""otbl_advance replays small boxes' steps from a CUDA graph after three plain
ones (otbl_capi.cu step_graph); whatever changes a step's launches drops it.
The same box advanced in one call, and step by step over changes of the CTA tiles
and a rebind of its state arrays, ends bit for bit where plain otbl_substep calls
end."""
import numpy as np
import pytest

from opentbl_b200 import Box, config
from opentbl_b200.config import replace
from opentbl_b200.ensemble import Graph

from helpers import setup

pytestmark = pytest.mark.gpu

STATE = ("u", "v", "w", "p", "rhsupa", "rhsvpa", "rhswpa")


def test_replay_is_the_step():
    torch = pytest.importorskip("torch")

    # the last chunks hold 3 planes, 3 (v) and 4 (u, w) rows
    cfg = replace(config.SMALL, nx=73, ny=59)
    init, coef = setup(cfg)
    plain, once, split = (Box(cfg, init, coef) for _ in range(3))
    for _ in range(12):
        for m in (1, 2, 3):
            plain.substep(m, m == 1)
    l0 = once.launches
    once.advance(3)
    per = (once.launches - l0) / 3
    once.advance(9)
    assert once.launches - l0 == 12 * per  # replayed kernels are counted too
    assert once.replays == 9
    split.advance(5)
    assert split.replays == 2
    for tile in (64, 32):  # half and quarter tiles: plain steps, not the old graph
        split.set_tuning((tile,) * 3)
        split.advance(2)
    assert split.replays == 2
    split.set_tuning((128,) * 3)
    split.sync()
    own = {n: torch.from_numpy(split.field(n)).cuda() for n in STATE}
    torch.cuda.synchronize()
    split.bind_state({n: t.data_ptr() for n, t in own.items()})
    for _ in range(3):
        split.advance(1)
    for b in (plain, once, split):
        b.sync()
    for n in STATE:
        # tiempo enters genflu's filter only through its < 20 window here, so
        # plain substeps (which do not advance it) agree too
        np.testing.assert_array_equal(once.field(n), plain.field(n))
        np.testing.assert_array_equal(split.field(n), plain.field(n))


def test_captured_steps_are_not_plain_steps():
    """A graph of four steps records them without running them, so the next
    three plain steps build no step graph; the fourth replays one."""
    cfg = config.TINY
    b = Box(cfg, *setup(cfg))
    g = Graph([b], 4)
    g.launch()
    g.sync()
    b.advance(3)
    b.sync()
    assert b.replays == 0
    b.advance(2)
    b.sync()
    assert b.replays == 2
    g.close()


def test_replay_after_rebind():
    """The step captured for one box is not replayed for the box that the
    context is re-bound to."""
    a = config.TINY
    c = replace(a, lx=14.0, lz=5.0, re_theta=350.0)
    b, fresh = Box(a, *setup(a)), Box(c, *setup(c))
    b.advance(5)
    b.sync()
    assert b.replays == 2
    b.rebind(c, *setup(c))
    b.advance(3)
    b.sync()  # the old step graph is destroyed once the stream is idle
    b.advance(2)
    assert b.replays == 4
    fresh.advance(5)
    for x in (b, fresh):
        x.sync()
    for n in STATE:
        np.testing.assert_array_equal(b.field(n), fresh.field(n))
