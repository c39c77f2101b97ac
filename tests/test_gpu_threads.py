"""Contexts driven from different host threads (include/otbl.h): three boxes
whose kernels take different amounts of shared memory, each stepped, sampled
and captured into graphs by a thread of its own at the same time, end bit for
bit where the same calls end one box after the other."""
import threading
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from opentbl_b200 import Box, config
from opentbl_b200.config import replace
from opentbl_b200.ensemble import Graph

from helpers import setup

pytestmark = pytest.mark.gpu

STATE = ("u", "v", "w", "p", "rhsupa", "rhsvpa", "rhswpa")
ROUNDS = 12


def drive(cfg, init, coef, start=None):
    """A box's whole life on the calling thread: plain and replayed steps, a
    graph per round, statistics; returns its state and accumulators."""
    b = Box(cfg, init, coef)
    if start:
        start.wait()
    for _ in range(ROUNDS):
        b.advance(1)
        g = Graph([b], 2)
        g.launch()
        g.sync()
        g.close()
        b.statsp()
    b.sync()
    out = {n: b.field(n) for n in STATE}
    out["stats"] = b.stats()[0]
    b.close()
    return out


def test_three_threads_equal_alone():
    # the kernels of 513 planes and of 129 rows take more than 48 KB where those
    # of the smallest box take less
    boxes = []
    for nx, ny, nz in ((33, 41, 32), (513, 41, 32), (65, 129, 64)):
        cfg = replace(config.TINY, nx=nx, ny=ny, nz=nz, lx=12.0 * nx / 33, name=f"thread-{nx}")
        boxes.append((cfg, *setup(cfg)))
    alone = [drive(*b) for b in boxes]
    start = threading.Barrier(len(boxes), timeout=120)
    with ThreadPoolExecutor(len(boxes)) as pool:
        mix = [f.result() for f in [pool.submit(drive, *b, start) for b in boxes]]
    for a, m in zip(alone, mix):
        for n in a:
            np.testing.assert_array_equal(m[n], a[n])
