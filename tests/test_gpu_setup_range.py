"""The per-triangle setup's height range, walked by a block over a shared
stack: the footprints where its batches change size (one cell, a few, more
straddling cells than the stack takes at once), charts off the cell lattice,
mirrored ones and repeated tiles. The record equals the oracle's bit for bit
(the range is a minimum and a maximum over the same cells)."""
import numpy as np
import pytest

import dmap_b200 as dm
import py_oracle
import helpers
from dmap_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 8, 64, 512, 1024])
def test_height_range_equals_the_oracle(oracle, n):
    ctx = dm.Context(0)
    sc = scenes.quad_scene(n) if n < 8 else helpers.chart_scene(n)
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc, keep_f64=True)
    for t in range(len(sc.tris)):
        assert np.array_equal(dev.triangle_info(t), cpu.triangle_info(t)[:11])
