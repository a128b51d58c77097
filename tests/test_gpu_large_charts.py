"""The FP32 node test on charts of many tiles. Its widening follows the cell's
own texture coordinates, not the largest of the whole chart: near the chart's
origin it admits the cells that the FP64 test admits, but for the few a ray
passes within the ray's own rounding of."""
import numpy as np
import pytest

import dmap_b200 as dm
from dmap_b200 import scenes

pytestmark = pytest.mark.gpu

ST_LEAF = 2


@pytest.mark.parametrize("n,tiles", [(32, 12000), (256, 1024), (1024, 64)])
def test_cells_near_the_origin_of_a_large_chart(n, tiles):
    """Within the first tile coordinates are at most 2, so a box is widened by
    some 2^-18 at most, under 1/250 of a cell (the smallest is 2^-10). A ray
    meets the cells it would miss by that only: a few of each thousand, times
    the sides of the cells on its way. 5% leaves room for the slab's rounding."""
    ctx = dm.Context(0)
    h = scenes.sine_noise_heights(n, 5, 0.2)
    asset = scenes.Asset(scenes.close_tile(h, repeat=True).astype(np.float32), repeat=True)
    s, z = float(tiles), [0.0, 0.0, 1.0]
    tri = np.concatenate([[0, 0, 0], [s, 0, 0], [0, s, 0], z, z, z, [0, 0], [s, 0], [0, s]])
    sc = scenes.Scene([asset], tri[None], np.zeros(1, np.int32), name="tiles", extent=s)
    dev = dm.Scene.from_synthetic(ctx, sc, keep_f64=True)
    rng = np.random.default_rng(n)
    p = np.zeros((2000, 3))
    p[:, :2] = rng.random((2000, 2))
    eye = p + np.array([0.0, 0.0, 0.6]) + 0.2 * rng.normal(size=p.shape)
    eye[:, 2] = 0.2 + np.abs(eye[:, 2])
    rays = np.zeros((2000, 8), np.float32)
    rays[:, 0:3], rays[:, 3:6], rays[:, 7] = eye, p - eye, np.inf
    ref, s64 = dev.intersect(rays, dm.TraversalOptions(precision="f64"), stats=True)
    opt = dm.TraversalOptions(schedule="simple", leaf_precision="f64")
    hits, s32 = dev.intersect(rays, opt, stats=True)
    assert np.array_equal(hits["tri"], ref["tri"]) and np.array_equal(hits["t"], ref["t"])
    assert (ref["tri"] >= 0).sum() > 1000
    assert s32[:, ST_LEAF].sum() <= 1.05 * s64[:, ST_LEAF].sum()
