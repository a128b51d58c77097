"""Occlusion queries of the FP32 wavefront: which root a ray's record holds.
The leaf rounds end a ray at the first root they accept, filtered or not; the
last walk finishes the leaf it is in, as the one-thread-per-ray schedule does."""
import numpy as np
import pytest

import dmap_b200 as dm
import helpers
import py_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return dm.Context(0)


def _rays(oracle, sc, n):
    cpu = py_oracle.CpuScene(oracle, sc)
    return np.concatenate([helpers.near_surface_rays(cpu, n, seed=5), helpers.aimed_rays(cpu, n, seed=6)[0]])


@pytest.mark.parametrize("leaf", ["f32", "f64"])
@pytest.mark.parametrize("order", ["nearest", "index"])
def test_last_walk_reports_the_leafs_nearest_root(ctx, oracle, order, leaf):
    """Rounds 0 (every leaf in the last walk) against the simple schedule, records bit for bit."""
    sc = helpers.small_sphere(16)
    dev = dm.Scene.from_synthetic(ctx, sc)
    rays = _rays(oracle, sc, 1500)
    opt = dict(order=order, leaf_precision=leaf, mode="occluded")
    a = dev.intersect(rays, dm.TraversalOptions(rounds=0, **opt))
    b = dev.intersect(rays, dm.TraversalOptions(schedule="simple", **opt))
    assert (a["tri"] >= 0).sum() > 1000
    assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("leaf", ["f32", "f64"])
@pytest.mark.parametrize("order", ["nearest", "index"])
def test_opaque_mask_keeps_occlusion_records(ctx, oracle, order, leaf):
    """A mask that rejects nothing leaves every occlusion record as it is."""
    sc = helpers.small_sphere(16)
    plain, masked = dm.Scene.from_synthetic(ctx, sc), dm.Scene.from_synthetic(ctx, sc)
    masked.set_opacity(np.ones((3, 5), np.uint8))
    rays = _rays(oracle, sc, 1500)
    for rounds in (0, 1, 2):
        opt = dm.TraversalOptions(order=order, rounds=rounds, leaf_precision=leaf, mode="occluded")
        a, b = plain.intersect(rays, opt), masked.intersect(rays, opt)
        assert (a["tri"] >= 0).sum() > 1000
        assert a.tobytes() == b.tobytes()
