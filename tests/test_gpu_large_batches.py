"""Batches large enough for what small ones cannot reach: walk rounds whose
picks wait for company (32 rays and more per warp), leaf rounds that take
sixteen jobs at a time and make hit records while the kernel runs, and visit
caps that run out before and after a park."""
import ctypes as C

import numpy as np
import pytest

import dmap_b200 as dm
import helpers
from dmap_b200 import scenes

pytestmark = pytest.mark.gpu

N = 300_000    # some 100 rays per warp of the walk, 150 jobs per warp of the leaves
SLICE = 10_000 # three rays per warp


def _rays(sc, n, seed):
    """Rays from around the surface toward random points of its base."""
    rng = np.random.default_rng(seed)
    p, m = scenes.base_points(sc, n, seed=seed)
    eye = p + rng.uniform(0.02, 1.0, (n, 1)) * m + 0.2 * rng.normal(size=(n, 3))
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 3:6], rays[:, 7] = eye, p - eye, np.inf
    return rays


@pytest.mark.parametrize("mode", ["closest", "occluded"])
@pytest.mark.parametrize("leaf", ["f32", "f64"])
@pytest.mark.parametrize("scene", ["mask", "tree"])
def test_large_batch_equals_its_slices(scene, leaf, mode):
    """A ray's answer does not depend on the batch: bit for bit that of the
    same ray in a batch of a few rays per warp, and with the FP64 leaf the
    closest hits are the simple schedule's."""
    ctx = dm.Context(0)
    sc = helpers.small_sphere(16) if scene == "mask" else scenes.cube_sphere_scene(4, 5, patches=list(range(150)))
    dev = dm.Scene.from_synthetic(ctx, sc)
    rays = _rays(sc, N, 7)
    opt = dm.TraversalOptions(leaf_precision=leaf, mode=mode)
    whole = dev.intersect(rays, opt)
    assert (whole["tri"] >= 0).sum() > N // 2
    parts = np.concatenate([dev.intersect(rays[k:k + SLICE], opt) for k in range(0, N, SLICE)])
    assert whole.tobytes() == parts.tobytes()
    if leaf == "f64" and mode == "closest":
        ref = dev.intersect(rays, dm.TraversalOptions(schedule="simple", leaf_precision=leaf))
        assert whole.tobytes() == ref.tobytes()


@pytest.mark.parametrize("rounds", [0, 1, 2])
@pytest.mark.parametrize("cap", [9, 30, 100])
def test_visit_cap_in_rounds(cap, rounds):
    """A ray whose cap did not run out has the uncapped query's record; one
    whose cap did keeps what it found, never anything nearer than the hit."""
    ctx = dm.Context(0)
    sc = helpers.small_sphere(32)
    dev = dm.Scene.from_synthetic(ctx, sc)
    rays = _rays(sc, 4000, 8)
    full = dev.intersect(rays, dm.TraversalOptions(rounds=rounds, leaf_precision="f64"))
    o = dm.TraversalOptions(rounds=rounds, leaf_precision="f64", node_visit_cap=cap).c()
    hits = np.empty(len(rays), dm.HIT64)
    st = dm.lib().dmap_intersect_host(dev.h, rays.ctypes.data, dm.F32, len(rays), C.byref(o), hits.ctypes.data, dm.F64,
                                      None)
    out = (hits["flags"] & dm.HIT_CAPPED) != 0
    assert st == (6 if out.any() else 0)  # DMAP_ERR_LIMIT
    assert cap > 30 or out.sum() > 100
    assert hits[~out].tobytes() == full[~out].tobytes()
    assert (hits["t"][out] >= full["t"][out]).all()
