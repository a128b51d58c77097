"""The wavefront walk's groups of four lanes per ray, where they can go
wrong: batches that fill no warp, one warp and a ragged number of them;
triangle counts around the 32 boxes of a ballot and the last one of the
candidate mask; charts whose root level is past the 64 bits of open groups
(the wider bits), mirrored and off the cell lattice. Every record equals the
oracle's bit for bit with the FP64 leaf, in both orders."""
import ctypes as C

import numpy as np
import pytest

import dmap_b200 as dm
import py_oracle
import helpers
from dmap_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return dm.Context(0)


def _equal(cpu, dev, rays, order, rounds):
    ho, _ = cpu.intersect(rays, order=order)
    hd = dev.intersect(rays, dm.TraversalOptions(order=order, rounds=rounds, leaf_precision="f64"), np.float64)
    hit = ho[:, 10] >= 0
    assert np.array_equal(hd["tri"], np.where(hit, ho[:, 10], -1).astype(np.int32))
    assert np.array_equal(hd["t"][hit], ho[hit, 0]) and np.array_equal(hd["st"][hit], ho[hit, 1:3])
    assert np.array_equal(hd["ng"][hit], ho[hit, 5:8])
    assert np.array_equal(hd["i"][hit], ho[hit, 8].astype(np.int32))
    return int(hit.sum())


@pytest.mark.parametrize("order", ["nearest", "index"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 1025])
def test_batch_sizes(ctx, oracle, n, order):
    sc = helpers.small_sphere(16)
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc)
    rays = helpers.near_surface_rays(cpu, n, seed=n)
    for rounds in (0, 1, 2):
        _equal(cpu, dev, rays, order, rounds)


@pytest.mark.parametrize("order", ["nearest", "index"])
@pytest.mark.parametrize("tris", [2, 30, 32, 34, 254, 256])
def test_candidate_mask_edges(ctx, oracle, tris, order):
    sc = scenes.cube_sphere_scene(4, 5, patches=list(range(tris // 2)))
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc)
    assert dev.n_tri == tris
    rays = np.concatenate([helpers.near_surface_rays(cpu, 400, seed=tris), helpers.aimed_rays(cpu, 200)[0]])
    assert _equal(cpu, dev, rays, order, 2) > 100


@pytest.mark.parametrize("rounds", [0, 2])
@pytest.mark.parametrize("tiles", [1500, 3000, 12000])
def test_deep_charts(ctx, oracle, tiles, rounds):
    """A repeated 32 x 32 map over up to 12,000 tiles a side: root levels 15 (64 bits), 16 and 18."""
    h = scenes.sine_noise_heights(32, 5, 0.3)
    asset = scenes.Asset(scenes.close_tile(h, repeat=True).astype(np.float32), repeat=True)
    z = np.array([0.0, 0.0, 1.0])
    s = float(tiles)
    tri = np.concatenate([[0, 0, 0], [s, 0.1, 0], [0.2, s, 0], z, z, z, [0.3, 0.4], [s + 0.3, 0.7], [0.9, s + 0.4]])
    flip = np.concatenate([[0, 0, 3.0], [s, 0.1, 3.0], [0.2, s, 3.0], z, z, z, [0.3, 0.4], [0.9, s + 0.4],
                           [s + 0.3, 0.7]])
    sc = scenes.Scene([asset], np.stack([tri, flip]), np.zeros(2, np.int32), name="deep", extent=s)
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc)
    rng = np.random.default_rng(tiles)
    n = 300
    p = rng.random((n, 2)) * 0.45 * s
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:2], rays[:, 2] = p, rng.choice([-1.0, 1.5, 4.5], n)
    d = rng.normal(size=(n, 3))
    d[:, 2] = np.sign(1.5 - rays[:, 2] + 1e-3) * (0.3 + np.abs(d[:, 2]))
    rays[:, 3:6], rays[:, 7] = d, np.inf
    levels = {1500: 15, 3000: 16, 12000: 18}
    assert dev.triangle_info(0)[0] == levels[tiles]
    for order in ("nearest", "index"):
        assert _equal(cpu, dev, rays, order, rounds) > 100


@pytest.mark.parametrize("leaf", ["f32", "f64"])
@pytest.mark.parametrize("n", [1, 3, 8, 31, 500, 6000])
def test_leaf_rounds_agree(ctx, oracle, n, leaf):
    """The leaf kernel's batches (set up eight jobs at a time, searched by
    quads, records made in batches) against the last walk's inline leaves
    (rounds 0): the same records however the leaves are split, and the
    occlusion answers of the closest-hit query."""
    sc = helpers.small_sphere(32)
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc)
    rays = helpers.aimed_rays(cpu, n, seed=n)[0]
    base = dev.intersect(rays, dm.TraversalOptions(rounds=0, leaf_precision=leaf), np.float64)
    for rounds in (1, 2, 3):
        h = dev.intersect(rays, dm.TraversalOptions(rounds=rounds, leaf_precision=leaf), np.float64)
        assert np.array_equal(h.tobytes(), base.tobytes())
    for rounds in (0, 1, 2):
        o = dev.intersect(rays, dm.TraversalOptions(rounds=rounds, leaf_precision=leaf, mode="occluded"), np.float64)
        assert np.array_equal(o["tri"] >= 0, base["tri"] >= 0)


@pytest.mark.parametrize("cap", [1, 2, 3, 5, 9, 14, 22, 35])
def test_visit_cap_counts_cells_in_walk_order(ctx, oracle, cap):
    """A group is tested at once; the cap counts the cells the one-cell walk
    visits. The simple schedule counts them per root (at most 4 a triangle):
    what runs out there runs out here, what does not lasts here at 4 x cap."""
    sc = helpers.small_sphere(32)
    cpu, dev = py_oracle.CpuScene(oracle, sc), dm.Scene.from_synthetic(ctx, sc)
    rays = np.concatenate([helpers.near_surface_rays(cpu, 1500), helpers.aimed_rays(cpu, 500)[0]])
    rays = np.ascontiguousarray(rays, np.float32)

    def capped(schedule, c):
        o = dm.TraversalOptions(schedule=schedule, rounds=0, node_visit_cap=c, leaf_precision="f64").c()
        hits = np.empty(len(rays), dm.HIT64)
        st = dm.lib().dmap_intersect_host(dev.h, rays.ctypes.data, dm.F32, len(rays), C.byref(o), hits.ctypes.data,
                                          dm.F64, None)
        flags = (hits["flags"] & dm.HIT_CAPPED) != 0
        assert st == (6 if flags.any() else 0)  # DMAP_ERR_LIMIT
        return flags

    simple, wave, wide = capped("simple", cap), capped("wavefront", cap), capped("wavefront", 4 * cap)
    assert simple.any() and not (simple & ~wave).any() and not (wide & ~simple).any()
