"""The walk's shared memory grows with the triangles of a scene behind the
candidate mask (up to 256), past the size that needs no opt-in. The opt-in
belongs to the kernel, not to the scene."""
import subprocess
import sys
import threading
from pathlib import Path

import pytest
import torch

import dmap_b200 as dm
from dmap_b200 import scenes

pytestmark = pytest.mark.gpu


def test_threads_with_scenes_of_different_sizes():
    """Two contexts in two threads, scenes of 170 and 256 triangles: no launch
    is refused because the other thread's scene is smaller."""
    errors, barrier = [], threading.Barrier(2)

    def work(tris):
        try:
            ctx = dm.Context(0)
            dev = dm.Scene.from_synthetic(ctx, scenes.cube_sphere_scene(4, 5, patches=list(range(tris // 2))))
            rays = torch.tensor([[0, 0, 3.0, 0, 0, -1, 0, float("inf")]], device="cuda")
            hits = torch.empty(12, dtype=torch.int32, device="cuda")
            stream, opt = torch.cuda.Stream(), dm.TraversalOptions(rounds=0)
            torch.cuda.synchronize()
            barrier.wait(60)
            for k in range(20000):
                dev.intersect_device(rays.data_ptr(), dm.F32, 1, hits.data_ptr(), dm.F32, opt, stream=stream.cuda_stream)
                if k % 500 == 0:
                    stream.synchronize()
            stream.synchronize()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((tris, str(e)))

    threads = [threading.Thread(target=work, args=(n,)) for n in (170, 256)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


_FRESH = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[2])
import dmap_b200 as dm
from dmap_b200 import scenes
n = int(sys.argv[1])
sc = scenes.cube_sphere_scene(4, 5, patches=list(range(128)))
sc = scenes.Scene(sc.assets, sc.tris[:n], sc.tri_asset[:n], name="part", extent=sc.extent)
dev = dm.Scene.from_synthetic(dm.Context(0), sc)
assert dev.n_tri == n
rng = np.random.default_rng(n)
rays = np.zeros((600, 8), np.float32)
rays[:, 0:3] = 2.0 * scenes.uniform_direction(rng, 600)
rays[:, 3:6], rays[:, 7] = -rays[:, 0:3], np.inf
for order in ("nearest", "index"):
    ref = dev.intersect(rays, dm.TraversalOptions(order=order, schedule="simple", leaf_precision="f64"))
    assert (ref["tri"] >= 0).sum() > 100
    for rounds in (0, 2):
        h = dev.intersect(rays, dm.TraversalOptions(order=order, rounds=rounds, leaf_precision="f64"))
        assert h.tobytes() == ref.tobytes()
"""


@pytest.mark.parametrize("tris", [156, 157, 160, 161, 225, 252, 253, 256])
def test_sizes_in_a_fresh_process(tris):
    """Each size as the first of its process, which no larger scene's opt-in
    helps: every record equals the simple schedule's."""
    root = Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", _FRESH, str(tris), str(root)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
