"""The walk's shared memory grows with the triangles of a scene behind the
candidate mask (up to 256), past the size that needs no opt-in. The opt-in
belongs to the kernel, not to the scene."""
import threading

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
