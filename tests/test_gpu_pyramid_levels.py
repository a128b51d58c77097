"""The pyramid build without KEEP_F64 holds the FP64 levels from the first
tile's top on only. Its FP32 levels are those of the build that keeps all of
them, at the sizes around a tile (16) and a fold launch (256)."""
import numpy as np
import pytest

import dmap_b200 as dm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build", ["fold", "direct"])
@pytest.mark.parametrize("n", [1, 2, 8, 16, 32, 256, 512])
def test_fp32_levels_do_not_depend_on_what_is_kept(n, build):
    ctx = dm.Context(0)
    h = np.random.default_rng(n).random((n + 1, n + 1)).astype(np.float32)
    kept = dm.Asset(ctx, h, 0.3, 0.1, keep_f64=True, build=build)
    plain = dm.Asset(ctx, h, 0.3, 0.1, keep_f64=False, build=build)
    assert kept.n_levels == plain.n_levels
    for level in range(kept.n_levels):
        a, b = kept.level(level, "f32"), plain.level(level, "f32")
        assert all(np.array_equal(a[c], b[c]) for c in a)
