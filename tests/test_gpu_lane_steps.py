"""Both sides of every step of the plain renderer's and the ray queries' lanes-per-warp rule:
the largest frame or ray count of each lane count and the smallest of the next."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _full():
    import torch
    return 28 * torch.cuda.get_device_properties(0).multi_processor_count  # warps of the rule


def _size(tiles):
    """A frame of that many 8x4 tiles, its last column and row started only."""
    a = max(k for k in range(1, int(tiles ** 0.5) + 1) if tiles % k == 0)
    return 8 * a - 3, 4 * (tiles // a) - 1


@pytest.mark.parametrize("both,warps,lanes", [(0, 1, 4), (0, 1, 8), (0, 1, 16), (5, 4, 8), (5, 8, 16)])
@pytest.mark.parametrize("over", [0, 1])
def test_frames(ctx, both, warps, lanes, over):
    import torch
    most = lanes * (warps * _full() + 1) - 1  # pixels of the largest frame with `lanes` lanes
    w, h = _size(most // 32 + over)
    sc = scenes.small_random_scene(63, n_spheres=12, level=2, lights=2, refl=0.6, transparent=3, both=both)
    d = api.DeviceScene(ctx, sc)
    cam = scenes.look_at((1.0, 3.0, 9.0), (0, -0.5, 0), 55.0, w, h)
    a, b = (api.render(ctx, d, cam, 3, mode=m, outputs=("rgb",)) for m in ("plain", "wavefront"))
    assert torch.equal(a["rgb"], b["rgb"])
    for k in ("primary_rays", "shadow_rays", "secondary_rays", "shaded_hits"):
        assert a["stats"][k] == b["stats"][k], k


@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("over", [0, 1])
def test_queries(ctx, lanes, over):
    n = lanes * (_full() + 1) - 1 + over
    sc = scenes.small_random_scene(64, n_spheres=8, level=2)
    rng = np.random.default_rng(n)
    rays = np.concatenate([rng.uniform(-4, 4, (n, 3)), rng.normal(size=(n, 3))], 1).astype(np.float32)
    d, orc = api.DeviceScene(ctx, sc), oracle.Oracle(sc)
    ids, t = api.trace_closest(ctx, d, rays)
    oid, ot, _ = orc.closest(rays)
    assert np.array_equal(ids, oid) and np.array_equal(t[ids >= 0], ot[oid >= 0])
    assert np.array_equal(api.trace_any(ctx, d, rays), orc.any(rays))
