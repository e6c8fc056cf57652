"""The plain renderer at the image sizes where its lanes per warp change (4, 8, 16, 32 for
chains; 8, 16, 32 for ray trees, whose idle lanes take subtrees of the others): ragged images,
several samples and row bands give the wavefront renderer's bits, and a small one the
oracle's."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu

CHAIN = [(1, 1), (61, 47), (131, 143), (217, 171), (301, 250), (643, 481)]
TREE = [(3, 1), (61, 47), (385, 390), (389, 393), (1001, 605), (1203, 1031)]


@pytest.mark.parametrize("both,size", [(0, s) for s in CHAIN] + [(5, s) for s in TREE])
def test_plain_equals_wavefront_at_every_lane_count(ctx, both, size):
    import torch
    w, h = size
    sc = scenes.small_random_scene(63, n_spheres=12, level=2, lights=2, refl=0.6, transparent=3, both=both)
    dsc = api.DeviceScene(ctx, sc)
    cam = scenes.look_at((1.0, 3.0, 9.0), (0, -0.5, 0), 55.0, w, h)
    td = 4 if both else 3
    kw = dict(tree_records=True) if both and w * h < 200_000 else {}
    outs = ("rgb", "paths") if kw or not both else ("rgb",)
    a, b = (api.render(ctx, dsc, cam, td, mode=m, outputs=outs, **kw) for m in ("plain", "wavefront"))
    assert all(torch.equal(a[k], b[k]) for k in outs)
    for k in ("primary_rays", "shadow_rays", "secondary_rays", "shaded_hits"):
        assert a["stats"][k] == b["stats"][k], k
    if h > 2:  # a band of the frame, and two samples per pixel
        r = api.render(ctx, dsc, cam, td, outputs=("rgb",), rows=(1, h - 1))
        assert torch.equal(r["rgb"], a["rgb"][w:(h - 1) * w])
        s, t = (api.render(ctx, dsc, cam, td, spp=2, jitter_seed=4, mode=m, outputs=("rgb",))["rgb"]
                for m in ("plain", "wavefront"))
        assert torch.equal(s, t)
    if w == 61:
        orc = oracle.Oracle(sc)
        o = (orc.render_tree if both else orc.render)(cam, td, pixel_offset=0.5)
        assert np.abs(a["rgb"].cpu().numpy() - o["rgb"]).max() <= 1e-4


@pytest.mark.parametrize("n", [1, 5, 18_949, 37_901, 75_803])
def test_queries_at_every_lane_count(ctx, n):
    """Ray counts on both sides of the rule's steps, a last warp that is partly filled."""
    d = scenes.instanced_test_scene(5, n_instances=16)
    flat = scenes.small_random_scene(64, n_spheres=8, level=2)
    rng = np.random.default_rng(n)
    rays = np.concatenate([rng.uniform(-4, 4, (n, 3)), rng.normal(size=(n, 3))], 1).astype(np.float32)
    inst = api.InstancedScene(ctx, [api.DeviceScene(ctx, m) for m in d.meshes], d.instances, d.materials, d.lights)
    for scene, orc in ((api.DeviceScene(ctx, flat), oracle.Oracle(flat)), (inst, oracle.OracleInstanced(d))):
        ids, t = api.trace_closest(ctx, scene, rays)
        oid, ot, _ = orc.closest(rays)
        assert np.array_equal(ids, oid) and np.array_equal(t[ids >= 0], ot[oid >= 0])
        assert np.array_equal(api.trace_any(ctx, scene, rays), orc.any(rays))
