"""Gradient sums of eos_render_backward at the edges of its reductions: one pixel, ragged
images, more lights than one warp sum holds components, and object counts on both sides of
what a block sums in shared memory (24 B per light + 28 B per object <= 32 KB).  Against the
FP64 adjoint, to the 1e-3 of the largest component that the other adjoint tests allow for the
FP32 forward pass."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _cards(n_obj, n_lights):
    """n_obj tilted triangles, an object each, in a square facing the camera."""
    rng = scenes.rng_for(17)
    side = int(np.ceil(np.sqrt(n_obj)))
    k = np.arange(n_obj)
    c = np.stack([k % side, k // side, np.zeros(n_obj)], 1) * (2.0 / side) - np.array([1.0, 1.0, 0.0])
    corner = np.array([[0, 0, 0], [1.9, 0, 0.1], [0, 1.9, 0.2]]) / side
    v = (c[:, None] + corner[None]).reshape(-1, 3)
    nrm = rng.normal(size=v.shape) * 0.2 + np.array([0, 0, 1.0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    mats = [scenes.material(rng.uniform(0.2, 1, 3), 0.3, float(rng.uniform(3, 40)), 0.0) for _ in range(n_obj)]
    lights = [[*rng.uniform([-2, -2, 1], [2, 2, 3]), *rng.uniform(0.2, 1, 3)] for _ in range(n_lights)]
    return scenes.SceneData(v, nrm, np.arange(3 * n_obj).reshape(-1, 3), k, mats, np.array(lights))


@pytest.mark.parametrize("n_obj,n_lights,w,h,spp", [(4, 1, 1, 1, 1), (9, 32, 33, 17, 1), (1169, 1, 61, 47, 1),
                                                    (1170, 1, 61, 47, 2), (30, 3, 257, 129, 1)])
def test_gradient_sums_match_fp64(ctx, n_obj, n_lights, w, h, spp):
    import torch
    sc = _cards(n_obj, n_lights)
    dsc = api.DeviceScene(ctx, sc)
    cams = [scenes.look_at((x, 0.05, 2.2), (0, 0, 0), 50.0, w, h) for x in (-0.1, 0.2)]
    r = [api.render(ctx, dsc, c, 0, spp=spp, jitter_seed=3, outputs=("rgb", "paths"), device=True) for c in cams]
    paths = torch.cat([x["paths"] for x in r])
    g = torch.from_numpy(np.random.default_rng(1).normal(size=(2 * w * h, 3)).astype(np.float32)).cuda()
    gm, gl = api.render_backward(ctx, dsc, cams, 0, paths, g, spp=spp, jitter_seed=3)
    mp = sc.materials.astype(np.float64).copy()
    mp[:, 6] = np.log(mp[:, 6])
    p = paths.cpu().numpy()
    assert (p[:, 0] >= 0).any()
    _, om, ol = oracle.Oracle(sc).frozen_f64(cams, w, h, 0.5, 0, p[:, :8], p[:, 8:].view(np.uint32), mp,
                                             sc.lights.astype(np.float64), g=g.cpu().numpy().astype(np.float64),
                                             spp=spp, jitter_seed=3)
    gm, gl = gm.cpu().numpy(), gl.cpu().numpy()
    for name, a, b in [("kd", gm[:, :3], om[:, :3]), ("ks", gm[:, 3:6], om[:, 3:6]), ("shininess", gm[:, 6], om[:, 6]),
                       ("colour", gl[:, :3], ol[:, :3]), ("position", gl[:, 3:], ol[:, 3:])]:
        assert np.abs(a - b).max() <= 1e-3 * max(np.abs(b).max(), 1e-12), name
