"""The specular lobe's slope s (V.R)^(s-1) where (V.R)^s itself is below every float: a
grazing view whose geometry is exact in 32 bits (hit at the origin, light above it, V.R =
2^-20, s = 7.53125: (V.R)^s = 2^-150.6, (V.R)^(s-1) = 2^-130.6), with an image gradient large
enough that the light's gradient is an ordinary number."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tree", [False, True])
def test_slope_of_an_underflowed_lobe(ctx, tree):
    import torch
    v = np.array([[-32, -32, 0], [96, -32, 0], [-32, 96, 0]], np.float32)
    sc = scenes.SceneData(v, np.tile(np.float32([0, 0, 1]), (3, 1)), np.array([[0, 1, 2]]), np.zeros(1),
                          [scenes.material((0, 0, 0), 1.0, 7.53125, 0.0)], np.array([[0, 0, 1, 1, 1, 1]], np.float32))
    h = 2.0 ** -20
    cam = scenes.CameraData(*(np.array(a, np.float32) for a in ([1, 0, h], [-1, 0, -h], [0, 1, 0], [0, 0, 1])), 1, 1)
    d = api.DeviceScene(ctx, sc)
    paths = api.render(ctx, d, cam, 0, outputs=("paths",), tree_records=tree)["paths"]
    g = torch.full((1, 3), 2.0 ** 100, device="cuda")
    _, gl = api.render_backward(ctx, d, [cam], 0, paths, g, tree_records=tree)
    p = paths.cpu().numpy().reshape(1, -1)
    hits, masks = (p[:, 0:1], p[:, 1:2].view(np.uint32)) if tree else (p[:, :8], p[:, 8:].view(np.uint32))
    assert hits[0, 0] == 0 and masks[0, 0] == 0
    mats = sc.materials.astype(np.float64).copy()
    mats[:, 6] = np.log(mats[:, 6])
    _, _, want = oracle.Oracle(sc).frozen_f64([cam], 1, 1, 0.5, 0, hits, masks, mats, sc.lights.astype(np.float64),
                                              g=g.cpu().numpy().astype(np.float64), tree=tree)
    want = want[0, 3]
    assert abs(want + 3 * 2.0 ** 100 * 7.53125 * h ** 6.53125) <= 1e-9 * abs(want)  # -3 g s (V.R)^(s-1)
    # (V.R)^(s-1) and s times it are subnormal numbers of 18 bits or more: 2 x 2^-19, and powf's 4 ulp
    assert abs(gl.cpu().numpy()[0, 3] - want) <= 1e-5 * abs(want)
