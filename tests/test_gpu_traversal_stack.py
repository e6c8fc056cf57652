"""Rays whose traversal stack passes its shared-memory column several times over: thin
triangles piled on one another, leaves of one triangle, every column size.  Hit ids and
paths equal the oracle's, flat and as instances, in both modes."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _pile(n):
    rng = scenes.rng_for(91)
    V, N, F = scenes.foliage_cluster(n, rng, radius=0.3)  # edges up to 1 in a ball of radius 0.3
    mats = [scenes.material((0.5, 0.4, 0.3), 0.2, 16, 0.4)]
    lights = [[2, 3, 4, 1, 1, 1], [-3, 2, 1, 1, 1, 1]]
    return scenes.SceneData(V, N, F, np.zeros(len(F)), mats, np.array(lights))


@pytest.mark.parametrize("stack", [8, 16, 32])
@pytest.mark.parametrize("width,instanced", [(4, False), (2, False), (4, True)])
def test_deep_stacks_match_oracle(ctx, stack, width, instanced):
    sc = _pile(4000)
    cam = scenes.look_at((0.3, 0.4, 1.5), (0, 0, 0), 50.0, 67, 45)
    mesh = api.DeviceScene(ctx, sc, leaf_size=1, layout="fixed", width=width)
    scene, orc = mesh, oracle.Oracle(sc)
    if instanced:
        places = [(0, np.hstack([np.eye(3), np.array([[0.1 * k], [0.05 * k], [-0.2 * k]])]), 0) for k in range(5)]
        d = scenes.InstancedData([sc], places, sc.materials, sc.lights)
        scene = api.InstancedScene(ctx, [mesh], d.instances, d.materials, d.lights)
        orc = oracle.OracleInstanced(d)
    o = orc.render(cam, 2, pixel_offset=0.5)
    assert (o["hits"][:, 0] >= 0).mean() > 0.3
    for mode in ("plain", "wavefront"):
        g = api.render(ctx, scene, cam, 2, pixel_offset=0.5, mode=mode, outputs=("paths",), device=False,
                       stack_depth=stack)
        assert np.array_equal(g["paths"][:, :8], o["hits"]), mode
        assert np.array_equal(g["paths"][:, 8:].view(np.uint32), o["shadows"]), mode
