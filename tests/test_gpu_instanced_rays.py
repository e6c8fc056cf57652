"""Rays that a two-level scene's traversal cannot take in its fma box test's form: parallel to
an axis in world space, in an instance's object space (quarter turns) or in both, and ones
whose |o / d| passes its limit.  Nearest hits, any hits and whole frames equal the oracle's."""
import numpy as np
import pytest

import oracle
from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _quarter_turns():
    rng = scenes.rng_for(23)
    v, f = scenes.icosphere(2)
    V, N, F = scenes.foliage_cluster(300, rng, radius=0.8)
    unused = [scenes.material((0.5, 0.5, 0.5), 0.2, 16, 0.0)]
    meshes = [scenes.SceneData(v, v, f, np.zeros(len(f)), unused, np.zeros((0, 6))),
              scenes.SceneData(V, N, F, np.zeros(len(F)), unused, np.zeros((0, 6)))]
    places, mats = [], []
    for k in range(14):
        M = np.zeros((3, 4))
        if k % 3 < 2:  # a signed permutation of the axes: exactly representable
            M[np.arange(3), rng.permutation(3)] = rng.choice([-1.0, 1.0], 3)
        else:
            M[:, :3] = scenes.random_rotation(rng)
        M[:, 3] = rng.uniform(-2.5, 2.5, 3)
        places.append((k % 2, M, k))
        mats.append(scenes.material(rng.uniform(0.2, 1, 3), 0.3, 16, 0.4 * (k % 2)))
    return scenes.InstancedData(meshes, places, np.array(mats), np.array([[1, 6, 2, 1, 1, 1], [0, 0, 7.0, 1, 1, 1]]))


def _scene(ctx, d):
    return api.InstancedScene(ctx, [api.DeviceScene(ctx, m) for m in d.meshes], d.instances, d.materials, d.lights)


@pytest.mark.parametrize("small", [0.0, -0.0, 1e-31, 1e-36])
def test_axis_parallel_queries_match_oracle(ctx, small):
    d = _quarter_turns()
    rng = np.random.default_rng(5)
    n = 3000
    o = rng.uniform(-4, 4, (n, 3))
    dirs = np.full((n, 3), small)
    axis = rng.integers(3, size=n)
    dirs[np.arange(n), axis] = rng.choice([-1.0, 1.0], n)
    two = rng.random(n) < 0.3  # parallel to a plane only
    dirs[two, (axis[two] + 1) % 3] = rng.normal(size=two.sum())
    rays = np.concatenate([o, dirs], 1).astype(np.float32)
    scene, orc = _scene(ctx, d), oracle.OracleInstanced(d)
    ids, t = api.trace_closest(ctx, scene, rays)
    oid, ot, _ = orc.closest(rays)
    assert np.array_equal(ids, oid) and np.array_equal(t[ids >= 0], ot[oid >= 0])
    assert np.array_equal(api.trace_any(ctx, scene, rays), orc.any(rays))
    assert (ids >= 0).mean() > 0.1


@pytest.mark.parametrize("w,h", [(64, 48), (65, 49)])
def test_axis_aligned_view_matches_oracle(ctx, w, h):
    d = _quarter_turns()
    cam = scenes.look_at((0, 0, 7.0), (0, 0, 0), 60.0, w, h)  # columns and rows of parallel rays
    scene = _scene(ctx, d)
    for off in (0.0, 0.5):
        o = oracle.OracleInstanced(d).render(cam, 2, pixel_offset=off)
        for mode in ("plain", "wavefront"):
            g = api.render(ctx, scene, cam, 2, pixel_offset=off, mode=mode, outputs=("paths",), device=False)
            assert np.array_equal(g["paths"][:, :8], o["hits"]), (mode, off)
            assert np.array_equal(g["paths"][:, 8:].view(np.uint32), o["shadows"]), (mode, off)
