"""Samples per pixel at the edges of the wavefront's sample mean: groups of 8, 16 and 32 lanes,
the first counts past a warp (33, 64) and mixes of them in one pass, chains and ray trees, on
ragged images whose last tiles hold padding paths."""
import numpy as np
import pytest

from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("both", [0, 3])
def test_plain_wavefront_and_batch_agree(ctx, both):
    import torch
    sc = scenes.small_random_scene(81, n_spheres=7, level=2, lights=2, refl=0.5, transparent=1, both=both)
    d = api.DeviceScene(ctx, sc)
    counts = [8, 16, 32, 33, 64, 1, 2, 4, 31]
    cams = [scenes.look_at((1.0, 2.5, 8.0 - 0.1 * k), (0, -0.5, 0), 55.0, 37 + 2 * k, 23 + k) for k in range(len(counts))]
    want = []
    for c, n in zip(cams, counts):
        a, b = (api.render(ctx, d, c, 2, 0.5, spp=n, jitter_seed=5, mode=m, outputs=("rgb",))["rgb"]
                for m in ("plain", "wavefront"))
        assert torch.equal(a, b), n
        want.append(a)
    jobs = [api.BatchJob(d, c, 2, 0.5, n, 5) for c, n in zip(cams, counts)]
    outs = api.make_batch_outputs(jobs, ("rgb",))
    api.render_batch(ctx, jobs, outs)
    assert all(torch.equal(o["rgb"], w) for o, w in zip(outs, want))
