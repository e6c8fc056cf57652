"""Wavefront passes of several chunks.  32 lights and trace depth 7 take 2,312 B of queues a
path, so the 16 GB rule cuts a pass after 7.4M paths: at a job's end (four 1080p views) and
inside a job (a 4K view), two lanes per chunk, the bounces' buffers and events used again."""
import numpy as np
import pytest

from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,spp", [([(1920, 1080)] * 4, 1), ([(3840, 2160), (333, 251)], 1),
                                       ([(961, 541), (1101, 1003)], 5)])
def test_chain_pass_of_several_chunks(ctx, sizes, spp):
    import torch
    sc = scenes.small_random_scene(73, n_spheres=6, level=2, lights=32, refl=0.5)
    assert sc.n_lights == 32
    d = api.DeviceScene(ctx, sc)
    paths = sum(-(-w // 8) * -(-h // 4) * 32 * spp for w, h in sizes)
    assert paths > (16 << 30) // (2 * 32 + 2 * (36 + 32 * 32) + 16 * 8)
    cams = [scenes.look_at((4 * np.cos(0.5 * k), 2.5, 4 * np.sin(0.5 * k) + 4), (0, -0.5, 0), 55.0, w, h)
            for k, (w, h) in enumerate(sizes)]
    jobs = [api.BatchJob(d, c, 7, 0.5, spp, 9) for c in cams]
    outs = api.make_batch_outputs(jobs, ("rgb",))
    for _ in range(2):  # capture, then replay
        for o in outs:
            o["rgb"].fill_(-1.0)
        st = api.render_batch(ctx, jobs, outs)
    want = [api.render(ctx, d, c, 7, 0.5, spp=spp, jitter_seed=9, outputs=("rgb",)) for c in cams]
    assert all(torch.equal(o["rgb"], w["rgb"]) for o, w in zip(outs, want))
    for k in ("primary_rays", "shadow_rays", "secondary_rays", "shaded_hits"):
        assert st[k] == sum(w["stats"][k] for w in want), k
