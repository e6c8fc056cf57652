"""A batch of more paths than the device has queue memory for in one chunk: the chunks get
smaller (2^24 paths instead of up to 2^25) and the images stay the same."""
import numpy as np
import pytest

from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def test_batch_renders_where_its_largest_chunk_does_not_fit(ctx):
    """17 views of 1080p (35M paths) at 232 B of queues a path: 7.7 GB in chunks of 2^25
    paths, 3.9 GB in chunks of 2^24; 5.5 GB are left free."""
    import torch
    own = api.Context(0)
    hog = None
    try:
        d = api.DeviceScene(own, scenes.small_random_scene(71, n_spheres=5, level=3, lights=1, refl=0.6))
        cams = [scenes.look_at((4 * np.cos(a), 2.5, 4 * np.sin(a) + 4), (0, -0.5, 0), 55.0, 1920, 1080)
                for a in np.linspace(0.2, 2.9, 17)]
        jobs = [api.BatchJob(d, c, 1, 0.5) for c in cams]
        outs = api.make_batch_outputs(jobs, ("rgba8",))
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        leave = int(5.5 * 2**30)
        assert free > leave
        hog = torch.empty(free - leave, dtype=torch.uint8, device="cuda")
        for _ in range(2):  # capture, then replay
            st = api.render_batch(own, jobs, outs)
        assert st["primary_rays"] == 17 * 1920 * 1080 and st["secondary_rays"] > 0
        hog = None
        torch.cuda.empty_cache()
        for c, o in zip(cams, outs):
            assert torch.equal(o["rgba8"], api.render(ctx, d, c, 1, 0.5, outputs=("rgba8",))["rgba8"])
    finally:
        del hog
        own.close()
        torch.cuda.empty_cache()
