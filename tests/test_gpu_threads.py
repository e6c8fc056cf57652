"""Several contexts, threads and streams: scenes are freed and scratch grows while another
thread captures a graph or has an asynchronous batch in flight, a context works on a caller's
stream, and two contexts render and rebuild at once.  The results are the bits of a context
that works alone."""
import threading

import numpy as np
import pytest

from eos_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _scene(k, spheres=6):
    return scenes.small_random_scene(k, n_spheres=spheres, level=3, lights=2, refl=0.5)


def _cam(w, h, a=0.7):
    return scenes.look_at((5 * np.cos(a), 2.5, 5 * np.sin(a)), (0, -0.5, 0), 55.0, w, h)


def _in_thread(fn):
    """Runs fn in a thread and raises what it raised."""
    failed = []

    def body():
        try:
            fn()
        except BaseException as e:  # noqa: BLE001 -- handed to the caller
            failed.append(e)

    t = threading.Thread(target=body)
    t.start()
    return t, failed


def test_free_and_growth_while_another_thread_captures(ctx):
    """A scene's end and a scratch buffer's growth neither fail in, nor end, another thread's
    stream capture."""
    import torch
    other = api.Context(0)
    try:
        d = api.DeviceScene(other, _scene(1))
        rgb = api.render(other, d, _cam(64, 48), 1, outputs=("rgb",), device=False)["rgb"]
        assert rgb.any()
        spare = api.DeviceScene(other, _scene(2))

        def work():
            assert other.lib.eos_scene_destroy(spare.h) == 0
            spare.h = None
            big = api.render(other, d, _cam(320, 240), 1, outputs=("rgb",), device=False)["rgb"]  # grows out.rgb
            assert big.any()

        x = torch.zeros(1024, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            x.add_(1)
            t, failed = _in_thread(work)
            t.join()
            x.add_(1)
        assert not failed, failed
        g.replay()
        torch.cuda.synchronize()
        assert bool((x == 2).all())
    finally:
        other.close()


def test_scene_ends_while_another_context_renders_it(ctx):
    """A scene destroyed right behind another context's asynchronous batch: the batch ends
    before the scene's memory is given to the next scene."""
    import torch
    a, b = api.Context(0), api.Context(0)
    try:
        cams = [_cam(640, 480, 0.3 * k) for k in range(6)]
        want = []
        for round_ in range(3):
            d = api.DeviceScene(a, _scene(3, spheres=12))
            jobs = [api.BatchJob(d, c, 3) for c in cams]
            outs = [{"rgba8": torch.zeros((c.height, c.width, 4), dtype=torch.uint8).pin_memory().numpy()} for c in cams]
            if not want:
                api.render_batch(b, jobs, outs)
                want = [o["rgba8"].copy() for o in outs]
                for o in outs:
                    o["rgba8"][:] = 0
            api.render_batch(b, jobs, outs, async_outputs=True)
            d.close()
            again = [api.DeviceScene(a, _scene(40 + k, spheres=12)) for k in range(2)]
            b.synchronize()
            assert all(np.array_equal(o["rgba8"], w) for o, w in zip(outs, want)), round_
            for s in again:
                s.close()
    finally:
        b.close()
        a.close()


@pytest.mark.parametrize("builder", ["ploc", "lbvh"])
def test_callers_stream(ctx, tmp_path, builder):
    """Build, render, batch, gradients, queries, rebuild and growth on a caller's stream and
    back on the context's own: the bits of a context that never changed streams."""
    import torch

    def all_of(c, k):
        d = api.DeviceScene(c, _scene(50 + k, spheres=4 + 20 * k), builder=builder)
        d.save(tmp_path / "s.eos")
        raw = (tmp_path / "s.eos").read_bytes()
        cam = _cam(96 + 64 * k, 72)
        f = api.render(c, d, cam, 2, outputs=("rgb", "paths"), device=False)
        w = api.render(c, d, cam, 2, outputs=("rgb",), mode="wavefront", device=False)
        out = [{"rgb": np.zeros((cam.width * cam.height, 3), np.float32)}]
        api.render_batch(c, [api.BatchJob(d, cam, 2)], out)
        rays = np.random.default_rng(k).normal(size=(3001 * (k + 1), 6)).astype(np.float32)
        ids, t = api.trace_closest(c, d, rays)
        occ = api.trace_any(c, d, rays)
        gm, gl = api.render_backward(c, d, [cam], 2, f["paths"], np.ones_like(f["rgb"]), device=False)
        d.close()
        assert np.isfinite(gm).all() and np.isfinite(gl).all() and gm.any()
        return [raw[:56] + raw[60:], f["rgb"], f["paths"], w["rgb"], out[0]["rgb"], ids, t, occ]

    alone, moved = api.Context(0), api.Context(0)
    try:
        want = [all_of(alone, k) for k in range(3)]
        streams = [torch.cuda.Stream().cuda_stream, None, torch.cuda.Stream().cuda_stream]
        for order in ((0, 1, 2), (2, 0, 1)):
            for k, s in zip(order, streams):
                moved.set_stream(s)
                got = all_of(moved, k)
                assert got[0] == want[k][0]
                assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(got[1:], want[k][1:]))
    finally:
        moved.close()
        alone.close()


def test_two_contexts_on_two_threads(ctx):
    """One thread captures batches of ever new shapes while the other builds, renders and
    frees scenes."""
    import torch
    a, b = api.Context(0), api.Context(0)
    try:
        d = api.DeviceScene(a, _scene(7))
        cams = [_cam(64 + 8 * k, 48 + 4 * k) for k in range(24)]
        want = [api.render(ctx, d, c, 2, outputs=("rgb",), device=False)["rgb"] for c in cams]
        first = api.DeviceScene(b, _scene(8, spheres=20))
        ref = api.render(b, first, _cam(80, 60), 1, outputs=("rgb",), device=False)["rgb"]
        first.close()
        torch.cuda.synchronize()

        def rebuild():
            for k in range(40):
                s = api.DeviceScene(b, _scene(8, spheres=20))
                r = api.render(b, s, _cam(80, 60), 1, outputs=("rgb",), device=False)["rgb"]
                assert np.array_equal(r, ref), k
                assert b.lib.eos_scene_destroy(s.h) == 0
                s.h = None

        t, failed = _in_thread(rebuild)
        try:
            for c, w in zip(cams, want):
                out = [{"rgb": np.zeros((c.width * c.height, 3), np.float32)}]
                api.render_batch(a, [api.BatchJob(d, c, 2)], out)
                assert np.array_equal(out[0]["rgb"], w)
        finally:
            t.join()
        assert not failed, failed
    finally:
        b.close()
        a.close()
