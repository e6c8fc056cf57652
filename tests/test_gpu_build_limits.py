"""Builds whose blocks give up waiting for an earlier block's sum (the test limit of
eos_ctx_set_build_polls, no fault or hang): the call returns EOS_ERR_TIMEOUT and makes no
scene, and the same context then builds the same bytes as one that never had a limit."""
import numpy as np
import pytest

from eos_b200 import api
from eos_b200._lib import EosError
from tests.test_gpu_ploc import _equal_triangles

pytestmark = pytest.mark.gpu

TIMEOUT = 4


def _bytes(d, path):
    d.save(path)
    raw = path.read_bytes()
    return raw[:56] + raw[60:]  # without the build time


# clustering rounds of 224 and 480 triangles a tile, levels of 256 nodes a tile
@pytest.mark.parametrize("builder,n", [("ploc", 1121), ("ploc", 40_000), ("ploc", 150_000), ("lbvh", 9_000),
                                       ("lbvh", 150_000)])
def test_build_that_gives_up_ends_with_its_status(tmp_path, builder, n):
    sc = _equal_triangles(np.random.default_rng(n).normal(size=(n, 3)) * 10.0)
    kw = dict(builder=builder, leaf_size=1)
    with_limits, without = api.Context(0), api.Context(0)
    try:
        want = _bytes(api.DeviceScene(without, sc, **kw), tmp_path / "a.eos")
        for polls in (0, 1, 0, 8, 200, 0):
            with_limits.set_build_polls(polls)
            try:
                d = api.DeviceScene(with_limits, sc, **kw)
            except EosError as e:
                assert e.code == TIMEOUT
            else:  # with some polls every sum may come in time
                assert polls > 0 and _bytes(d, tmp_path / "b.eos") == want
                d.close()
            with_limits.set_build_polls()
            d = api.DeviceScene(with_limits, sc, **kw)
            assert d.info()["builder"] == (2 if builder == "ploc" else 1)
            assert _bytes(d, tmp_path / "b.eos") == want
            d.close()
    finally:
        with_limits.close()
        without.close()
