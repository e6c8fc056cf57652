"""PLOC trees at the sizes where the builder's rounds change: one block's last rounds only
(at most 1,024 clusters), one more, whole and started tiles of 224 and 480 clusters, and the
count at which tiles change.  Every triangle's record position equals the restatement's, in
ragged clouds and where all areas tie (rounds that merge nothing)."""
import numpy as np
import pytest

from eos_b200 import api
from oracle import ploc as oracle_ploc
from tests.test_gpu_ploc import _equal_triangles, _pos_of_id

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 33, 1024, 1025, 1120, 1121, 2 * 224 * 5 + 1, 224 * 148, 224 * 148 + 1, 480 * 71 + 7])
@pytest.mark.parametrize("spread", ["cloud", "half at one place"])
def test_record_positions_match_restatement(ctx, tmp_path, n, spread):
    rng = np.random.default_rng(n)
    c = rng.normal(size=(n, 3)) * 10.0
    if spread != "cloud":
        c[: min(n // 2, 90)] = 0.25  # their areas tie; a chain of 90 stays within the refit's depth
    sc = _equal_triangles(c)
    d = api.DeviceScene(ctx, sc, builder="ploc", leaf_size=2)
    _, order = d.morton()
    lo, hi = oracle_ploc.leaf_boxes(sc.verts, sc.tris, order)
    _, _, position = oracle_ploc.build(lo, hi)
    d.save(tmp_path / "s.eos")
    expect = np.empty(n, np.int64)
    expect[order.astype(np.int64)] = position
    got = _pos_of_id(tmp_path / "s.eos")
    if d.info()["builder"] == 2:
        assert np.array_equal(got, expect)
    else:  # deeper than the refit walks: the LBVH's order
        assert spread != "cloud" and np.array_equal(got[order.astype(np.int64)], np.arange(n))
