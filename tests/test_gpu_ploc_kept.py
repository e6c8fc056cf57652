"""The PLOC builder keeps its tree wherever the restatement's is shallow enough for the
traversal (depth + 2 <= 96), also through rounds that merge nothing and forced rounds: a tree
that it lost there would come back as an LBVH, which renders the same."""
import numpy as np
import pytest

from eos_b200 import api
from oracle import ploc as oracle_ploc
from tests.test_gpu_ploc import _equal_triangles, _pos_of_id

pytestmark = pytest.mark.gpu


def _depth(child, n):
    level = np.zeros(2 * n - 1, np.int64)
    for k in range(n - 2, -1, -1):  # parents are made after their children
        level[child[k]] = level[k] + 1
    return int(level.max())


@pytest.mark.parametrize("n", [2, 33, 1024, 1121, 2 * 224 * 5 + 1, 224 * 148 + 1])
@pytest.mark.parametrize("same", [0, 40, 90, 300])
def test_builder_stays_where_the_restated_tree_is_shallow(ctx, tmp_path, n, same):
    c = np.random.default_rng(n).normal(size=(n, 3)) * 10.0
    c[: min(n // 2, same)] = 0.25
    sc = _equal_triangles(c)
    d = api.DeviceScene(ctx, sc, builder="ploc", leaf_size=2)
    _, order = d.morton()
    child, _, position = oracle_ploc.build(*oracle_ploc.leaf_boxes(sc.verts, sc.tris, order))
    assert (d.info()["builder"] == 2) == (_depth(child, n) + 2 <= 96)
    if d.info()["builder"] == 2:
        d.save(tmp_path / "s.eos")
        expect = np.empty(n, np.int64)
        expect[order.astype(np.int64)] = position
        assert np.array_equal(_pos_of_id(tmp_path / "s.eos"), expect)
    d.close()
