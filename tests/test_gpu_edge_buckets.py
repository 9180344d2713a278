"""GPU: edge lists with buckets longer than a warp sorts, on memory in use before.

Point 0 is the centre of a circle (sphere), so its bucket of the edge
extraction holds an edge to every other point: sizes on both sides of the 256
entries one warp sorts, and one that is sorted by a block in several steps.  A
larger tree built and closed before leaves its own counts in the memory that
the next tree's buffers are taken from.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def around_centre(dim, k):
    rng = np.random.default_rng(100 * dim + k)
    d = rng.standard_normal((k, dim))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([np.zeros((1, dim)), d])


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("k", [255, 256, 257, 300, 1500])
def test_hub_edges_match_oracle(vd, oracle, dim, k):
    t = vd.delaunay(np.random.default_rng(7).random((20_000, dim)), seed=1)
    t.edges()
    t.close()
    p = around_centre(dim, k)
    t = vd.delaunay(p, seed=5)
    e = t.edges()
    t.close()
    assert np.count_nonzero(e[:, 0] == 0) == k
    assert np.array_equal(e, oracle.Triangulation(p, seed=5).edges())
