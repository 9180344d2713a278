"""GPU: where a one-point insertion starts, against the oracle.

The walk of ``insert_point`` ends at the first simplex whose stored sphere
certainly holds the point, or at the one that contains it; only then is the
point compared with vertices.  A lattice (every sphere through 8 points: no
certain answer), its points repeated at once and much later, points a last
place away from a vertex, and the same far from the origin, where the high
halves of the coordinates agree.
"""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mixed_points(dim, shift):
    g = np.stack(np.meshgrid(*[np.arange(4.0)] * dim, indexing="ij"), -1).reshape(-1, dim) + shift
    rng = np.random.default_rng(dim)
    g = g[rng.permutation(len(g))]
    near = np.where(g[:6] == 0.0, 2.0**-60, np.nextafter(g[:6], np.inf))
    inner = shift + 3.0 * rng.random((40, dim))
    p = np.concatenate([g[:10], g[3:4], g[10:], near, g[:5], inner, near[2:4], inner[7:9]])
    return p


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shift", [0.0, 1000.0])
def test_one_by_one_matches_oracle(vd, oracle, dim, shift):
    p = mixed_points(dim, shift)
    t = vd.DelaunayTree(p)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        for q in p:
            t.insert_point(q)
    # one by one keeps the first of equal points, the oracle the first in its own
    # order: it gets the first ones only, and its indices are mapped back
    first = np.sort(np.unique(p, axis=0, return_index=True)[1])
    want = first[oracle.Triangulation(p[first]).edges().astype(np.int64)]
    assert len(t.duplicates()) == len(p) - len(first) == 10
    assert np.array_equal(t.edges(), want)
    assert t.check_delaunay()
    far = p[0].copy()
    far[dim - 1] += 1e5
    with pytest.raises(vd.VDError) as ei:
        t.insert_point(far)
    assert ei.value.status == 6
    assert np.array_equal(t.edges(), want)
