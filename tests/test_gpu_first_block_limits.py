"""GPU: the block that inserts the first points of a fresh call, at the limits of its shared memory.

Inputs on both sides of the vertex capacity (644 points in 3D, 1,665 in 2D) and inputs whose star outgrows its
facet list (512: the centre of points on a sphere or circle), where the block gives up and the rounds insert
everything.  The edge list must equal the oracle's either way."""
import warnings

import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def check(vd, oracle, p, seed):
    t = vd.DelaunayTree(p)
    t.set_first_block(1 << 20)
    # one level for every point (priority levels start at this size), so that
    # the block takes all of them or none
    t.set_schedule(first_prefix=len(p), growth=2.0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        t.add_points_to_tree(p, seed=seed)
    o = oracle.Triangulation(p, seed=seed)
    assert np.array_equal(t.edges(), o.edges())
    assert t.check_delaunay()
    st = t.stats()
    assert st["inserted"] + st["duplicates"] == len(p)
    assert st["live_simplices"] == len(t.simplices()[0])
    rounds = st["rounds"]
    t.close()
    return rounds


@pytest.mark.parametrize("dim,n", [(3, 1), (3, 643), (3, 644), (3, 645), (2, 1664), (2, 1665), (2, 1666)])
def test_vertex_capacity(vd, oracle, dim, n):
    p = W.uniform_points(n, dim, 70 + n)
    if n == 1:  # a single point has no extent to size a super simplex from
        p = np.vstack([p, p + 0.5])
    check(vd, oracle, p, 3)


@pytest.mark.parametrize("dim", [2, 3])
def test_star_above_the_facet_list(vd, oracle, dim):
    rng = np.random.default_rng(dim)
    u = rng.normal(size=(600, dim))
    p = np.vstack([u / np.linalg.norm(u, axis=1, keepdims=True), np.zeros((1, dim))])
    for seed in (1, 2):
        check(vd, oracle, p, seed)


@pytest.mark.parametrize("dim", [2, 3])
def test_more_copies_than_points(vd, oracle, dim):
    p = W.uniform_points(60, dim, 5)
    check(vd, oracle, np.vstack([p] * 8), 4)
