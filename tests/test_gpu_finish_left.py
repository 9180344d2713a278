"""GPU: what k_finish leaves is taken by the next round, and equal points of different sets do not leave one another.

The round before k_finish has each simplex vote for the best of the points in it; votes for points that are in by
now must not keep a point that is left out of the next round.
"""
import warnings

import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_the_next_round_takes_what_is_left(vd, dim):
    base = W.uniform_points(20_000, dim, 41)
    g = np.linspace(0.15, 0.85, 5 if dim == 2 else 3)
    centres = np.stack(np.meshgrid(*[g] * dim, indexing="ij"), -1).reshape(-1, dim)
    t = vd.DelaunayTree(base)
    for seed in range(8):
        crowd = 1e-4 * W.uniform_points(13 * len(centres), dim, 100 + seed).reshape(-1, 13, dim) + centres[:, None]
        crowd[:, 12] = crowd[:, 0]  # two equal points in each: left, or one of them
        crowd = crowd.reshape(-1, dim)
        t.reset(base)
        t.add_points_to_tree(base, seed=seed)
        before = t.stats()["rounds"]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", RuntimeWarning)
            t.add_points_to_tree(crowd, seed=seed)
        # crowds are far from one another: a round that brings the points in, one that inserts every better
        # twin and one that drops the others
        assert t.stats()["rounds"] - before == 3
        assert t.path_counts()["finished_points"] > 0 and len(t.duplicates()) == len(centres)
        assert t.check_delaunay()
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_equal_points_of_different_sets(vd, oracle, dim):
    rng = np.random.default_rng(42)
    p = rng.random((40, dim))
    q = np.concatenate([p, p[:9]])[rng.permutation(49)]  # and equal points within a set
    sets = [p, q, p, q, p, p[::-1].copy(), q, p]
    t = vd.DelaunayTree.create(dim)
    off = np.cumsum([0] + [len(s) for s in sets])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        uv, eoff = t.batch(np.concatenate(sets), off, seed=3)
    assert t.path_counts()["finished_points"] >= 100  # of 200 in the sets without equal points
    for k, s in enumerate(sets):
        if len(s) == 40:
            assert np.array_equal(uv[eoff[k]:eoff[k + 1]].astype(np.int64), oracle.Triangulation(s, seed=3).edges())
    assert len(t.duplicates()) == 3 * 9
    assert t.check_delaunay()
    t.close()
