"""GPU: paths that only some calls take are taken here, against the oracle.

Rounds replayed from captured graphs (the third build on one tree with one seed is the first that replays
everything), points inserted under locks at the end of a call, and what such an insertion has to leave: regions
that do not fit a warp and new simplices when the slots run out.
"""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_replayed_rounds(vd, oracle, dim):
    a, b = W.uniform_points(20_000, dim, 31), W.uniform_points(20_000, dim, 32)
    large = W.uniform_points(90_000, dim, 33)  # makes the tree's arrays move
    want = {id(p): oracle.Triangulation(p, seed=1).edges() for p in (a, b, large)}
    t = vd.DelaunayTree(a)
    for i, p in enumerate((a, a, a, b, a, large, a, large, large, b, a, a)):
        t.reset(p)
        t.add_points_to_tree(p, seed=1)
        assert np.array_equal(t.edges(), want[id(p)]), i
        n = t.path_counts()["replayed_rounds"]
        assert n <= t.stats()["rounds"]
        if i in (2, 3, 4, 8, 10, 11):  # captured before on arrays that have not moved since
            assert n > 10, i
        if i in (0, 5):
            assert n == 0, i
    assert t.path_counts()["captured_rounds"] > 0
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [600, 4096, 30_000])
def test_finished_points(vd, oracle, dim, n):
    p = W.uniform_points(n, dim, 34)
    t = vd.delaunay(p, seed=1)
    assert 0 < t.path_counts()["finished_points"] <= n
    assert np.array_equal(t.edges(), oracle.Triangulation(p, seed=1).edges())
    done = t.path_counts()["finished_points"]
    t.add_points_to_tree(W.uniform_points(1000, dim, 35) * 0.5 + 0.25, seed=1)
    assert t.path_counts()["finished_points"] > done
    assert t.check_delaunay()
    t.reset(p)
    assert t.path_counts()["finished_points"] == 0
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_regions_that_do_not_fit_are_left(vd, oracle, dim):
    rng = np.random.default_rng(36)
    u = rng.normal(size=(800, dim))
    shell = u / np.linalg.norm(u, axis=1, keepdims=True)
    centre = 1e-3 * rng.normal(size=(40, dim))
    t = vd.DelaunayTree(np.concatenate([shell, centre]))
    t.add_points_to_tree(shell, seed=2)
    done = t.path_counts()["finished_points"]
    t.add_points_to_tree(centre, seed=2)
    assert t.path_counts()["finished_points"] - done < 39  # one goes in before, and some do not fit
    assert t.stats()["max_cavity"] > (64 if dim == 2 else 128)
    assert np.array_equal(t.edges(), oracle.Triangulation(np.concatenate([shell, centre]), seed=2).edges())
    t.close()


def test_slots_run_out(vd, oracle):
    """160 groups of 50 + 50 points on two skew lines: a group has a simplex for every pair of neighbours on one line
    and neighbours on the other, so a point adds far more slots than a call sets aside for it.  They run out while
    the last 4,000 points are inserted under locks (34,000 asked for in vain)."""
    rng = np.random.default_rng(37)
    parts = []
    for g in range(160):
        s, r = rng.uniform(-0.1, 0.1, (2, 50))
        o = 4.0 * np.array([g % 6, g // 6 % 6, g // 36])
        parts += [o + np.stack([s, 0 * s, 0 * s], 1), o + np.stack([0 * r, r, 0 * r + 1], 1)]
    p = np.concatenate(parts)
    t = vd.delaunay(p, seed=1)
    assert t.path_counts()["finished_points"] > 1000
    assert t.stats()["slots"] > 660_000
    assert t.check_delaunay()
    assert np.array_equal(t.edges(), oracle.Triangulation(p, seed=1).edges())
    t.close()
