"""GPU: the last points of a call, inserted under locks, against the oracle.

Calls of every small size (all of their points may be left at the end), a call
onto a larger tree, points crowded into a tiny cube (every pair of insertions
conflicts), a lattice (every test a tie), equal points among the last ones
(the best priority survives, as in the rounds) and several sets at once.
"""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(vd, parts, seed):
    t = vd.DelaunayTree(np.concatenate(parts))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        for p in parts:
            t.add_points_to_tree(p, seed=seed)
    return t


def check(vd, oracle, parts, seed):
    t = build(vd, parts, seed)
    p = np.concatenate(parts)
    assert np.array_equal(t.edges(), oracle.Triangulation(p, seed=seed).edges())
    assert t.check_delaunay()
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [2, 33, 600, 4096, 4097, 30_000])
def test_sizes(vd, oracle, dim, n):
    check(vd, oracle, [np.random.default_rng(n).random((n, dim))], 3)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 31, 500, 3000])
def test_onto_a_tree(vd, oracle, dim, n):
    rng = np.random.default_rng(n)
    check(vd, oracle, [rng.random((8000, dim)), rng.random((n, dim)), rng.random((n, dim))], 2)


@pytest.mark.parametrize("dim", [2, 3])
def test_crowded(vd, oracle, dim):
    rng = np.random.default_rng(4)
    crowd = 0.5 + 1e-7 * rng.random((400, dim))
    check(vd, oracle, [rng.random((5000, dim)), crowd], 1)


@pytest.mark.parametrize("dim", [2, 3])
def test_lattice(vd, oracle, dim):
    g = np.stack(np.meshgrid(*[np.arange(12.0)] * dim, indexing="ij"), -1).reshape(-1, dim)
    rng = np.random.default_rng(5)
    check(vd, oracle, [g[rng.permutation(len(g))]], 1)


@pytest.mark.parametrize("dim", [2, 3])
def test_equal_points(vd, oracle, dim):
    rng = np.random.default_rng(6)
    p = rng.random((2000, dim))
    p = np.concatenate([p, p[:300], p[:200], p[100:150]])[rng.permutation(2550)]
    t = build(vd, [p], 4)
    o = oracle.Triangulation(p, seed=4)
    assert len(t.duplicates()) == o.num_duplicates() == 550
    assert np.array_equal(t.edges(), o.edges())
    t.close()


def test_many_sets(vd, oracle):
    rng = np.random.default_rng(8)
    sets = [rng.random((n, 3)) for n in (5, 40, 300, 900, 17)]
    for e, p in zip(vd.delaunay_batch(sets, seed=2), sets):
        assert np.array_equal(e, oracle.Triangulation(p, seed=2).edges())
