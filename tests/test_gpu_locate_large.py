"""GPU: conflict regions that outgrow a warp's lists, against the oracle's exact test of every simplex.

The lists hold 64 simplices in 2D and 192 in 3D, the wide form's 1,024; larger regions are found by a block with bits
and lists as long as the tree.  Points on a circle or sphere are in conflict with the centre all at once, so their
number sets the size of its region.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shell(n, dim, seed):
    u = np.random.default_rng(seed).normal(size=(n, dim))
    return u / np.linalg.norm(u, axis=1, keepdims=True)


def regions(oracle, t, p, q):
    dim = p.shape[1]
    v, _ = t.simplices()
    sv, _ = oracle.super_vertices(p)
    xyz = np.vstack([sv[:, :dim], p])
    ids = np.where(v < 0, -v - 1, v + dim + 1)[:, : dim + 1]
    big = len(xyz) + 1  # the query is newer than every vertex
    return [np.array([i for i, s in enumerate(ids)
                      if oracle.insphere_sos(xyz[s], x, np.append(s, big).astype(np.int32)) > 0], dtype=np.int64) for x in q]


@pytest.mark.parametrize("dim,n", [(2, n) for n in (*range(60, 70), *range(1020, 1030), 3000)] +
                         [(3, n) for n in (40, *range(66, 74, 2), 160, *range(354, 370, 3), 700)])
def test_sizes_about_the_limits(vd, oracle, dim, n):
    p = shell(n, dim, n)
    t = vd.delaunay(p, seed=1)
    q = np.vstack([np.zeros(dim), np.full(dim, 1e-3)])
    for a, b in zip(t.locate(q), regions(oracle, t, p, q)):
        assert np.array_equal(a, b)
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_large_ones_among_many(vd, oracle, dim):
    rng = np.random.default_rng(2)
    p = np.vstack([shell(2500 if dim == 2 else 500, dim, 3), 3 + rng.random((3000, dim)),
                   shell(120 if dim == 2 else 60, dim, 4) / 8 - 4])
    t = vd.delaunay(p, seed=1)
    q = np.vstack([np.full(dim, -4.0), 3 + rng.random((700, dim)), np.zeros(dim), 3 + rng.random((500, dim)),
                   np.full(dim, 0.01), np.full(dim, -4.001), np.full(dim, 1e4)])
    large = [0, 701, 1202, 1203]
    got = t.locate(q)
    for i, want in zip(large + [5, 900], regions(oracle, t, p, q[large + [5, 900]])):
        assert np.array_equal(got[i], want)
    assert len(got[701]) > 1024 and len(got[1204]) == 0
    for i in range(0, 1204, 50):
        assert np.array_equal(got[i], t.locate(q[i]))
    # counts alone, and a buffer that is one id short
    from voronoids_gb300 import _native
    L = _native.load()
    off = np.zeros(len(q) + 1, dtype=np.int64)
    i64p = ctypes.POINTER(ctypes.c_int64)
    args = (t._h, q.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), len(q), off.ctypes.data_as(i64p))
    assert L.vd_locate_points(*args, None, 0) == 6  # the last query is outside
    assert np.array_equal(np.diff(off), [len(r) for r in got])
    off[:] = -1
    ids = np.zeros(sum(len(r) for r in got) - 1, dtype=np.int64)
    assert L.vd_locate_points(*args, ids.ctypes.data_as(i64p), len(ids)) == 1
    assert np.array_equal(np.diff(off), [len(r) for r in got])
    t.close()


def test_one_huge_region_in_a_full_chunk(vd):
    """65,536 queries, one of them in conflict with 20,000 simplices: room and work are the sum of the regions,
    not the queries times the largest."""
    rng = np.random.default_rng(5)
    p = np.vstack([shell(20_000, 2, 6), 3 + rng.random((20_000, 2))])
    t = vd.delaunay(p, seed=1)
    q = 3 + rng.random((65_537, 2))
    q[40_000] = 0.0
    got = t.locate(q)
    assert len(got[40_000]) >= 19_998
    size = np.array([len(r) for r in got])
    for i in [*np.argsort(size)[-10:], 0, 65_535, 65_536]:
        assert np.array_equal(got[i], t.locate(q[i]))
    v, _ = t.simplices()
    inner = np.all((v[:, :3] >= 0) & (v[:, :3] < 20_000), axis=1)  # triangles of circle points alone
    assert np.all(np.isin(np.flatnonzero(inner), got[40_000]))
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_many_large_regions(vd, oracle, dim):
    """More large regions than blocks run at once."""
    p = shell(1500 if dim == 2 else 500, dim, 7)
    t = vd.delaunay(p, seed=1)
    rng = np.random.default_rng(8)
    q = (rng.random((700, dim)) - 0.5) * 0.02
    got = t.locate(q)
    pick = [0, 1, 350, 698, 699]
    for i, want in zip(pick, regions(oracle, t, p, q[pick])):
        assert np.array_equal(got[i], want)
    assert min(len(r) for r in got) > 1024
    t.close()
