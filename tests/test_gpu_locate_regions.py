"""GPU: conflict regions of every size a query can have, against the oracle's exact test of every simplex.

Small regions are found by a warp with lists in shared memory (192 simplices in 3D, 64 in 2D), larger ones by a thread
with lists in global memory: the centre of points on a sphere or circle is in conflict with nearly every simplex.
Queries on vertices, outside the super simplex and in calls of one query are covered too."""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def regions(oracle, p, v, q, dim):
    sv, _ = oracle.super_vertices(p)
    xyz = np.vstack([sv[:, :dim], p])
    ids = np.where(v < 0, -v - 1, v + dim + 1)[:, : dim + 1]
    big = len(xyz) + 1  # the query is newer than every vertex
    return [np.array([i for i, s in enumerate(ids)
                      if oracle.insphere_sos(xyz[s], x, np.append(s, big).astype(np.int32)) > 0], dtype=np.int64) for x in q]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("kind", ["uniform", "lattice", "shell"])
def test_regions_match_the_oracle(vd, oracle, dim, kind):
    rng = np.random.default_rng(dim)
    if kind == "uniform":
        p = W.uniform_points(300, dim, 9)
    elif kind == "lattice":
        p = W.lattice_points(6 if dim == 3 else 16, dim) / 16
    else:
        u = rng.normal(size=(150, dim))
        p = u / np.linalg.norm(u, axis=1, keepdims=True)
    t = vd.delaunay(p, seed=1)
    v, _ = t.simplices()
    q = np.vstack([p.mean(axis=0) + (rng.random((12, dim)) - 0.5) * np.ptp(p, axis=0), p[:3], p.mean(axis=0)[None],
                   (p[:4] + p[4:8]) / 2])
    want = regions(oracle, p, v, q, dim)
    got = t.locate(q)
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.array_equal(t.locate(q[5]), want[5])
    if kind == "shell":
        assert max(len(b) for b in want) > (192 if dim == 3 else 64)
    far = p.mean(axis=0) + 1e4
    mixed = t.locate(np.vstack([far[None], q[:2], far[None]]))
    assert [len(a) for a in mixed] == [0, len(want[0]), len(want[1]), 0]
    t.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_more_ids_than_the_first_guess(vd, oracle, dim):
    rng = np.random.default_rng(7)
    u = rng.normal(size=(60 if dim == 2 else 90, dim))
    p = u / np.linalg.norm(u, axis=1, keepdims=True)
    t = vd.delaunay(p, seed=1)
    v, _ = t.simplices()
    q = (rng.random((40, dim)) - 0.5) * 0.2
    for a, b in zip(t.locate(q), regions(oracle, p, v, q, dim)):
        assert np.array_equal(a, b)
    t.close()
