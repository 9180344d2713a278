"""GPU: a tree without a super simplex (vd_tree_create) is empty, whatever trees were freed before it.

Its device memory is what earlier trees gave back, their counters included, so each query is made right after a
larger tree is gone.
"""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_created_tree_is_empty(vd, dim):
    p = W.uniform_points(40_000, dim, 11)
    p[-5:] = p[:5]  # duplicates are counted too
    for ask in ("stats", "num_edges", "edges", "simplices", "check", "duplicates", "ids"):
        with pytest.warns(RuntimeWarning):
            t = vd.delaunay(p, seed=1)
        t.edges()
        t.locate(p[:9])
        t.close()
        t = vd.DelaunayTree.create(dim)
        if ask == "stats":
            st = t.stats()
            assert st.pop("live_simplices") == 1  # the root that a reset writes
            assert not any(st.values()), st
        elif ask == "num_edges":
            assert t.num_edges() == 0
        elif ask == "edges":
            assert t.edges().shape == (0, 2)
        elif ask == "simplices":
            assert len(t.simplices()[0]) == 0
        elif ask == "check":
            ok, counts = t.check_delaunay(details=True)
            assert not ok and not any(counts.values())  # no super simplex to validate
        elif ask == "duplicates":
            assert len(t.duplicates()) == 0
        else:
            assert t.max_simplex_id == dim + 1
        uv = t.batch(p[:100], np.array([0, 60, 100]), seed=1)[0]
        assert len(uv) > 100
        t.close()
