"""GPU: every tier of the validator's signs (FP32 on split coordinates, FP64, exact) against the CPU validator.

A valid build's simplices are checked with other coordinates for its points, so that many simplices are inverted and
many facets not Delaunay; the violation counts must equal those of the oracle's big-integer validator.  The
coordinates are generic, on a coarse grid (exact ties and flat simplices) and scaled out of the FP32 tier's range."""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu

KEYS = ["non_positive", "asymmetric", "not_delaunay", "not_perturbed_delaunay", "hull_facets", "facets"]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("how", ["same", "noise", "grid", "huge", "tiny"])
def test_violations_match_the_cpu_validator(vd, oracle, dim, how):
    p = W.uniform_points(400, dim, 31 + dim)
    t = vd.delaunay(p, seed=1)
    v, nb = t.simplices()
    t.close()
    sv, _ = oracle.super_vertices(p)
    pts = np.vstack([sv[:, :dim], p])
    ids = np.where(v < 0, -v - 1, v + dim + 1).astype(np.int32)
    if dim == 2:
        ids[:, 3] = -1
    rng = np.random.default_rng(dim)
    moved = pts + (rng.random(pts.shape) - 0.5) * 0.1
    pts = {"same": pts, "noise": moved, "grid": np.round(moved * 16) / 16, "huge": moved * 2.0 ** 100,
           "tiny": moved * 2.0 ** -100}[how]
    ok, viol = vd.check_triangulation(pts, ids, nb)
    ref = oracle.validate(dim, pts, ids, nb)
    assert viol == {k: ref[k] for k in KEYS}
    assert ok == (how == "same")
