"""CPU: the stored-sphere tier of the conflict test (host build of
vd_predicates.cuh) never answers against the exact sign, whichever vertex is
its base, for simplices of every shape and scale and queries from far away to
within rounding of the circumsphere; and it does answer where it is meant to."""
import ctypes

import numpy as np
import pytest

dp = ctypes.POINTER(ctypes.c_double)
KINDS = ["uniform", "tiny", "far", "sliver", "flat", "super", "lattice", "mixed", "extreme"]


@pytest.fixture(scope="module")
def host():
    from voronoids_gb300 import build as B
    H = ctypes.CDLL(B.build_host())
    H.vdh_sphere_side.argtypes = [ctypes.c_int, dp, ctypes.c_int]
    return H


def _simplex(rng, dim, kind):
    p = rng.random((dim + 1, dim))
    if kind == "tiny":
        return 0.5 + (p - 0.5) * 10.0 ** -rng.uniform(1, 7)
    if kind == "far":
        return p + 10.0 ** rng.uniform(0, 8)
    if kind == "sliver":  # nearly on a common circle (line in 2D)
        p[-1] = p[0] + (p[1] - p[0]) * rng.random() + (rng.random(dim) - 0.5) * 10.0 ** -rng.uniform(1, 7)
        return p
    if kind == "flat":  # one short height
        p[:, -1] = 0.3 + (p[:, -1] - 0.5) * 10.0 ** -rng.uniform(1, 7)
        return p
    if kind == "super":  # one to dim vertices of a far super simplex
        k = rng.integers(1, dim + 1)
        p[:k] = 0.5 + (p[:k] - 0.5) * 20.0
        return p
    if kind == "lattice":
        return np.round(p * 4) / 4
    if kind == "mixed":
        return p * 10.0 ** rng.uniform(-3, 3, size=(dim + 1, 1))
    if kind == "extreme":  # beyond the range the tier serves, or at its limits
        return p * 2.0 ** rng.choice([-140, -61, -59, -26, -24, 19, 21, 59, 61, 140])
    return p


def _query(rng, s, dim, how):
    if how == 0:
        return rng.random(dim) * 1.2 - 0.1 + s.mean(axis=0) - 0.5
    d = s[1:] - s[0]
    try:
        c = s[0] + np.linalg.solve(2 * d, (d * d).sum(axis=1))
    except np.linalg.LinAlgError:
        return s.mean(axis=0)
    u = rng.normal(size=dim)
    u /= np.linalg.norm(u)
    r = np.linalg.norm(s[0] - c)
    return c + u * r * (1 + rng.choice([-1, 1]) * 10.0 ** -rng.uniform(0.5, 9))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dim", [2, 3])
def test_sphere_tier_is_sound(host, oracle, dim, kind):
    rng = np.random.default_rng(1000 * dim + KINDS.index(kind))
    sure, plain, total = 0, 0, 0
    for trial in range(1500):
        s = _simplex(rng, dim, kind)
        q = s[0].copy() if trial % 50 == 49 else _query(rng, s, dim, trial % 3)
        o = oracle.orient(s)
        if o == 0 or not np.isfinite(q).all():
            continue
        if o < 0:
            s[[0, 1]] = s[[1, 0]]
        P = np.zeros((dim + 2, 3))
        P[: dim + 1, :dim] = s
        P[dim + 1, :dim] = q
        want = oracle.insphere_exact(s, q)
        for rot in range(dim + 1):
            g = host.vdh_sphere_side(dim, P.ctypes.data_as(dp), rot)
            assert g == 0 or g == want, (s.tolist(), q.tolist(), rot, g, want)
            if trial % 3 == 0:
                plain += 1
                sure += g != 0
        total += 1
    assert total > 700
    if kind in ("uniform", "super"):  # the shapes it is meant for
        assert sure > plain // 2, (sure, plain)
