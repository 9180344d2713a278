"""What is timed: the calls a user of this framework makes, over the sizes they make them at.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (points, a reusable tree, a server, the buffers that results go to),
``run`` makes the call and returns everything it computes: sorted edge lists, the
validator's verdict and counts, conflict regions.  All outputs are whole numbers
and independent of the order in which simplices were created, so two runs agree
exactly.  A list whose length depends on the points is returned as the caller's
whole buffer (-1 past the end) with its length.

Kinds
  one_call   ``vd_delaunay``: host points in, host edges out, a new tree each
             time (the reference's ``voronoids.delaunay``)
  rebuild    ``vd_delaunay_device`` on a tree that the program keeps: points and
             edge list in device memory
  batch      ``DelaunayTree.batch_device``: many independent sets at once
  serve      ``Server``: mixed 2D / 3D requests submitted together, results read
  insert     ``insert_point`` for every point of a set (the reference's
             sequential path), then the edge list
  append     ``add_points_to_tree`` with most of a set, then with ten further
             parts of it, then the edge list
  locate     ``locate``: conflict regions of many query points in a built tree
  validate   ``check_delaunay`` on a built tree
"""
import ctypes
import math

import numpy as np
import torch

import voronoids_gb300 as V
from voronoids_gb300 import _native
from voronoids_gb300 import workloads as W


def listed():
    return [
        # a small set triangulated on its own: latency, launches and allocations only
        {"name": "one_call_3d_200", "kind": "one_call", "dim": 3, "n": 200},
        # the smallest configured workload: 10,000 uniform 2D points
        {"name": "one_call_2d_10k", "kind": "one_call", "dim": 2, "n": 10_000},
        # a mid-sized one-shot call; the reference switches from its sequential path at 1e5 points
        {"name": "one_call_3d_100k", "kind": "one_call", "dim": 3, "n": 100_000},
        # the headline workload: 1M uniform 3D points, rebuilt with resident buffers
        {"name": "rebuild_3d_1m", "kind": "rebuild", "dim": 3, "n": 1_000_000, "points": "uniform"},
        # the same in the plane, an odd count
        {"name": "rebuild_2d_1m", "kind": "rebuild", "dim": 2, "n": 1_000_003, "points": "uniform"},
        # near-degenerate input: jittered lattice and tight clusters (filters and exact tier, huge regions)
        {"name": "rebuild_3d_degenerate", "kind": "rebuild", "dim": 3, "n": 262_144, "points": "near_degenerate"},
        # many sets of mixed size in one call
        {"name": "batch_3d_256", "kind": "batch", "dim": 3, "sets": 256, "lo": 32, "hi": 65_536},
        # a burst of service requests, both dimensions
        {"name": "serve_48", "kind": "serve", "requests": 48, "lo": 100, "hi": 200_000},
        # points arriving one at a time
        {"name": "insert_3d_500", "kind": "insert", "dim": 3, "n": 500},
        # points arriving in parts, on a tree that already holds most of them
        {"name": "append_3d_100k", "kind": "append", "dim": 3, "n": 100_003},
        # queries against a finished tree
        {"name": "locate_3d_4k", "kind": "locate", "dim": 3, "n": 100_000, "queries": 4096},
        # validation of a finished tree
        {"name": "validate_3d_300k", "kind": "validate", "dim": 3, "n": 300_000},
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one_call", "one_call", "rebuild", "rebuild", "batch", "serve", "insert", "append", "locate",
                       "validate"])
    dim = rng.choice([2, 3])
    if kind == "one_call":
        return {"kind": kind, "dim": dim, "n": _between(rng, 20, 100_000)}
    if kind == "rebuild":
        if rng.random() < 0.25:
            return {"kind": kind, "dim": 3, "n": 2 * _between(rng, 1000, 131_072), "points": "near_degenerate"}
        return {"kind": kind, "dim": dim, "n": _between(rng, 300, 1_000_000), "points": "uniform"}
    if kind == "batch":
        return {"kind": kind, "dim": dim, "sets": _between(rng, 2, 256), "lo": 32, "hi": 65_536}
    if kind == "serve":
        return {"kind": kind, "requests": _between(rng, 2, 48), "lo": 100, "hi": 200_000}
    if kind == "insert":
        return {"kind": kind, "dim": dim, "n": _between(rng, 50, 500)}
    if kind == "append":
        return {"kind": kind, "dim": dim, "n": _between(rng, 1000, 100_000)}
    if kind == "locate":
        return {"kind": kind, "dim": dim, "n": _between(rng, 1000, 100_000), "queries": _between(rng, 1, 4096)}
    return {"kind": kind, "dim": 3, "n": _between(rng, 1000, 300_000)}


def _sizes(count, lo, hi):
    """`count` sizes, log-uniform in [lo, hi) (one per equal share of the range, mixed up)."""
    u = (np.arange(count) + 0.5) / count
    s = np.floor(np.exp(np.log(lo) + u * (np.log(hi) - np.log(lo)))).astype(np.int64)
    return s[np.argsort(W.splitmix64(count, count), kind="stable")]


def _dims(count):
    return np.where(W.splitmix64(1000 + count, count) & np.uint64(1), 3, 2)


def _points(case, n, seed):
    if case.get("points") == "near_degenerate":
        return W.c3_points(n, seed=1_000_003 + seed)
    return W.uniform_points(n, case["dim"], 2_000_003 + seed)


def _edge_cap(dim, n):
    return (10 if dim == 3 else 4) * n + 64


def _host_edges(dim, n, dtype=np.int64):
    return np.full((_edge_cap(dim, n), 2), -1, dtype=dtype)


def _device_edges(dim, n):
    return torch.full((_edge_cap(dim, n), 2), -1, dtype=torch.int32, device="cuda")


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _i64(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))


def _ok(rc, what):
    if rc != _native.VD_OK:
        raise V.VDError(rc, what)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        sizes, dims = _sizes(case["requests"], case["lo"], case["hi"]), _dims(case["requests"])
        sets = [W.uniform_points(int(n), int(d), 3_000_017 + seed * 4099 + i) for i, (n, d) in enumerate(zip(sizes, dims))]
        return {"kind": kind, "sets": sets, "server": V.Server(pool_bytes=64 << 30, slots=3, max_batch_points=2_000_000),
                "uv": [_host_edges(p.shape[1], p.shape[0], np.int32) for p in sets]}
    dim = case["dim"]
    if kind == "batch":
        off = np.concatenate([[0], np.cumsum(_sizes(case["sets"], case["lo"], case["hi"]))]).astype(np.int64)
        n = int(off[-1])
        p = torch.from_numpy(W.uniform_points(n, dim, 4_000_037 + seed)).cuda()
        return {"kind": kind, "points": p, "offsets": off, "tree": V.DelaunayTree.create(dim), "uv": _device_edges(dim, n)}
    n = case["n"]
    p = _points(case, n, seed)
    if kind == "one_call":
        return {"kind": kind, "dim": dim, "points": p, "uv": _host_edges(dim, n)}
    if kind == "rebuild":
        return {"kind": kind, "points": torch.from_numpy(p).cuda(), "n": n, "tree": V.DelaunayTree.create(dim),
                "uv": _device_edges(dim, n)}
    if kind == "insert":
        return {"kind": kind, "points": p, "tree": V.DelaunayTree(p), "uv": _host_edges(dim, n)}
    if kind == "append":
        cut = [0, n - 10 * (n // 100)] + [n - k * (n // 100) for k in range(9, -1, -1)]
        return {"kind": kind, "points": p, "parts": [p[a:b] for a, b in zip(cut, cut[1:]) if b > a],
                "tree": V.DelaunayTree(p), "uv": _host_edges(dim, n)}
    tree = V.delaunay(p, seed=seed)
    if kind == "validate":
        return {"kind": kind, "tree": tree}
    # the simplices in an order of their own (by vertices), so that regions can be named
    # independently of the tree's numbering
    verts, _ = tree.simplices()
    rows = np.sort(verts, axis=1)
    name = np.empty(len(rows), dtype=np.int64)
    name[np.lexsort(rows.T[::-1])] = np.arange(len(rows))
    q = 0.05 + 0.9 * W.uniform_points(case["queries"], dim, 5_000_011 + seed)
    return {"kind": kind, "tree": tree, "queries": q, "name": name,
            "ids": torch.full((40 * len(q) + 1024,), -1, dtype=torch.int64, device="cuda")}


def run(state):
    kind, L = state["kind"], _native.load()
    m = ctypes.c_int64(0)
    if kind == "one_call":
        p, uv = state["points"], state["uv"]
        _ok(L.vd_delaunay(state["dim"], p.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), p.shape[0], 0, _i64(uv),
                          uv.shape[0], ctypes.byref(m)), "vd_delaunay")
        return [uv, m.value]
    if kind == "rebuild":
        uv = state["uv"]
        _ok(L.vd_delaunay_device(state["tree"]._h, ctypes.c_void_p(state["points"].data_ptr()), state["n"], 0,
                                 ctypes.c_void_p(uv.data_ptr()), uv.shape[0], ctypes.byref(m)), "vd_delaunay_device")
        return [uv, m.value]
    if kind == "batch":
        uv = state["uv"]
        eoff = state["tree"].batch_device(state["points"].data_ptr(), state["offsets"], 0, uv.data_ptr(), uv.shape[0])
        return [uv, eoff]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(p) for p in state["sets"]]
        done = 0
        while done < len(ids):
            done += len(server.poll(timeout_ms=1000))
        for i, uv in zip(ids, state["uv"]):
            st = ctypes.c_int(0)
            _ok(L.vd_server_result(server._h, i, _ptr(uv), uv.shape[0], ctypes.byref(m), ctypes.byref(st)),
                "vd_server_result")
            _ok(st.value, "request")
        return state["uv"]
    if kind in ("insert", "append"):
        tree, uv = state["tree"], state["uv"]
        tree.reset(state["points"])
        if kind == "insert":
            for p in state["points"]:
                tree.insert_point(p)
        else:
            for part in state["parts"]:
                tree.add_points_to_tree(part)
        _ok(L.vd_edges(tree._h, _i64(uv), uv.shape[0], ctypes.byref(m)), "vd_edges")
        return [uv, m.value]
    if kind == "validate":
        ok, counts = state["tree"].check_delaunay(details=True)
        return [int(ok), counts]
    regions, ids = state["tree"].locate(state["queries"]), state["ids"]
    size = np.array([len(r) for r in regions], dtype=np.int64)
    key = (np.repeat(np.arange(len(size), dtype=np.int64), size) << 32) | state["name"][np.concatenate(regions)]
    ids[: len(key)] = torch.from_numpy(key).cuda().sort().values
    return [size, ids]


def _set_work(dim, n):
    """Bytes (points in, edges out) and operations (one in-sphere determinant per facet of the result) of one set."""
    edges, facets, det = (7.7, 13.5, 80) if dim == 3 else (3.0, 3.0, 30)
    return np.array([8 * dim * n + 8 * edges * n, facets * det * n])


def work(case):
    kind = case["kind"]
    if kind == "serve":
        w = sum(_set_work(int(d), int(n)) for n, d in zip(_sizes(case["requests"], case["lo"], case["hi"]),
                                                         _dims(case["requests"])))
    elif kind == "batch":
        w = sum(_set_work(case["dim"], int(n)) for n in _sizes(case["sets"], case["lo"], case["hi"]))
    elif kind == "locate":
        # a region of about 20 (4) simplices and its outer shell are tested per query
        tests, det = (47, 80) if case["dim"] == 3 else (10, 30)
        simplices = 20 if case["dim"] == 3 else 4
        w = case["queries"] * np.array([8 * case["dim"] + 8 * simplices + 32 * tests, tests * det])
    elif kind == "validate":
        per, facets, det = (6.75, 13.5, 80) if case["dim"] == 3 else (2.0, 3.0, 30)
        w = case["n"] * np.array([32 * per + 8 * case["dim"], facets * det])
    else:
        w = _set_work(case["dim"], case["n"])
    return {"bytes": float(w[0]), "flops": float(w[1])}
