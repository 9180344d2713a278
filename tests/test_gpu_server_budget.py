"""GPU: the server's budget counts what its batches really take, small ones too, and refuses nothing it took before."""
import time

import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


def run(srv, sets):
    ids = [srv.submit(p) for p in sets]
    left, end = set(ids), time.time() + 60
    while left and time.time() < end:
        left -= set(srv.poll(timeout_ms=100))
    assert not left
    return [srv.result(i) for i in ids]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [100, 5000, 300_000])
def test_reserved_bytes_cover_a_batch(vd, dim, n):
    import torch
    p = W.uniform_points(n, dim, 61)
    srv = vd.Server(pool_bytes=8 << 30, slots=1)
    run(srv, [p])  # kernels loaded
    srv.close()
    vd.trim_memory()
    free = torch.cuda.mem_get_info()[0]
    srv = vd.Server(pool_bytes=8 << 30, slots=1)
    run(srv, [p])
    vd.trim_memory()  # arrays that the tree has outgrown
    held = free - torch.cuda.mem_get_info()[0]
    peak = srv.stats()["peak_bytes_in_flight"]
    srv.close()
    # device memory comes to the pool in blocks of 32 MB, for small arrays and for large ones
    assert held <= peak + 64 * MB
    assert peak <= 2 * held


@pytest.mark.parametrize("dim,per", [(2, 700), (3, 1850)])
def test_what_fits_the_budget_is_taken(vd, dim, per):
    p = [W.uniform_points(n, dim, 62) for n in (4000, 3000, 4000)]
    srv = vd.Server(pool_bytes=per * 4000 + 4096, slots=3)  # exactly the largest request
    for e, q in zip(run(srv, p), p):
        t = vd.delaunay(q)
        assert np.array_equal(e, t.edges())
        t.close()
    st = srv.stats()
    assert 0 < st["peak_bytes_in_flight"] <= st["budget"] and st["bytes_in_flight"] == 0
    i = srv.submit(W.uniform_points(4001, dim, 63))
    while i not in srv.poll(timeout_ms=100):
        pass
    with pytest.raises(vd.VDError) as e:
        srv.result(i)
    assert e.value.status == 3
    srv.close()
