"""GPU: device memory after trees are freed: at most 512 MB stay with the library, at once, and none after a trim.

On a stream of the tree's own and on a caller's, which nobody waits for."""
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("own", [True, False])
def test_freed_memory_returns(vd, own):
    import torch
    stream = None if own else torch.cuda.Stream()
    p = W.uniform_points(1_500_000, 3, 21)
    vd.delaunay(p[:100_000]).close()  # kernels loaded, their local memory set up
    vd.trim_memory()
    free = torch.cuda.mem_get_info()[0]
    t = vd.DelaunayTree.create(3, stream=None if own else stream.cuda_stream)
    t.reset(p)
    t.add_points_to_tree(p, seed=1)
    held = free - torch.cuda.mem_get_info()[0]
    assert held > 1536 * MB
    t.close()
    assert free - torch.cuda.mem_get_info()[0] <= (512 + 64) * MB
    vd.trim_memory()
    assert free - torch.cuda.mem_get_info()[0] <= 64 * MB
    t = vd.delaunay(p[:1000], seed=1)  # and the pool is still there
    assert t.check_delaunay()
    t.close()


def test_trim_with_a_live_tree(vd):
    p = W.uniform_points(50_000, 3, 22)
    t = vd.delaunay(p, seed=1)
    e = t.edges()
    vd.trim_memory()
    assert t.check_delaunay() and (t.edges() == e).all()
    t.close()
