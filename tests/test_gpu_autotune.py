"""GPU: the autotuner ranks configurations by builds that replay captured rounds, as a tuned batch's repeated builds do."""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_the_timed_build_replays_its_rounds(vd, dim):
    torch = pytest.importorskip("torch")
    off = np.array([0, 40_000, 600_000, 600_700])  # so large that the last configurations differ in their grids
    d = torch.from_numpy(W.uniform_points(int(off[-1]), dim, 51)).cuda()
    t = vd.DelaunayTree.create(dim)
    t.autotune_batch(d.data_ptr(), off, sample_points=int(off[-1]))
    # the last build is one that was timed; few of its chunks may differ from the builds' before it
    assert t.path_counts()["replayed_rounds"] >= 0.8 * t.stats()["rounds"]
    t.close()
