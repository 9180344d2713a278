"""GPU: the autotuner ranks configurations by builds that replay captured rounds, as a tuned batch's repeated builds do."""
import numpy as np
import pytest

from voronoids_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_timed_builds_replay_their_rounds(vd, dim):
    torch = pytest.importorskip("torch")
    off = np.array([0, 3000, 20_000, 20_700])
    d = torch.from_numpy(W.uniform_points(int(off[-1]), dim, 51)).cuda()
    t = vd.DelaunayTree.create(dim)
    t.autotune_batch(d.data_ptr(), off, sample_points=int(off[-1]))
    n = t.path_counts()
    # every configuration's rounds are captured once and replayed in the build that is timed
    assert n["captured_rounds"] > 100 and n["replayed_rounds"] >= 0.9 * n["captured_rounds"]
    t.close()
