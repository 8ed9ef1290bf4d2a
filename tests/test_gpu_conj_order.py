"""Order of a step's conjunctions (needs a B200): by TCA and then by record,
for batches on both sides of the one-CTA sort and steps on both sides of its
chunk size, with many equal TCAs."""

import numpy as np
import pytest

import oracle
from mizuba_b200.polyjectory import polyjectory

pytestmark = pytest.mark.gpu


def meetings_pj(n, n_times, order=3):
    """n objects on straight lines through the origin, in n_times groups that
    pass it at the same instant: pairs of one group have equal TCAs."""
    rng = np.random.default_rng(n)
    trajs = []
    for k in range(n):
        t0 = 0.25 + 0.5 * (k % n_times) / n_times
        v = rng.normal(0.0, 1.0, 3)
        v *= rng.uniform(0.5, 2.0) / np.linalg.norm(v)
        c = np.zeros((1, order + 1, 7))
        c[0, 0, :3], c[0, 1, :3] = -t0 * v, v
        c[0, 0, 2] += 1e-3 * (k + 1)
        c[0, 0, 3:6] = v
        c[0, 0, 6] = 2.0
        trajs.append(c)
    return polyjectory(trajs, [np.array([0.0, 1.0])] * n, [0] * n)


@pytest.mark.parametrize("n, n_times, interval", [
    (12, 1, 1.0), (32, 3, 1.0),    # one CTA
    (33, 1, 1.0), (63, 2, 0.5), (66, 1, 1.0), (70, 2, 0.5),  # past it, either side of a chunk
    (150, 1, 1.0), (150, 7, 0.21),  # several chunks in one step, and in several
])
def test_order(n, n_times, interval):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    pj = meetings_pj(n, n_times)
    thresh = 3.0
    r = oracle.run(pj, thresh, interval)["conjunctions"]
    g = mzb.device_conjunctions(pj, thresh, interval).conjunctions
    assert len(g) == len(r) >= n
    for f in ("i", "j", "tca", "dca", "ri", "vi", "rj", "vj"):
        assert np.array_equal(g[f], r[f]), f
