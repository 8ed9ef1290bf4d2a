"""Partner lists of every length class (needs a B200): objects crossing one
point, so that all their boxes overlap and object k has n - 1 - k partners.
The sizes sit at the edges of the list sorts (8 partners in registers, 1,024
in shared memory, beyond them in place) and, at the largest, past the pair
queue a call starts with, so that it grows and the walk runs again."""

import numpy as np
import pytest

import oracle
from mizuba_b200.polyjectory import polyjectory
from parity import assert_dense_equal, assert_trees_pairs_equal

pytestmark = pytest.mark.gpu


def crossing_pj(n, seed, order=3):
    rng = np.random.default_rng(seed)
    trajs = []
    for _ in range(n):
        c = np.zeros((1, order + 1, 7))
        v = rng.normal(0.0, 10.0, 3)
        v = np.sign(v) * np.maximum(np.abs(v), 1.0)
        c[0, 0, :3] = rng.uniform(-0.1, 0.1, 3) - 0.5 * v
        c[0, 1, :3] = v
        c[0, 0, 3:6] = v
        c[0, 0, 6], c[0, 1, 6] = -0.5, 1.0
        trajs.append(c)
    return polyjectory(trajs, [np.array([0.0, 1.0])] * n, [0] * n)


@pytest.mark.parametrize("walk", [0, 1, 2])
@pytest.mark.parametrize("n", [9, 10, 33, 1026])
def test_partner_list_lengths(n, walk):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    mzb.release_scratch()  # the queue starts at its first size
    pj = crossing_pj(n, seed=n)
    thresh, interval = 1e-3, 1.0
    r = oracle.run(pj, thresh, interval)
    assert len(r["bp"][0]) == n * (n - 1) // 2
    g = mzb.device_conjunctions(pj, thresh, interval, tuning={"broad_walk": walk})
    assert_dense_equal(g, r)
    assert_trees_pairs_equal(g, r)
    # Types: the pairs of two secondaries and those with a masked object go.
    types = np.random.default_rng(5).choice(np.array([1, 2, 4], np.int32), n)
    types[0] = 1
    r = oracle.run(pj, thresh, interval, otypes=types)
    g = mzb.device_conjunctions(pj, thresh, interval, otypes=types, tuning={"broad_walk": walk})
    assert_trees_pairs_equal(g, r)
