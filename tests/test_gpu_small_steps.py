"""Step sort in shared memory and the smaller BVH CTAs (needs a B200): object
counts around the powers of two of the sorting network, its limit and the CTA
sizes' limits, with equal codes, no-data objects and boxes with the largest
code."""

import numpy as np
import pytest

import oracle
from mizuba_b200.polyjectory import polyjectory
from parity import assert_dense_equal, assert_trees_pairs_equal

pytestmark = pytest.mark.gpu


def grid_pj(n, seed, order=2):
    """Points on a coarse grid (equal codes), a corner object (largest code),
    and every seventh object without data."""
    rng = np.random.default_rng(seed)
    trajs, times = [], []
    for k in range(n):
        if k % 7 == 3:
            trajs.append(np.zeros((0, order + 1, 7)))
            times.append(np.zeros(0))
            continue
        c = np.zeros((1, order + 1, 7))
        c[0, 0, :3] = rng.integers(0, 12, 3) * 100.0 if k % 11 else 1100.0
        c[0, 0, 6] = c[0, 0, 0]
        trajs.append(c)
        times.append(np.array([0.0, 1.0]))
    return polyjectory(trajs, times, [0] * n)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 64, 65, 511, 512, 513, 1023, 1025, 2047, 2048, 2049, 4097])
@pytest.mark.parametrize("steps", [1, 150])
def test_small_steps(n, steps):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    pj = grid_pj(n, n)
    kinds = np.full(n, 2, np.int32)  # secondaries only: no pairs to narrow
    kinds[0] = 1
    r = oracle.run(pj, 1e-3, 1.0 / steps, otypes=kinds)
    g = mzb.device_conjunctions(pj, 1e-3, 1.0 / steps, otypes=kinds)
    assert_dense_equal(g, r)
    assert_trees_pairs_equal(g, r)
