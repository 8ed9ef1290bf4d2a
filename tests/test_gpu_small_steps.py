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


def clusters_pj(sizes, n, seed, order=2):
    """n objects spread over a box, the first ones in tight clusters of the
    given sizes: one cell of the sort's top bits each, told apart by the low
    bits only."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1000.0, 1000.0, (n, 3))
    at = 0
    for k, size in enumerate(sizes):
        cell = np.floor(rng.uniform(-400.0, 400.0, 3))
        pos[at:at + size] = cell * (2000.0 / 1024) + rng.uniform(0.2, 1.2, (size, 3))
        at += size
    order_ = rng.permutation(n)
    trajs = []
    for k in order_:
        c = np.zeros((1, order + 1, 7))
        c[0, 0, :3] = pos[k]
        c[0, 0, 6] = np.linalg.norm(pos[k])
        trajs.append(c)
    return polyjectory(trajs, [np.array([0.0, 1.0])] * n, [0] * n)


def longest_run(codes, bits=40):
    mask = int(np.bitwise_or.reduce(codes ^ codes[0]))
    ones = [b for b in range(64) if mask >> b & 1][-bits:]
    top = np.uint64(sum(1 << b for b in ones))
    key = np.sort(codes & top)
    _, cnt = np.unique(key, return_counts=True)
    return int(cnt.max())


@pytest.mark.parametrize("sizes, long", [((), False), ((20, 30), False), ((40, 60), False), ((150, 400), True),
                                         ((2000, 3), True)])
@pytest.mark.parametrize("n", [2049, 4096, 9001])
def test_runs_of_equal_top_bits(sizes, long, n):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    pj = clusters_pj(sizes, n, seed=n + len(sizes))
    kinds = np.full(n, 2, np.int32)
    kinds[0] = 1
    r = oracle.run(pj, 1e-3, 1.0, otypes=kinds)
    assert (longest_run(r["mcodes"][0]) > 64) == long
    for threads in (0, 256, 512):
        g = mzb.device_conjunctions(pj, 1e-3, 1.0, otypes=kinds, tuning={"sort_threads": threads})
        assert_dense_equal(g, r)
        assert_trees_pairs_equal(g, r)
