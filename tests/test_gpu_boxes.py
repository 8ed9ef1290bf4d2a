"""Boxes whose floats the FMA enclosure cannot decide (needs a B200): bounds
placed on and next to the midpoints between floats, where the plain form must
take the reference formulation, and steps that hold many segments of an
object, the last of them undecided."""

import numpy as np
import pytest

import oracle
from mizuba_b200.polyjectory import polyjectory
from parity import assert_dense_equal

pytestmark = pytest.mark.gpu


def pj_on_midpoints(order, seed):
    """Constant and slowly moving objects whose bound minus the radius lies
    on, or within a few ulps of, the midpoint of two floats."""
    rng = np.random.default_rng(seed)
    radius = 0.5
    trajs, times = [], []
    for k in range(200):
        x = np.float32(rng.uniform(100.0, 9000.0))
        mid = (float(x) + float(np.nextafter(x, np.float32(np.inf)))) / 2
        ns = int(rng.integers(1, 6))
        c = np.zeros((ns, order + 1, 7))
        for v in (0, 1, 2, 6):
            c[:, 0, v] = mid + radius
            for _ in range(int(rng.integers(0, 3))):
                c[:, 0, v] = np.nextafter(c[:, 0, v], np.inf)
        if k % 3 == 0:  # a rising tail: the enclosure's lower bound stays c_0
            c[:, 1, :3] = rng.uniform(0.0, 1e-9, 3)
            c[:, order, 0] = 1e-13
        if k % 5 == 0:  # a segment far away, so that another decides the fold
            c[0, 0, :3] += 50.0
        trajs.append(c)
        times.append(np.linspace(0.0, 1.0, ns + 1))
    return polyjectory(trajs, times, [0] * len(trajs))


@pytest.mark.parametrize("order", [2, 18, 19, 20, 25, 32])
@pytest.mark.parametrize("interval", [1.0, 0.23])
def test_undecided_bounds(order, interval):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    pj = pj_on_midpoints(order, order)
    r = oracle.run(pj, 1.0, interval, otypes=np.full(pj.n_objs, 2, np.int32))
    g = mzb.device_conjunctions(pj, 1.0, interval, otypes=np.full(pj.n_objs, 2, np.int32))
    assert_dense_equal(g, r)
    # The mixed form's boxes contain them.
    m = mzb.device_conjunctions(pj, 1.0, interval, otypes=np.full(pj.n_objs, 2, np.int32), form="mixed")
    assert np.all(m.aabbs[:, :, 0] <= g.aabbs[:, :, 0]) and np.all(m.aabbs[:, :, 1] >= g.aabbs[:, :, 1])
