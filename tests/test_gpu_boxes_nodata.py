"""Box pass of catalogues in which many objects have no data (needs a B200):
no boxes, and no time, for those."""

import numpy as np
import pytest

import oracle
from mizuba_b200 import synth
from mizuba_b200.polyjectory import polyjectory
from parity import assert_dense_equal

pytestmark = pytest.mark.gpu


def without(pj, empty):
    trajs, times = [], []
    for i in range(pj.n_objs):
        tr, tm, _ = pj[i]
        trajs.append(np.zeros_like(np.array(tr)[:0]) if i in empty else np.array(tr))
        times.append(np.zeros(0) if i in empty else np.array(tm))
    return polyjectory(trajs, times, [0] * pj.n_objs)


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_no_data_objects_cost_nothing(form):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    n, interval = 5000, 3.0 / 1440.0
    whole = synth.build_polyjectory(synth.base_elements(n, np.random.default_rng(n)), 0.4)
    few = without(whole, set(np.random.default_rng(1).choice(n, n // 5, replace=False).tolist()))
    ms = []
    for pj in (whole, few):
        t = []
        for _ in range(9):
            g = mzb.device_conjunctions(pj, 5.0, interval, form=form)
            t.append(g.stage_ms["aabb"])
        ms.append(float(np.median(t)))
        if form == "plain":
            s = (0, 40, 191)
            for k in s:
                assert_dense_equal(g, oracle.run(pj, 5.0, interval, step_begin=k, step_end=k + 1), k)
    assert ms[1] < 1.25 * ms[0], ms
