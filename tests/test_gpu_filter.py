"""The narrow phase's filter and both paths of the reference formulation
behind it (needs a B200): in the plain form every counter of the report and
every record must be the oracle's, whatever the filter settles by itself, for
orders on both sides of its shared-memory and register limits, sub-intervals
from whole segments down to slivers, and few (a warp per item) and many (a
thread per item) items left to the reference formulation."""

import numpy as np
import pytest

import oracle
from mizuba_b200 import synth
from parity import assert_trees_pairs_equal, conj_match

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mzb():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200

    return mizuba_b200


def same_records(g, r):
    assert len(g) == len(r)
    for f in ("i", "j", "tca", "dca", "ri", "vi", "rj", "vj"):
        assert np.array_equal(g[f], r[f]), f


@pytest.mark.parametrize("order", [2, 3, 4, 7, 12, 18, 19, 21, 22, 25, 31, 32])
@pytest.mark.parametrize("thresh, interval_min", [(8.0, 3.0), (60.0, 11.3), (1e-3, 0.9)])
def test_counters_and_records(mzb, order, thresh, interval_min):
    el = synth.base_elements(260, np.random.default_rng(100 + order), 0.1)
    el = np.concatenate([el, synth.shell_elements(60, np.random.default_rng(7))])
    pj = synth.build_polyjectory(el, 0.06, order=order)
    r = oracle.run(pj, thresh, interval_min / 1440.0)
    assert r["np_report"][0] > 0
    g = mzb.device_conjunctions(pj, thresh, interval_min / 1440.0)
    assert_trees_pairs_equal(g, r)
    assert g.np_report == r["np_report"]
    same_records(g.conjunctions, r["conjunctions"])
    m = mzb.device_conjunctions(pj, thresh, interval_min / 1440.0, form="mixed")
    conj_match(m.conjunctions, r["conjunctions"], thresh)


def test_many_items_left(mzb):
    pj = synth.build_polyjectory(synth.base_elements(300, np.random.default_rng(3), 0.0), 0.1, order=18)
    thresh, interval = 1500.0, 3.0 / 1440.0
    r = oracle.run(pj, thresh, interval)
    # Every item with a minimum below the threshold is left: the thread path.
    assert len(r["conjunctions"]) > 6144
    g = mzb.device_conjunctions(pj, thresh, interval)
    assert g.np_report == r["np_report"]
    same_records(g.conjunctions, r["conjunctions"])
