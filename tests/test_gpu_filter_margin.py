"""The narrow phase's filter where its error margin decides (needs a B200):
pairs whose coefficients do not fall off, so that the interpolation's rounding
is as large as it gets, with the threshold a few units in the last place above
the reference formulation's smallest Bernstein coefficient (it keeps the item),
and encounters with the threshold next to the minimum.  Every counter and
record must be the oracle's."""

import math

import numpy as np
import pytest

import oracle
from mizuba_b200.polyjectory import polyjectory

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mzb():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200

    return mizuba_b200


def smallest_coefficient(ci, cj):
    """The reference formulation on [0, 1] (conjunctions_jit.cpp:68-264,
    narrow_phase.cpp:95-152) for pairs of one-segment objects, coefficients
    (order + 1, 3, pairs): min of the squared distance's Bernstein coefficients."""
    op1 = len(ci)
    n = op1 - 1
    x = [(math.cos((2 * (n - m) + 1) / (2 * op1) * math.pi) + 1) / 2 for m in range(op1)]
    f = []
    for m in range(op1):
        a, b = ci[n], cj[n]
        for k in range(n - 1, -1, -1):
            a, b = ci[k] + a * x[m], cj[k] + b * x[m]
        d = a - b
        f.append((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
    for k in range(n):
        for j in range(n, k, -1):
            f[j] = (f[j] - f[j - 1]) / (x[j] - x[j - k - 1])
    for k in range(n - 1, -1, -1):
        for j in range(k, n):
            f[j] = f[j] - x[k] * f[j + 1]
    t = [f[k] / math.comb(n, k) for k in range(op1)]
    out = t[0]
    for k in range(1, op1):
        t = [t[j] + t[j + 1] for j in range(len(t) - 1)]
        out = np.minimum(out, t[0])
    return out


def pair_pj(ci, cj):
    """Two objects with one segment over [0, 1] each."""
    tr = []
    for c in (ci, cj):
        s = np.zeros((1, len(c), 7))
        s[0, :, :3] = c
        tr.append(s)
    return polyjectory(tr, [np.array([0.0, 1.0])] * 2, [0, 0])


def same(mzb, pj, thresh, forms=("plain",)):
    r = oracle.run(pj, thresh, 1.0, n_threads=1)
    for form in forms:
        g = mzb.device_conjunctions(pj, thresh, 1.0, form=form)
        a, b = g.conjunctions, r["conjunctions"]
        if form == "plain":
            assert g.np_report == r["np_report"]
        assert len(a) == len(b)
        for f in ("i", "j", "tca", "dca", "ri", "vi", "rj", "vj"):
            assert np.array_equal(a[f], b[f]), f
    return r


@pytest.mark.parametrize("growth", [0.8, 1.0, 1.2])
@pytest.mark.parametrize("order", [2, 3, 8, 15, 18, 20, 22, 25, 28, 31, 32])
def test_flat_coefficients(mzb, order, growth):
    rng = np.random.default_rng(order)
    n = 240
    shape = (2, order + 1, 3, n)
    c = rng.uniform(0.3, 1.0, shape) * rng.choice([-1.0, 1.0], shape) * np.exp(rng.uniform(0.0, 6.0, n))
    c *= growth ** np.arange(order + 1)[:, None, None]
    c[0, 0, 0] += np.abs(c[0, :, 0]).sum(axis=0) * rng.uniform(0.0, 2.5, n)
    low = smallest_coefficient(c[0], c[1])
    kept = 0
    for k in np.nonzero(low > 0)[0]:
        r = same(mzb, pair_pj(c[0, :, :, k], c[1, :, :, k]), math.sqrt(low[k]) * (1 + 1e-15))
        kept += r["np_report"][1] == 0
    assert kept > 20  # the threshold lies where the reference keeps the item


@pytest.mark.parametrize("order", [2, 5, 12, 18, 25, 32])
def test_threshold_at_the_minimum(mzb, order):
    rng = np.random.default_rng(50 + order)
    for k in range(24):
        ci, cj = rng.normal(0.0, 1.0, (2, order + 1, 3)) * (0.5 ** np.arange(order + 1))[:, None]
        cj[1] += rng.normal(0.0, 30.0, 3)
        s = rng.uniform(0.2, 0.8)
        at = s ** np.arange(order + 1)
        cj[0] += at @ ci - at @ cj + rng.normal(0.0, 1.0, 3) * 10.0 ** rng.uniform(-3.0, 0.5)
        dca = oracle.run(pair_pj(ci, cj), 1e3, 1.0, n_threads=1)["conjunctions"]["dca"]
        for d in dca:
            for e in (0.0, 1e-15, -1e-15, 1e-12, -1e-12, 1e-8, -1e-8, -1e-3):
                same(mzb, pair_pj(ci, cj), d * (1 + e), ("plain", "mixed"))


def test_more_left_than_the_queue_expects(mzb):
    """A first call whose filter leaves nearly every item: its queue is grown
    and the narrow phase run again."""
    from mizuba_b200 import synth

    pj = synth.build_polyjectory(synth.base_elements(400, np.random.default_rng(9), 0.0), 0.1, order=18)
    thresh, interval = 3000.0, 3.0 / 1440.0
    r = oracle.run(pj, thresh, interval)
    mzb.release_scratch()
    for _ in range(2):
        for form in ("plain", "mixed"):
            g = mzb.device_conjunctions(pj, thresh, interval, form=form)
            a, b = g.conjunctions, r["conjunctions"]
            assert g.np_report[0] >= r["np_report"][0] and len(a) == len(b) > 10000
            for f in ("i", "j", "tca", "dca", "ri", "vi", "rj", "vj"):
                assert np.array_equal(a[f], b[f]), f
            if form == "plain":
                assert g.np_report == r["np_report"]


@pytest.mark.parametrize("thresh", [900.0, 1100.0, 1300.0, 1600.0])
def test_root_items_around_two_a_warp(mzb, thresh):
    from mizuba_b200 import synth

    pj = synth.build_polyjectory(synth.base_elements(150, np.random.default_rng(9), 0.0), 0.1, order=18)
    r = oracle.run(pj, thresh, 3.0 / 1440.0)
    assert 1200 < len(r["conjunctions"]) < 3000  # root items: these and some more
    g = mzb.device_conjunctions(pj, thresh, 3.0 / 1440.0)
    assert g.np_report == r["np_report"]
    a, b = g.conjunctions, r["conjunctions"]
    assert len(a) == len(b)
    for f in ("i", "j", "tca", "dca", "ri", "vi", "rj", "vj"):
        assert np.array_equal(a[f], b[f]), f
