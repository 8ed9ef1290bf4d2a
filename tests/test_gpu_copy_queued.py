"""Copies of a result to device memory that are still queued on the default
stream when the result is freed (needs a B200): the next call takes the freed
block, and must not write to it before they have read it."""

import ctypes as ct

import numpy as np
import pytest

from mizuba_b200 import synth

pytestmark = pytest.mark.gpu


def test_copies_queued_behind_other_work():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb
    from mizuba_b200 import _native

    L = _native.core()
    n, thresh, interval = 2000, 5.0, 3.0 / 1440.0
    pjs = [mzb.to_device(synth.build_polyjectory(synth.base_elements(n, np.random.default_rng(k)), 0.1))
           for k in (1, 2)]

    def call(pj):
        res = ct.c_void_p()
        opts = _native.MzbOpts()
        assert L.mzb_conjunctions(pj._h, thresh, interval, None, ct.byref(opts), ct.byref(res)) == 0
        return res

    want = {}
    for k in (0, 1, 0):  # both sizes known, the block of the last one spare
        res = call(pjs[k])
        s = int(L.mzb_result_n_steps_run(res))
        nodes = int(L.mzb_result_n_tree_nodes(res))
        if k == 0:
            shapes = {"aabbs": (s, n + 1, 8), "srt_aabbs": (s, n + 1, 8), "mcodes": (s, n, 2), "srt_mcodes": (s, n, 2),
                      "srt_idx": (s, n), "trees": (nodes, 12)}
            for name, shape in shapes.items():
                a = np.zeros(shape, np.int32)
                assert getattr(L, "mzb_result_copy_" + name)(res, a.ctypes.data) == 0
                want[name] = a
        L.mzb_result_free(res)
    for _ in range(3):
        out = {name: torch.zeros(a.shape, dtype=torch.int32, device="cuda") for name, a in want.items()}
        res = call(pjs[0])
        torch.cuda.synchronize()
        assert L.mzb_result_copy_trees(res, out["trees"].data_ptr()) == 0
        torch.cuda._sleep(int(2e8))  # 0.1 s of other work ahead of the copies
        for name, a in out.items():
            if name != "trees":
                assert getattr(L, "mzb_result_copy_" + name)(res, a.data_ptr()) == 0
        L.mzb_result_free(res)
        res = call(pjs[1])
        L.mzb_result_free(res)
        torch.cuda.synchronize()
        for name, a in out.items():
            assert np.array_equal(a.cpu().numpy(), want[name]), name


@pytest.mark.parametrize("extra", [-1, 0, 1, 2])
def test_copies_around_the_size_that_takes_the_lanes(extra):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")

    pj = synth.build_polyjectory(synth.base_elements(3, np.random.default_rng(1), 0.0), 0.05, order=18)
    t = np.random.default_rng(2).uniform(0.0, 0.05, (16 << 20) // (3 * 56) + extra)
    got = pj.state_meval(t)
    for k in range(0, len(t), 10000):  # 1.7 MB at a time: one copy
        part = pj.state_meval(t[k:k + 10000])
        assert np.array_equal(got[:, k:k + 10000].view(np.uint64), part.view(np.uint64))
