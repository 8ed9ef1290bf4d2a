"""The step sort that the autotuner can choose (needs a B200) is the default's."""

import numpy as np
import pytest

from mizuba_b200 import synth

pytestmark = pytest.mark.gpu


def test_tuned_sort_is_no_slower_than_the_default():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    pj = synth.build_polyjectory(synth.base_elements(20000, np.random.default_rng(2)), 0.1)  # 48 steps

    def sort_ms(tuning):
        t = [mzb.device_conjunctions(pj, 2.0, 3.0 / 1440.0, form="mixed", tuning=tuning).stage_ms["morton_sort"]
             for _ in range(9)]
        return float(np.median(t))

    tuned = mzb.autotune(pj, 2.0, 3.0 / 1440.0)
    ms = sort_ms({"sort_threads": tuned["sort_threads"]}), sort_ms({})
    assert ms[0] < 1.1 * ms[1], ms
