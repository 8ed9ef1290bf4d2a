"""Results copied to pageable memory and files piece by piece (needs a B200):
sizes around the piece and the size from which several threads share the
work, each compared with the same data fetched in one small piece."""

import os

import numpy as np
import pytest

from mizuba_b200 import synth

pytestmark = pytest.mark.gpu
PIECE = 2 << 20


@pytest.fixture(scope="module")
def mzb():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200

    return mizuba_b200


@pytest.mark.parametrize("extra", [-1, 0, 1, 40])
@pytest.mark.parametrize("pieces", [1, 2, 3, 11])
def test_states(mzb, pieces, extra):
    pj = synth.build_polyjectory(synth.base_elements(3, np.random.default_rng(1), 0.0), 0.05, order=18)
    n_t = pieces * PIECE // (3 * 56) + extra
    t = np.random.default_rng(2).uniform(0.0, 0.05, n_t)
    got = pj.state_meval(t)
    for k in range(0, n_t, 10000):  # 1.7 MB at a time: one copy
        part = pj.state_meval(t[k:k + 10000])
        assert np.array_equal(got[:, k:k + 10000].view(np.uint64), part.view(np.uint64))


def test_files_and_arrays(mzb, tmp_path):
    pj = synth.build_polyjectory(synth.base_elements(1500, np.random.default_rng(4), 0.0), 0.2, order=18)
    d = mzb.device_conjunctions(pj, 20.0, 3.0 / 1440.0)
    c = mzb.conjunctions(pj, 20.0, 3.0 / 1440.0, data_dir=str(tmp_path / "out"))
    for key in ("aabbs", "srt_aabbs", "mcodes", "srt_mcodes", "srt_idx", "conjunctions"):
        a, b = getattr(d, key), getattr(c, key)
        assert a.nbytes > 0 and np.array_equal(np.ascontiguousarray(a).view(np.uint8),
                                               np.ascontiguousarray(b).view(np.uint8)), key
    assert os.path.getsize(tmp_path / "out" / "bvh") > 4 * PIECE
    for k in range(d.n_cd_steps):
        assert np.array_equal(d.get_bvh_tree(k).view(np.uint8), c.get_bvh_tree(k).view(np.uint8))
        assert np.array_equal(d.get_aabb_collisions(k).view(np.uint8), c.get_aabb_collisions(k).view(np.uint8))
