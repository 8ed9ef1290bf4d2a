"""Step sort of catalogues with objects without data and with clusters (needs a
B200): their order is that of a stable sort, and neither costs a step much more
than one without them."""

import numpy as np
import pytest

from mizuba_b200.polyjectory import polyjectory

pytestmark = pytest.mark.gpu


def scattered_pj(n, empty, seed):
    """n points over a box, the given ones without data: codes that vary in
    all their bits, hardly two with equal top bits."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1000.0, 1000.0, (n, 3))
    trajs, times = [], []
    for k in range(n):
        c = np.zeros((0 if k in empty else 1, 3, 7))
        if len(c):
            c[0, 0, :3] = pos[k]
            c[0, 0, 6] = np.linalg.norm(pos[k])
        trajs.append(c)
        times.append(np.array([0.0, 1.0][:2 * len(c)]))
    return polyjectory(trajs, times, [0] * n)


@pytest.mark.parametrize("n", [2049, 6000])
def test_no_data_objects(n):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    kinds = np.full(n, 2, np.int32)  # secondaries only: no pairs to narrow
    kinds[0] = 1
    ms = {}
    for k in (0, 1, 64, 65, 66, 500, n - 65, n - 1):
        empty = set(np.random.default_rng(k).choice(np.arange(1, n), k, replace=False).tolist())
        pj = scattered_pj(n, empty, seed=n)
        t = []
        for _ in range(9):
            g = mzb.device_conjunctions(pj, 1e-3, 1.0 / 192, otypes=kinds)
            t.append(g.stage_ms["morton_sort"])
        ms[k] = float(np.median(t))
        for s in (0, 191):
            assert np.array_equal(g.srt_idx[s], np.lexsort((np.arange(n), g.mcodes[s], [i in empty for i in range(n)])))
            assert np.array_equal(g.srt_mcodes[s], g.mcodes[s][g.srt_idx[s]])
            assert np.array_equal(g.srt_aabbs[s][:n], g.aabbs[s][g.srt_idx[s]])
    assert ms[66] < 1.4 * ms[64] and ms[500] < 1.4 * ms[64], ms


@pytest.mark.parametrize("size", [8, 9, 32, 33, 60])
def test_many_runs(size):
    """Many clusters whose members share the top bits: runs ordered by a thread
    or by a warp each, in about the time of a step without any."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    n, steps = 6000, 192
    kinds = np.full(n, 2, np.int32)
    kinds[0] = 1
    ms = []
    for clusters in (0, 60):
        rng = np.random.default_rng(size)
        pos = rng.uniform(-1000.0, 1000.0, (n, 3))
        cells = np.floor(rng.uniform(-400.0, 400.0, (clusters, 3))) * (2000.0 / 1024)
        pos[:clusters * size] = np.repeat(cells, size, axis=0) + rng.uniform(0.6, 1.0, (clusters * size, 3))
        pos = pos[rng.permutation(n)]
        trajs = np.zeros((n, 1, 3, 7))
        trajs[:, 0, 0, :3] = pos
        trajs[:, 0, 0, 6] = np.linalg.norm(pos, axis=1)
        pj = polyjectory(list(trajs), [np.array([0.0, 1.0])] * n, [0] * n)
        t = []
        for _ in range(9):
            g = mzb.device_conjunctions(pj, 1e-3, 1.0 / steps, otypes=kinds)
            t.append(g.stage_ms["morton_sort"])
        ms.append(float(np.median(t)))
        for s in (0, steps - 1):
            assert np.array_equal(g.srt_idx[s], np.lexsort((np.arange(n), g.mcodes[s])))
            assert np.array_equal(g.srt_mcodes[s], g.mcodes[s][g.srt_idx[s]])
    assert ms[1] < 1.7 * ms[0], ms
