"""Device memory of SGP4 production and propagation (needs a B200): counted and
bounded while it is kept, given back to the device on release, and safe with
several threads."""

import pathlib
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GPES = pathlib.Path(__file__).resolve().parent / "golden" / "gpes.npz"
JD0 = 2460496.5


@pytest.fixture(scope="module")
def mzb():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200

    return mizuba_b200


def gpes(n):
    g = np.ascontiguousarray(np.load(GPES)["strack_20240705"])
    return np.ascontiguousarray(g[::len(g) // n][:n])


def test_memory_is_given_back(mzb):
    import torch

    mzb.make_sgp4_polyjectory(gpes(20), JD0, JD0 + 0.1)
    mzb.release_scratch()
    assert mzb.scratch_bytes() == 0
    before = torch.cuda.mem_get_info()[0]
    for n in (1500, 12000):  # 200 MB of coefficients, 1.6 GB
        pj, _ = mzb.make_sgp4_polyjectory(gpes(n), JD0, JD0 + 1.0)
        size = pj.arrays["traj"].nbytes
        del pj
        mzb.sgp4_propagate(gpes(100), np.linspace(0.0, 1440.0, 10))  # a synchronisation
        held = mzb.scratch_bytes()
        assert size <= held <= 2 << 30 if n == 1500 else held <= 2 << 30
        assert before - torch.cuda.mem_get_info()[0] <= held + (64 << 20)
    mzb.release_scratch()
    assert mzb.scratch_bytes() == 0
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_threads(mzb):
    jobs = [(gpes(60), 0.5), (gpes(300), 0.2), (gpes(40), 1.0)]

    def produce(k):
        pj, _ = mzb.make_sgp4_polyjectory(jobs[k][0], JD0, JD0 + jobs[k][1])
        st, err = mzb.sgp4_propagate(jobs[k][0], np.linspace(0.0, 1440.0, 30))
        return pj.arrays["traj"].tobytes(), pj.arrays["time"].tobytes(), st.tobytes(), err.tobytes()

    want = [produce(k) for k in range(len(jobs))]
    for _ in range(4):
        got = [None] * len(jobs)

        def work(k):
            got[k] = produce(k)

        ts = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert got == want
