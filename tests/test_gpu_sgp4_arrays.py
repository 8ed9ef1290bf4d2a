"""mzb_sgp4_propagate on arrays of every kind (needs a B200): device arrays at
odd byte offsets give what aligned ones and host arrays give."""

import itertools
import pathlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GPES = pathlib.Path(__file__).resolve().parent / "golden" / "gpes.npz"


@pytest.fixture(scope="module")
def lib():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200  # noqa: F401
    from mizuba_b200 import _native

    return _native.core()


def on_device(a, offset):
    """A copy of a in device memory, `offset` bytes behind an aligned address."""
    import torch

    raw = torch.zeros(a.nbytes + 64, dtype=torch.uint8, device="cuda")
    raw[offset:offset + a.nbytes] = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()
    return raw


def inputs(n=40, t=7):
    g = np.ascontiguousarray(np.load(GPES)["strack_20240705"][:n])
    return g, np.linspace(0.0, 1440.0, t)


def host_result(lib, g, ts, fill=0.0):
    out, err = np.full((len(g), len(ts), 6), fill), np.full((len(g), len(ts)), -1, np.int32)
    assert lib.mzb_sgp4_propagate(g.ctypes.data, len(g), ts.ctypes.data, len(ts), out.ctypes.data,
                                  err.ctypes.data) == 0, lib.mzb_last_error()
    return out, err


@pytest.mark.parametrize("offsets", list(itertools.product((0, 1, 4), (0, 4), (0, 2, 8), (0, 1))))
def test_unaligned_device_arrays(lib, offsets):
    g, ts = inputs()
    out, err = host_result(lib, g, ts)
    d = [on_device(a, o) for a, o in zip((g, ts, np.zeros_like(out), np.zeros_like(err)), offsets)]
    p = [x.data_ptr() + o for x, o in zip(d, offsets)]
    assert lib.mzb_sgp4_propagate(p[0], len(g), p[1], len(ts), p[2], p[3]) == 0, lib.mzb_last_error()
    got = [x.cpu().numpy()[o:o + a.nbytes] for x, o, a in zip(d[2:], offsets[2:], (out, err))]
    assert np.array_equal(got[0], out.view(np.uint8).reshape(-1))
    assert np.array_equal(got[1], err.view(np.uint8).reshape(-1))
    for x, o, a in zip(d[2:], offsets[2:], (out, err)):  # nothing beside them
        rest = x.cpu().numpy()
        assert not rest[:o].any() and not rest[o + a.nbytes:].any()


@pytest.mark.parametrize("device", [False, True])
def test_no_state_is_nan(lib, device):
    import torch

    g, ts = inputs(24)
    g["e0"][::3] = 0.999  # below the surface: an error at every time
    g["bstar"][1::3] = 0.5  # decays within the day
    out, err = host_result(lib, g, ts, fill=3.0)
    if device:
        d = [torch.from_numpy(a.view(np.uint8).reshape(-1).copy()).cuda() for a in (g, ts, np.full_like(out, 3.0), err)]
        assert lib.mzb_sgp4_propagate(d[0].data_ptr(), len(g), d[1].data_ptr(), len(ts), d[2].data_ptr(),
                                      d[3].data_ptr()) == 0, lib.mzb_last_error()
        out = d[2].cpu().numpy().view(np.float64).reshape(out.shape)
        err = d[3].cpu().numpy().view(np.int32).reshape(err.shape)
    state = (err == 0) | (err == 6)
    assert state.any() and (~state).any()
    assert np.isfinite(out[state]).all() and np.isnan(out[~state]).all()
