"""A batch of 2^32 broad-phase pairs or more is refused (needs a B200), also
where the pairs of 8,192 neighbouring objects alone exceed 2^32 by a little."""

import numpy as np
import pytest

from mizuba_b200.polyjectory import polyjectory

pytestmark = pytest.mark.gpu


def test_too_many_pairs():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mizuba_b200 as mzb

    # 8,192 objects that sweep the whole space and as many points as bring the
    # pairs, all filed under the former, just above 2^32.
    big = 8192
    small = (2**32 - big * (big - 1) // 2) // big + 8
    n = big + small
    pairs = big * small + big * (big - 1) // 2
    assert 2**32 < pairs < 2**32 + n  # modulo 2^32 it would fit the queue
    c = np.zeros((n, 3, 7))
    c[:big, 0, :3] = -1000.0
    c[:big, 1, :3] = 2000.0
    c[:big, 1, 6] = 2000.0
    k = np.arange(small)
    pos = np.stack([k % 81, k // 81 % 81, k // 6561], axis=1) * 20.0 - 800.0
    c[big:, 0, :3] = pos
    c[big:, 0, 6] = np.linalg.norm(pos, axis=1)
    pj = polyjectory.from_arrays(c.reshape(-1), np.stack([np.arange(n) * 21, np.ones(n)], axis=1),
                                 np.tile([0.0, 1.0], n), np.arange(n) * 2, np.zeros(n, np.int32), 2)
    with pytest.raises(RuntimeError, match="too many broad-phase pairs"):
        mzb.device_conjunctions(pj, 1e-3, 1.0)
    torch.cuda.synchronize()
