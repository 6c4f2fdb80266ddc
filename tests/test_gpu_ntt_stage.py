"""Stage passes of 8-lane transforms (csrc/ntt.cu, shape 4) against the oracle:
the smallest (two layers), odd and even layer counts per pass, one pass of
seven layers, the first split into two, no start layer, wide and narrow twiddles."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_d,start", [(2, 0), (3, 0), (3, 1), (5, 0), (7, 0), (8, 0), (8, 1), (9, 2), (13, 2),
                                         (15, 0), (16, 3)])
def test_ntt_stage_passes_match_oracle(cuda_device, monkeypatch, log_d, start):
    import torch

    import flock_challenge_gb300 as F

    monkeypatch.setenv("FLOCK_NTT_VARIANT", "4")
    rng = np.random.default_rng(log_d * 19 + start)
    data = rng.integers(0, 2**63, (1 << (log_d + 3)) * 2, dtype=np.uint64)
    data |= rng.integers(0, 2, data.shape, dtype=np.uint64) << np.uint64(63)
    d = torch.from_numpy(data.view(np.uint8).copy()).cuda()
    F.ntt(F.Context(0), d, log_d, 3, start)
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint64), O.ntt_interleaved(data, 8, start))
