"""The deep-table pass beyond 64 lanes, and the one-layer table pass that goes
first where pairs of table layers would end a layer off it (csrc/ntt.cu), against
the oracle: the pass fixed, or through the autotuner, whose candidates all write
the transform (tuned shapes are checked whichever it picks)."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_d,log_lanes,start,variant", [
    (9, 7, 0, "3"), (10, 7, 1, "3"),  # 128 lanes, three layers left
    (5, 6, 1, None), (9, 6, 1, None), (12, 6, 0, None), (15, 6, 1, None),  # 64 lanes, an odd number of table layers
    (9, 8, 0, None), (10, 8, 1, None), (11, 8, 2, None)])
def test_ntt_deep_table_pass_wide_codes(cuda_device, monkeypatch, log_d, log_lanes, start, variant):
    import torch

    import flock_challenge_gb300 as F

    if variant:
        monkeypatch.setenv("FLOCK_NTT_VARIANT", variant)
    rng = np.random.default_rng(log_d * 23 + log_lanes + start)
    data = rng.integers(0, 2**63, (1 << (log_d + log_lanes)) * 2, dtype=np.uint64)
    data |= rng.integers(0, 2, data.shape, dtype=np.uint64) << np.uint64(63)
    d = torch.from_numpy(data.view(np.uint8).copy()).cuda()
    F.ntt(F.Context(0), d, log_d, log_lanes, start)
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint64), O.ntt_interleaved(data, 1 << log_lanes, start))
