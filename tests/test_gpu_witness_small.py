"""Witness generation on both sides of the small form's limit (csrc/witness.cu:
2^14 slots) and with a ragged last block, against the oracle."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_log,n", [(4, 16), (4, 9), (8, 129), (14, 16384), (14, 9000), (15, 16385)])
def test_witness_around_the_small_form(cuda_device, n_log, n):
    import torch

    import flock_challenge_gb300 as F

    blocks = O.compressions(n_log, 900 + n)[:n]
    d = torch.from_numpy(blocks.view(np.uint8).copy()).cuda()
    got = F.generate_witness(d, n, n_log)
    torch.cuda.synchronize()
    for g, w in zip(got, O.witness(blocks, n_log)):
        assert np.array_equal(g.cpu().numpy(), np.ascontiguousarray(w).view(np.uint8))
