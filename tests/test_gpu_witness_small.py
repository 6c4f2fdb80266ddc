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


def test_witness_into_buffers_on_an_8_byte_boundary(cuda_device):
    import torch

    import flock_challenge_gb300 as F

    n_log, n = 4, 9
    blocks = O.compressions(n_log, 77)[:n]
    d = torch.from_numpy(blocks.view(np.uint8).copy()).cuda()
    nbytes = (1 << (14 + n_log)) // 8
    bufs = [torch.zeros(nbytes + 16, dtype=torch.uint8, device="cuda") for _ in range(3)]
    stripe = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    F.check(F.lib().flock_witness(F._dptr(d), n, n_log, *(F._dptr(b[8:]) for b in bufs), F._dptr(stripe), None),
            "flock_witness")
    torch.cuda.synchronize()
    got = [b[8:8 + nbytes] for b in bufs] + [stripe]
    for g, w in zip(got, O.witness(blocks, n_log)):
        assert np.array_equal(g.cpu().numpy(), np.ascontiguousarray(w).view(np.uint8))
    assert all(int(b[:8].sum()) == 0 and int(b[8 + nbytes:].sum()) == 0 for b in bufs)
