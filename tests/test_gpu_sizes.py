"""Proof bytes against the oracle's at sizes whose level shapes differ (code
sizes and rates of the recursive opening, grids of the round kernels)."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2", [9, 11, 12, 13, 15])
def test_proofs_match_oracle_across_sizes(cuda_device, log2):
    import flock_challenge_gb300 as F

    blocks = O.compressions(log2, 1000 + log2)
    got = F.Blake3Setup(1 << log2).prove_fast(blocks)
    want = O.prove(blocks, log2)
    assert len(got) == len(want)
    assert np.array_equal(np.frombuffer(got, np.uint8), np.frombuffer(want, np.uint8))
