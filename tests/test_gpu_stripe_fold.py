"""Lincheck's stripe fold (csrc/lincheck.cu) runs on every proof: proof bytes at
the edges of its stages of 256 outer indices and of its split of the stages over
parts (one stage at 2^8, a part per stage up to 2^10, uneven parts above)."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 257, 1024, 1025, 2049])
def test_stripe_fold_edges_match_oracle(cuda_device, n):
    import flock_challenge_gb300 as F

    log2 = max(8, (n - 1).bit_length())
    blocks = O.compressions(log2, 77 + n)[:n]
    got = F.Blake3Setup(n).prove_fast(blocks)
    assert np.array_equal(np.frombuffer(got, np.uint8), np.frombuffer(O.prove(blocks, log2), np.uint8))
