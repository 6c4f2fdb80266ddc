"""Zerocheck's multilinear rounds across the forms of csrc/zerocheck.cu: grouped
and small rounds (2^11), rounds 0..5 on the tensor cores from 2^12 on, where the
weighted variables grow with the size (six at 2^12 and 2^13, nine at 2^16), with
ragged inputs: proof bytes against the oracle's."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048, 2049, 4096, 6000, 1 << 15, 1 << 16])
def test_zerocheck_round_forms_match_oracle(cuda_device, n):
    import flock_challenge_gb300 as F

    log2 = (n - 1).bit_length()
    blocks = O.compressions(log2, 53 + n)[:n]
    got = F.Blake3Setup(n).prove_fast(blocks)
    assert np.array_equal(np.frombuffer(got, np.uint8), np.frombuffer(O.prove(blocks, log2), np.uint8))
