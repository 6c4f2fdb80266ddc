"""Ligerito rounds on the tensor cores (csrc/ligerito.cu) start above 2^17 pairs:
proof bytes where the first folds have 2^18 pairs (2^13 compressions, the first
size that splits the first message off the basis), just below, and with ragged
inputs, and the chain relation, whose basis always stands alone."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 8191, 8192, 16000])
def test_tile_rounds_match_oracle(cuda_device, n):
    import flock_challenge_gb300 as F

    log2 = (n - 1).bit_length()
    blocks = O.compressions(log2, 31 + n)[:n]
    got = F.Blake3Setup(n).prove_fast(blocks)
    assert np.array_equal(np.frombuffer(got, np.uint8), np.frombuffer(O.prove(blocks, log2), np.uint8))


def test_tile_rounds_chain_matches_oracle(cuda_device):
    import flock_challenge_gb300 as F

    blocks = F.chain_inputs(1 << 13, 5)
    got = F.Blake3Setup(1 << 13).prove_chain(blocks)
    assert np.array_equal(np.frombuffer(got, np.uint8), np.frombuffer(O.prove_chain(blocks), np.uint8))
