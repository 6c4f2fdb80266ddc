"""Zerocheck's grouped rounds (csrc/zerocheck.cu) from 2^12 compressions on, which a
proof takes whose outer challenges hold a 0 or 1 (FLOCK_ZC_MMA=0 takes them for
every proof): two, three and six grouped rounds, then the hand-over of the eq
tables to the small or the plain rounds. Proof bytes against the oracle's."""
import pytest

import flock_challenge_gb300 as F
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 8191, 1 << 16])
def test_grouped_rounds_match_oracle(cuda_device, monkeypatch, n):
    log2 = (n - 1).bit_length()
    blocks = O.compressions(log2, 19 + n)[:n]
    want = O.prove(blocks, log2)
    setup, launches = F.Blake3Setup(n), F._proto_lib().flock_kernel_launches
    ran = {}
    for mma in ("1", "0"):
        monkeypatch.setenv("FLOCK_ZC_MMA", mma)
        for _ in range(2):  # the first proof of a size tunes its transforms
            before = launches()
            assert setup.prove_fast(blocks) == want
        ran[mma] = launches() - before
    # the tensor-core rounds' fold of A and its unweighting fall away
    assert ran["1"] - ran["0"] == 2
