"""A prover without pinned host memory (FLOCK_PINNED=0, as where it cannot be had):
the same proofs and verdicts, and a kernel whose wait gave up is still reported."""
import pytest

import flock_challenge_gb300 as F
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2", [8, 11, 13, 14])
def test_unpinned_prover_proves_and_reports_give_ups(cuda_device, monkeypatch, log2):
    monkeypatch.setenv("FLOCK_PINNED", "0")
    blocks = O.compressions(log2, 71 + log2)
    want = O.prove(blocks, log2)
    setup = F.Blake3Setup(1 << log2)
    assert setup.prove_fast(blocks) == want
    assert F.verify(want, ctx=setup.ctx)
    setup.set_kernel_wait_limit(0)
    with pytest.raises(F.FlockError, match="timeout"):
        setup.prove_fast(blocks)
    setup.set_kernel_wait_limit()
    assert setup.prove_fast(blocks) == want


def test_unpinned_prover_proves_chains(cuda_device, monkeypatch):
    monkeypatch.setenv("FLOCK_PINNED", "0")
    blocks = F.chain_inputs(1 << 12, 9)
    assert F.Blake3Setup(1 << 12).prove_chain(blocks) == O.prove_chain(blocks)
