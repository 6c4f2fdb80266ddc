"""Waits inside the tensor-core kernels that run out (csrc/tc.cuh): the kernel ends
in order (its copies and MMAs first), the call returns a timeout, and the same
context then proves the oracle's bytes. A limit of zero gives up at the first
wait; the small limits run out, or do not, part way through."""
import ctypes

import numpy as np
import pytest

import flock_challenge_gb300 as F
import oracle_lib as O

pytestmark = pytest.mark.gpu


# 2^8 compressions: the stripe fold alone; 2^13: zerocheck and Ligerito rounds
# too; 2^14: the stripe fold of the c statistic comes first
@pytest.mark.parametrize("log2", [8, 13, 14])
def test_kernel_wait_limit_ends_in_a_timeout_and_the_context_recovers(cuda_device, log2):
    blocks = O.compressions(log2, 41 + log2)
    want = O.prove(blocks, log2)
    setup = F.Blake3Setup(1 << log2)
    for limit in (0, 1, 300, 1000, 3000, 10000, 0):
        setup.set_kernel_wait_limit(limit)
        try:
            got = setup.prove_fast(blocks)
            assert limit != 0 and got == want
        except F.FlockError as e:
            assert "timeout" in str(e)
    setup.set_kernel_wait_limit()
    assert setup.prove_fast(blocks) == want
    with pytest.raises(F.FlockError, match="argument"):
        setup.set_kernel_wait_limit((1 << 31) + 1)


class KernelWait(ctypes.Structure):
    _fields_ = [("fault", ctypes.c_void_p), ("limit", ctypes.c_uint32)]


# (a proof whose limit is zero never reaches its Ligerito rounds)
@pytest.mark.parametrize("fold", [0, 1])
def test_ligerito_round_gives_up_in_order(cuda_device, fold):
    import torch

    L = ctypes.CDLL(F.lib_path())
    launch = L._Z25flock_launch_lig_fold_msgPKvS0_miPKmPvS3_S3_iRK15FlockKernelWaitP11CUstream_st
    pairs = (1 << 17) + 128 * 200
    gen = torch.Generator(device="cuda").manual_seed(3)
    f, b = (torch.randint(-(1 << 63), (1 << 63) - 1, (4 * pairs << fold,), dtype=torch.int64, device="cuda",
                          generator=gen) for _ in range(2))
    out = torch.zeros(2, 4 * pairs, dtype=torch.int64, device="cuda")
    grid = L._Z19flock_lig_fold_gridm(ctypes.c_size_t(pairs))
    r = (ctypes.c_uint64 * 2)(0x0123456789ABCDEF, 0xFEDCBA9876543210)

    def run(limit):
        part = torch.zeros(grid, 3, 2, dtype=torch.int64, device="cuda")
        fault = torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = KernelWait(fault.data_ptr(), limit)
        rc = launch(F._dptr(f), F._dptr(b), ctypes.c_size_t(2 * pairs), fold, r, F._dptr(out[0]), F._dptr(out[1]),
                    F._dptr(part), grid, ctypes.byref(kw), None)
        assert rc == 0
        torch.cuda.synchronize()
        return int(fault[0]), part.cpu().numpy()

    ok, want = run(1 << 31)
    assert ok == 0 and want[:, :2].any()
    for limit in (0, 1, 300, 1000, 0):
        gave_up, got = run(limit)
        assert gave_up or (limit and np.array_equal(got, want))
    ok, got = run(1 << 31)
    assert ok == 0 and np.array_equal(got, want)
