"""The tensor-core kernels by themselves where their counts are largest: operands
of all ones, one pair left out of every block's accumulation, so that each
count is odd and its parity one. The last size of each is that of the largest proof
(2^21 compressions), whose counts reach 883,071 and 299,775."""
import ctypes

import numpy as np
import pytest

import flock_challenge_gb300 as F
import oracle_lib as O

pytestmark = pytest.mark.gpu

ONES = (1 << 128) - 1


class KernelWait(ctypes.Structure):
    _fields_ = [("fault", ctypes.c_void_p), ("limit", ctypes.c_uint32)]


def _words(x):
    return np.array([x & (2**64 - 1), x >> 64], np.uint64)


def _product():
    ones = _words(ONES)
    return np.array(O.gf_mul(ones, ones), np.uint64)


@pytest.mark.parametrize("fold,pairs", [(0, (1 << 17) + 128), (0, 1 << 27), (1, (1 << 17) + 128), (1, 1 << 26)])
def test_ligerito_round_counts(cuda_device, fold, pairs):
    import torch

    L = ctypes.CDLL(F.lib_path())
    launch = L._Z25flock_launch_lig_fold_msgPKvS0_miPKmPvS3_S3_iRK15FlockKernelWaitP11CUstream_st
    grid = L._Z19flock_lig_fold_gridm(ctypes.c_size_t(pairs))
    # a pair's values (all ones, 0); with a fold each of them twice, which any challenge folds to itself
    f, b = (torch.zeros(pairs, 2, 1 + fold, 2, dtype=torch.int64, device="cuda") for _ in range(2))
    f[:, 0] = -1
    b[:, 0] = -1
    tiles = pairs // 128
    f[[128 * (tiles * c // grid) for c in range(grid)], 0] = 0
    out = torch.zeros((2, pairs, 2, 2) if fold else (2, 1), dtype=torch.int64, device="cuda")
    part = torch.zeros(grid, 3, 2, dtype=torch.int64, device="cuda")
    fault = torch.zeros(1, dtype=torch.int32, device="cuda")
    r = (ctypes.c_uint64 * 2)(0x0123456789ABCDEF, 0xFEDCBA9876543210)
    kw = KernelWait(fault.data_ptr(), 1 << 31)
    rc = launch(F._dptr(f), F._dptr(b), ctypes.c_size_t(2 * pairs), fold, r, F._dptr(out[0]), F._dptr(out[1]),
                F._dptr(part), grid, ctypes.byref(kw), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(fault[0]) == 0
    want = np.broadcast_to(_product(), (grid, 2, 2))
    assert np.array_equal(part.cpu().numpy().view(np.uint64)[:, :2], want)
    if fold:
        assert torch.equal(out[0], f[:, :, 0]) and torch.equal(out[1], b[:, :, 0])


@pytest.mark.parametrize("n_stripes", [32, 1 << 18])
def test_stripe_fold_counts(cuda_device, n_stripes):
    import torch

    L = ctypes.CDLL(F.lib_path())
    launch = L._Z20flock_launch_lc_foldPKvmS0_S0_iPvS1_RK15FlockKernelWaitP11CUstream_st
    L._Z27flock_lc_fold_scratch_bytesm.restype = ctypes.c_size_t
    cols, bits = 1 << 14, (8 * n_stripes).bit_length() - 1
    stages = n_stripes // 32
    parts = min(stages, 7)
    stripe = torch.full((n_stripes, cols), 255, dtype=torch.uint8, device="cuda")
    for p in range(parts):
        stripe[32 * (stages * p // parts)] = 254  # one outer index of the part
    lo_bits = bits // 2
    lo = torch.full((1 << lo_bits, 2), -1, dtype=torch.int64, device="cuda")
    hi = torch.zeros(1 << (bits - lo_bits), 2, dtype=torch.int64, device="cuda")
    hi[:, 0] = 1
    scratch = torch.zeros(L._Z27flock_lc_fold_scratch_bytesm(ctypes.c_size_t(n_stripes)), dtype=torch.uint8, device="cuda")
    z_vec = torch.zeros(cols, 2, dtype=torch.int64, device="cuda")
    fault = torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = KernelWait(fault.data_ptr(), 1 << 31)
    rc = launch(F._dptr(stripe), ctypes.c_size_t(n_stripes), F._dptr(lo), F._dptr(hi), lo_bits, F._dptr(scratch),
                F._dptr(z_vec), ctypes.byref(kw), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(fault[0]) == 0
    assert parts % 2 == 1 and bool((z_vec == -1).all())
    if parts > 1:  # each part's sums, behind the expanded eq bits (512 bytes per stripe)
        sums = scratch[512 * n_stripes:512 * n_stripes + parts * cols * 16]
        assert bool((sums == 255).all())
