"""Table passes of fixed depths (csrc/ntt.cu, FLOCK_NTT_TAB_END) against the oracle:
the one-layer table pass, first and alone, in front of the deep-table pass,
and stage passes behind table passes, in place and from a replicated message.
The launches of a call say that these passes are what ran."""
import ctypes

import numpy as np
import pytest

import flock_challenge_gb300 as F
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _fix(monkeypatch, variant, te):
    monkeypatch.setenv("FLOCK_NTT_VARIANT", variant)
    monkeypatch.setenv("FLOCK_NTT_TAB_END", str(te))


def _passes(variant, log_d, start, te):
    """Launches: pairs of table layers (one alone where odd), then one deep-table pass or stage passes of up to seven."""
    return (te - start + 1) // 2 + (1 if variant == "3" else (log_d - te + 6) // 7)


def _random(n, seed):
    rng = np.random.default_rng(seed)
    data = rng.integers(0, 2**63, 2 * n, dtype=np.uint64)
    return data | rng.integers(0, 2, data.shape, dtype=np.uint64) << np.uint64(63)


# te - start odd: the one-layer pass is first. Its blocks: one (layer 0) to 2^7, of 64 to 2^14 items.
DEEP = [("3", log_d, lanes, start, log_d - 3) for log_d, lanes, start in
        [(4, 6, 0), (5, 6, 1), (9, 6, 1), (9, 6, 0), (12, 6, 0), (11, 6, 7), (15, 6, 1), (8, 7, 0), (10, 8, 2), (7, 8, 4)]]
# stage passes from the end of no, one (odd and even) and several table passes, one and two of them, two layers left
STAGE = [("4", log_d, 3, start, te) for log_d, start, te in
         [(6, 0, 1), (8, 0, 2), (9, 2, 7), (12, 1, 4), (12, 1, 5), (15, 0, 6), (16, 2, 6), (16, 2, 9), (16, 2, 14)]]


@pytest.mark.parametrize("variant,log_d,lanes,start,te", DEEP + STAGE)
def test_ntt_from_fixed_table_ends_matches_oracle(cuda_device, monkeypatch, variant, log_d, lanes, start, te):
    import torch

    _fix(monkeypatch, variant, te)
    data = _random(1 << (log_d + lanes), log_d * 29 + lanes + start + te)
    want = O.ntt_interleaved(data, 1 << lanes, start)
    ctx, launches = F.Context(0), F._proto_lib().flock_kernel_launches
    for _ in range(2):  # the first call of a size makes its twiddles
        d = torch.from_numpy(data.view(np.uint8).copy()).cuda()
        before = launches()
        F.ntt(ctx, d, log_d, lanes, start)
        ran = launches() - before
        torch.cuda.synchronize()
        assert np.array_equal(d.cpu().numpy().view(np.uint64), want)
    assert ran == _passes(variant, log_d, start, te)


# the message replicated by the first pass: one-layer table pass, two-layer one, stage pass (level codes of 8 lanes)
@pytest.mark.parametrize("variant,rows_log,lanes,rate,te", [
    ("3", 8, 6, 1, 6), ("3", 4, 6, 1, 2), ("3", 9, 8, 2, 8), ("3", 8, 7, 3, 8), ("3", 9, 6, 1, 7), ("4", 9, 3, 2, 2),
    ("4", 9, 3, 1, 2), ("4", 12, 3, 1, 3)])
def test_replicated_message_from_fixed_table_ends_matches_oracle(cuda_device, monkeypatch, variant, rows_log, lanes,
                                                                 rate, te):
    import torch

    _fix(monkeypatch, variant, te)
    launch = ctypes.CDLL(F.lib_path())._Z16flock_launch_nttPvPKviiiP11CUstream_st
    z = _random(1 << (rows_log + lanes), rows_log + lanes + rate + te)
    src = torch.from_numpy(z.view(np.uint8).copy()).cuda()
    dst = torch.zeros(src.numel() << rate, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        before = F._proto_lib().flock_kernel_launches()
        assert launch(F._dptr(dst), F._dptr(src), rows_log + rate, lanes, rate, None) == 0
    assert F._proto_lib().flock_kernel_launches() - before == _passes(variant, rows_log + rate, rate, te)
    torch.cuda.synchronize()
    want = O.ntt_interleaved(np.tile(z, 1 << rate), 1 << lanes, rate)
    assert np.array_equal(dst.cpu().numpy().view(np.uint64), want)
    assert np.array_equal(src.cpu().numpy().view(np.uint64), z)
