"""Shifts of hg_sums_and_sizes at the end of their range are refused by the
host, with nothing written."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("shift", [2**64 - 1 - 5, 2**64 - 5, 2**64 - 1, 2**61, 11])
def test_shift_past_the_result(hg, shift, sign):
    """Five limbs moved up by `shift` end at 2^64 - 1, past 2^64, far past the
    result, and one limb past it; the last end leaves the carry no room."""
    import torch

    from hypergeometrica_gb300._lib import HG_ERR_ARG, HgSum, load

    a = torch.ones(5, dtype=torch.int64, device="cuda")
    out = torch.full((16,), -7, dtype=torch.int64, device="cuda")
    res = (ctypes.c_int64 * 2)(-7, -7)
    torch.cuda.synchronize()
    s = HgSum(a.data_ptr(), 5, a.data_ptr(), 5, out.data_ptr(), 16, 1, sign)
    up, none = ctypes.c_size_t(shift), ctypes.c_size_t(0)
    rc = load().hg_sums_and_sizes(ctypes.byref(s), ctypes.byref(up), ctypes.byref(none), 1, res, None, 0, None,
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == HG_ERR_ARG
    torch.cuda.synchronize()
    assert list(res) == [-7, -7] and bool((out == -7).all())
