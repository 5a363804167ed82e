"""Truncated transforms where the other tests do not reach: operands that come
from host memory in column slices, and outer passes without a twiddle table.
Each product equals the whole transform's (set_chunking(False)) limb for limb."""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _whole(x, y):
    """|x| |y| of device tensors by the whole transform on limbs."""
    import torch

    from hypergeometrica_gb300 import device as D
    from hypergeometrica_gb300._lib import set_chunking

    out = torch.empty(x.numel() + y.numel(), dtype=torch.int64, device="cuda")
    assert set_chunking(False)
    try:
        D.mul(x, y, out)
        D.sync()
    finally:
        set_chunking(True)
    return out


# (nx, ny) of products on 80-bit digits whose first pass runs slice by slice
# (from 2^19 points) and keeps 14 sixteenths of 2^19 points (128 rows of 4096
# digits, 5120 limbs), 15 of 2^20 (256 rows), 10 of 2^21 and 11 of 2^22 (16
# rows of 2^17 and 2^18 digits).  The lengths leave a partial row of an odd
# number of limbs, of one limb, or none; 327680 and 655360 limbs just fill the
# lower half of 2^19 and 2^20 points.
SLICED = [(300001, 260000), (327680, 232321), (700001, 500003), (655360, 500001), (640001, 560000),
          (1000003, 600011), (1638401, 1700003)]


@pytest.mark.parametrize("nx, ny", SLICED)
def test_sliced_uploads_on_digits(hg, nx, ny):
    import torch

    from hypergeometrica_gb300._lib import check
    from hypergeometrica_gb300.mpz import mul_host_pipeline

    x, y = W.limbs(nx, nx), W.limbs(ny + 1, ny, "ones" if ny % 2 else "uniform")
    want = _whole(*(torch.from_numpy(a.view(np.int64)).cuda() for a in (x, y))).cpu().numpy().view(np.uint64)
    for pinned in (False, True):
        hx, hy, out = x, y, np.full(nx + ny + 3, 7, dtype=np.uint64)
        if pinned:
            hx, hy, out = (torch.from_numpy(a.view(np.int64)).pin_memory().numpy().view(np.uint64) for a in (hx, hy, out))
        check(hg.load().hg_mul(hx.ctypes.data, nx, hy.ctypes.data, ny, out.ctypes.data, len(out)))
        assert np.array_equal(out[:nx + ny], want) and not out[nx + ny:].any(), pinned
        outs = [np.full(nx + ny, 7, dtype=np.uint64) for _ in range(3)]
        mul_host_pipeline([(hx, hy, o) for o in outs])
        for o in outs:
            assert np.array_equal(o, want), pinned


def test_no_table_above_2_27_points(hg):
    """Passes over more than 2^27 points form their twiddles: 9 sixteenths of
    2^28 points on digits, from device memory (two operands of 88 million
    limbs)."""
    import torch

    from hypergeometrica_gb300 import device as D

    g = torch.Generator(device="cuda").manual_seed(28)
    x, y = (torch.randint(-2**63, 2**63 - 1, (n,), generator=g, device="cuda") for n in (88000001, 87999998))
    got = torch.full((x.numel() + y.numel(),), -1, dtype=torch.int64, device="cuda")
    D.mul(x, y, got)
    D.sync()
    assert torch.equal(got, _whole(x, y))
