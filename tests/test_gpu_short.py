"""The kernels of short operands at the edges of their ranges: the one-CTA
schoolboy product (up to 1024 limbs), sums alone in their call (over the whole
GPU from 2^13 limbs on), and the scaled last pass of the spectrum entry
point, against exact integers and the oracle."""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64).copy()).cuda()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (31, 1), (32, 1), (33, 31), (48, 64 - 48), (64, 48), (100, 100),
                                   (924, 100), (512, 512), (1023, 1), (1000, 24), (1024, 1), (925, 100), (600, 500)])
def test_schoolboy(hg, oracle, nx, ny):
    from hypergeometrica_gb300 import device as D

    if nx < ny:
        nx, ny = ny, nx
    for dist in ("uniform", "ones", "sparse"):
        x, y = W.limbs(nx, nx, dist), W.limbs(7 * ny, ny, dist)
        want = hg.int_from_digits(x) * hg.int_from_digits(y)
        got = hg.multiply_storage_schoolboy(x, nx, y, ny)
        assert len(got) == nx + ny + 1 and hg.int_from_digits(got) == want
        import torch

        out = torch.full((nx + ny + 3,), -1, dtype=torch.int64, device="cuda")
        D.mul_schoolboy(_dev(x), _dev(y), out)
        D.sync()
        assert hg.int_from_digits(out.cpu().numpy().view(np.uint64)) == want


@pytest.mark.parametrize("n", [8191, 8192, 20000, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 300001])
def test_sums_alone(hg, n):
    """Carries and borrows through the whole length, cancelled tops, equal operands, twice in a row."""
    import torch

    from hypergeometrica_gb300 import series as S

    ones = np.full(n, np.uint64(2**64 - 1))
    one = np.array([1], dtype=np.uint64)
    top = np.zeros(n, dtype=np.uint64)
    top[-1] = 1
    u = W.limbs(n, n)
    low = u.copy()
    low[: n // 3] = W.limbs(n + 1, n // 3)
    cases = [(ones, one, 1, 1), (top, one, 1, -1), (one, top, 1, -1), (u, low, 1, -1), (low, u, -1, 1), (u, u, 1, -1),
             (u, ones, -1, -1), (u, one, 1, -1)]
    for a, b, sa, sb in cases:
        v = sa * hg.int_from_digits(a) + sb * hg.int_from_digits(b)
        for _ in range(2):
            ta, tb = _dev(a), _dev(b)
            out = torch.full((n + 2,), -1, dtype=torch.int64, device="cuda")
            rec = np.array([[ta.data_ptr(), len(a), tb.data_ptr(), len(b), out.data_ptr(), n + 2,
                             np.int64(sa).view(np.uint64), np.int64(sb).view(np.uint64)]], dtype=np.uint64)
            torch.cuda.synchronize()
            (sg, size), = S._sum_records(rec)
            assert hg.int_from_digits(out.cpu().numpy().view(np.uint64)) == abs(v)
            assert (int(sg), int(size)) == (-1 if v < 0 else 1, (abs(v).bit_length() + 63) // 64)


@pytest.mark.parametrize("L", [1, 3, 4, 9, 12, 13, 16, 17, 20])
@pytest.mark.parametrize("offset", [0, 1])
def test_spectrum_scaling(hg, L, offset):
    """ntt-reverse of ntt-forward returns the residues, canonical, also from
    an array on an odd 8-byte boundary (the passes without tile copies)."""
    import torch

    from hypergeometrica_gb300 import device as D

    for mod, p in enumerate(hg.scheme_moduli()):
        a = (W.limbs(L + mod, 1 << L) % np.uint64(p)).astype(np.uint64)
        a[:: 5] = p - 1
        t = torch.zeros((1 << L) + 1, dtype=torch.int64, device="cuda")[offset: offset + (1 << L)]
        t.copy_(_dev(a))
        D.ntt_forward(t, mod)
        D.ntt_reverse(t, mod)
        D.sync()
        assert np.array_equal(t.cpu().numpy().view(np.uint64), a), (L, mod)
