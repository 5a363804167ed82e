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


@pytest.mark.parametrize("na,sa,nb,sb", [(3, 0, 5, 2), (5, 7, 3, 0), (1, 100, 100, 0), (2048, 1, 2047, 2), (4000, 4200, 8190, 0),
                                         (9000, 0, 1, 9000), (70000, 3, 70001, 2), (1, 1 << 17, 1 << 17, 0)])
def test_shifted_sums_and_sizes(hg, na, sa, nb, sb):
    """hg_sums_and_sizes: operands moved up by whole limbs, with the sizes of
    other integers in the same call."""
    import torch

    from hypergeometrica_gb300 import series as S

    u, v = W.limbs(na, na), W.limbs(nb + 1, nb)
    w = np.concatenate([W.limbs(3, 11), np.zeros(5000, dtype=np.uint64)])
    ta, tb, tw = _dev(u), _dev(v), _dev(w)
    n = max(na + sa, nb + sb)
    for ga, gb in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
        want = ga * (hg.int_from_digits(u) << (64 * sa)) + gb * (hg.int_from_digits(v) << (64 * sb))
        out = torch.full((n + 4,), -1, dtype=torch.int64, device="cuda")
        rec = np.array([[ta.data_ptr(), na, tb.data_ptr(), nb, out.data_ptr(), n + 4, np.int64(ga).view(np.uint64),
                         np.int64(gb).view(np.uint64)]], dtype=np.uint64)
        vecs = np.array([[tw.data_ptr(), w.size], [tw.data_ptr() + 8 * 11, 5000]] * 20, dtype=np.uint64)
        res, sizes = S._sums_and_sizes(rec, vecs, np.array([[sa], [sb]]))
        assert hg.int_from_digits(out.cpu().numpy().view(np.uint64)) == abs(want)
        assert tuple(res[0]) == (-1 if want < 0 else 1, (abs(want).bit_length() + 63) // 64)
        assert sizes.tolist() == [11, 0] * 20


@pytest.mark.parametrize("size", [2, 3, 1024, 1025, (1 << 17) - 1, 1 << 17, (1 << 17) + 1])
def test_staged_host_products(hg, size):
    """Host products on both sides of the staging buffer's limit, results longer
    than the product, operands with high zeros."""
    import ctypes

    from hypergeometrica_gb300._lib import check, load

    nx = size - size * 2 // 5
    x, y = W.limbs(size, nx, "ones"), W.limbs(size + 1, size - nx)
    xz = np.concatenate([x, np.zeros(7, dtype=np.uint64)])
    vx, vy = hg.int_from_digits(x), hg.int_from_digits(y)
    out = np.full(size + 9, np.uint64(7))
    check(load().hg_mul(xz.ctypes.data, xz.size, y.ctypes.data, y.size, out.ctypes.data, out.size))
    assert hg.int_from_digits(out) == vx * vy
    out = np.full(2 * nx + 1, np.uint64(7))
    check(load().hg_sqr(x.ctypes.data, nx, out.ctypes.data, out.size))
    assert hg.int_from_digits(out) == vx * vx
    out = np.full(nx + 3, np.uint64(7))
    check(load().hg_mul_digit(x.ctypes.data, nx, ctypes.c_uint64(0xFFFFFFFFFFFFFFF1), out.ctypes.data, out.size))
    assert hg.int_from_digits(out) == vx * 0xFFFFFFFFFFFFFFF1


def test_service_sized_products(hg):
    """hg_svc_mul from several threads, among submitted products, against the direct product."""
    import threading

    import torch

    from hypergeometrica_gb300 import device as D

    wrong = []
    with D.Service(workspace_bytes=256 << 20, slots=2) as svc:
        def client(k):
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for j in range(12):
                    nx, ny = 150 + 997 * j * (k + 1), 101 + 311 * j
                    x, y = _dev(W.limbs(100 * k + j, nx)), _dev(W.limbs(5000 + 100 * k + j, ny))
                    square = j % 3 == 2
                    n = 2 * nx if square else nx + ny
                    out, want = torch.empty(n, dtype=torch.int64, device="cuda"), torch.empty(n, dtype=torch.int64, device="cuda")
                    size = svc.mul(x.data_ptr(), nx, None if square else y.data_ptr(), 0 if square else ny, out.data_ptr(), n)
                    D.sqr(x, want) if square else D.mul(x, y, want)
                    torch.cuda.current_stream().synchronize()
                    w = want.cpu().numpy()
                    if not torch.equal(out, want) or size != int(np.flatnonzero(w)[-1]) + 1:
                        wrong.append((k, j))
        ts = [threading.Thread(target=client, args=(k,)) for k in range(3)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert not wrong
        st = svc.stats()
        assert st["completed"] == st["submitted"] == 36 and st["failed"] == 0
