"""Truncated transforms and 80-bit digits: a product keeps 9 to 15 sixteenths
of the points where its size allows, and its coefficients may be digits of 80
bits.  Every length class that has its own plan (13 .. 22 bits: one or two
strided passes, outer passes of 16, 64, 128 and 256 rows) at the edges of each
cut, of limbs and of digits, against the oracle where that is quick and
against the whole transform on limbs (set_chunking(False)) limb for limb.
"""

import numpy as np
import pytest

from hypergeometrica_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch

    return torch.from_numpy(a.view(np.int64).copy()).cuda()


def _np(t):
    return t.cpu().numpy().view(np.uint64)


def _sizes(L):
    """Product sizes (limbs) around the cuts of 2^L points on limbs and of
    2^(L-1) and 2^L points on 80-bit digits, and odd ones between."""
    n, e = 1 << L, 1 << (L - 3)
    out = [n // 2 + 1, n - 1, n, n // 2 + e // 3, 6 * e + e // 5]
    for k in (5, 6, 7):
        out += [k * e - 1, k * e, k * e + 1]
    for k in range(9, 17):  # 5 limbs hold 4 digits
        for m in (L - 1, L):
            d = (k << (m - 4)) * 5 // 4
            if n // 2 < d <= n:
                out += [d - 5, d - 1, d]
    return out


@pytest.mark.parametrize("L", range(13, 23))
def test_products_and_squares(hg, oracle, L):
    import torch

    from hypergeometrica_gb300 import device as D
    from hypergeometrica_gb300._lib import set_chunking

    for j, size in enumerate(_sizes(L)):
        nx = size - size * (3 + j % 4) // 8
        ny = size - nx
        dist = ("uniform", "ones", "sparse")[j % 3]
        x, y = W.limbs(100 * L + j, nx, dist), W.limbs(7000 + 100 * L + j, ny, "uniform" if dist == "sparse" else dist)
        tx, ty = _dev(x), _dev(y)
        pad = (0, 1, 5000)[j % 3]  # limbs of out past the product, written as zeros
        got = torch.full((size + pad,), -1, dtype=torch.int64, device="cuda")
        D.mul(tx, ty, got)
        sq = torch.full((2 * (size // 2) + pad,), -1, dtype=torch.int64, device="cuda")
        D.sqr(tx, sq, nx=min(nx, size // 2))
        D.sync()
        if L <= 15:
            want = oracle.mpz_mul_ntt(x, y)[:size]
            wsq = oracle.mpz_square(x[: size // 2])[: 2 * min(nx, size // 2)]
        else:
            assert set_chunking(False)
            try:
                w, ws = torch.empty_like(got), torch.empty_like(sq)
                D.mul(tx, ty, w)
                D.sqr(tx, ws, nx=min(nx, size // 2))
                D.sync()
            finally:
                set_chunking(True)
            want, wsq = _np(w)[:size], _np(ws)
        assert np.array_equal(_np(got)[:size], want), (L, size)
        assert not _np(got)[size:].any(), (L, size)
        k = min(len(wsq), sq.numel())
        assert np.array_equal(_np(sq)[:k], wsq[:k]) and not _np(sq)[k:].any(), (L, size)


def test_host_products(hg, oracle):
    """hg_mul from host memory: column slices of a truncated outer pass."""
    for size in (5 << 10, (5 << 10) + 1, 6 << 11, 7 << 12, 21000, 23000):
        nx = size * 5 // 8
        x, y = W.limbs(size, nx), W.limbs(size + 1, size - nx)
        assert hg.int_from_digits(hg.mpz_mul_ntt(hg.MPZ(1, x), hg.MPZ(-1, y)).storage) == \
            hg.int_from_digits(oracle.mpz_mul_ntt(x, y))


@pytest.mark.parametrize("autotune", [False, True])
def test_batches(hg, autotune):
    """Mixed lengths and cuts in one batch, on both schedules, with results
    longer than the product; against products of whole transforms."""
    import torch

    from hypergeometrica_gb300 import device as D
    from hypergeometrica_gb300._lib import set_chunking

    sizes = sorted({s for L in (12, 13, 14, 15, 17, 18) for s in _sizes(L)})
    items, want = [], []
    assert set_chunking(False)
    try:
        for k, size in enumerate(sizes):
            nx = size * (4 + k % 3) // 8
            x = _dev(W.limbs(31 * k + 1, nx, ("uniform", "ones")[k % 2]))
            y = None if k % 5 == 4 else _dev(W.limbs(31 * k + 2, size - nx))
            n = 2 * nx if y is None else size
            nout = n + (0, 3, 9000)[k % 3]
            items.append((x, y, torch.full((nout,), -1, dtype=torch.int64, device="cuda")))
            w = torch.empty(nout, dtype=torch.int64, device="cuda")
            D.sqr(x, w) if y is None else D.mul(x, y, w)
            want.append(w)
        D.sync()
    finally:
        set_chunking(True)
    for schedule in ("per_pass", "persistent", None):
        b = D.Batch(items, autotune=autotune, schedule=schedule)
        for _, _, out in items:
            out.fill_(-1)
        b.run()
        D.sync()
        for k, (it, w) in enumerate(zip(items, want)):
            assert torch.equal(it[2], w), (schedule, sizes[k])
        b.close()


@pytest.mark.parametrize("L", [13, 14, 16, 17])
@pytest.mark.parametrize("offset", [0, 1])
def test_half_full_operands(hg, oracle, L, offset):
    """Operands that just fill, or just miss filling, the lower half of a
    transform's points (the first forward pass then skips its upper rows), as
    limbs and as digits, on and off a 16-byte boundary, alone and in batches."""
    import torch

    from hypergeometrica_gb300 import device as D

    items, want = [], []
    for half in (1 << (L - 1), (1 << (L - 1)) * 5 // 4):
        for nx in (half - 1, half, half + 1):
            ny = half // 2 + nx % 7
            x, y = W.limbs(L + nx, nx), W.limbs(2 * L + nx, ny, "ones")
            tx, ty = torch.zeros(nx + offset, dtype=torch.int64, device="cuda"), _dev(y)
            tx[offset:] = _dev(x)
            out = torch.full((nx + ny,), -1, dtype=torch.int64, device="cuda")
            D.mul(tx[offset:], ty, out)
            D.sync()
            w = oracle.mpz_mul_ntt(x, y)[: nx + ny]
            assert np.array_equal(_np(out), w), (L, nx, offset)
            items.append((tx[offset:], ty, out))
            want.append(torch.from_numpy(w.view(np.int64).copy()).cuda())
    for copies in (1, 40 if L < 16 else 4):  # a batch that fills the GPU runs on digits
        many = [(x, y, torch.empty_like(o)) for _ in range(copies) for x, y, o in items]
        for schedule in ("per_pass", "persistent"):
            b = D.Batch(many, autotune=False, schedule=schedule)
            for _, _, o in many:
                o.fill_(-1)
            b.run()
            D.sync()
            for k, (_, _, o) in enumerate(many):
                assert torch.equal(o, want[k % len(want)]), (L, k, copies, schedule)
            b.close()


@pytest.mark.parametrize("ny", [1 << 9, 5000, 1 << 15])
def test_chunk_edges(hg, ny):
    """A long operand in chunks whose last one has a limb, a row less one, a
    row, half a chunk and a whole chunk, on and off a 16-byte boundary (bulk
    copies, or per-thread loads), against one transform."""
    import torch

    from hypergeometrica_gb300 import device as D
    from hypergeometrica_gb300._lib import chunk_plan, set_chunking

    L, C, _ = chunk_plan(64 * ny, ny)
    y = _dev(W.limbs(ny, ny, "ones"))
    for K in (2, 3, 9):
        for rest in (1, 15, 16, 319, 320, 1023, 1024, 1281, C // 2 - 1, C // 2, C // 2 + 1, C - 1, C):
            nx = (K - 1) * C + rest
            x = torch.zeros(nx + 1, dtype=torch.int64, device="cuda")
            x[:nx] = _dev(W.limbs(nx, nx, ("uniform", "ones")[rest % 2]))
            got = torch.full((nx + ny + 3,), -1, dtype=torch.int64, device="cuda")
            off, want = torch.empty_like(got), torch.empty_like(got)
            D.mul(x[:nx], y, got)
            shifted = torch.zeros(nx + 1, dtype=torch.int64, device="cuda")
            shifted[1:] = x[:nx]
            D.mul(y, shifted[1:], off)
            assert set_chunking(False)
            try:
                D.mul(x[:nx], y, want)
                D.sync()
            finally:
                set_chunking(True)
            assert torch.equal(got, want), (ny, K, rest)
            assert torch.equal(off, want), (ny, K, rest)
