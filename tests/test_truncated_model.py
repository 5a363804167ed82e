"""The truncated transform's inverse (hg_ntt_rounds.cuh, TruncatedInverse),
modelled on the CPU.

A truncated transform keeps the first K of the n outputs that the top stages
of a pass give each column; the column's values past K are zero.  The model
runs the kernel's recursion with its own 64-bit steps (residues in [0, 2p),
folds by the sign of x - p, Shoup products) and checks that it returns n times
the column, for every K the kernels take, and that every value stays in
[0, 2p) below 2^64.
"""

import random

import pytest

MASK = (1 << 64) - 1
PS = tuple(c * (1 << 55) + 1 for c in (197, 174, 131))  # default-moduli, src/moduli.lisp:257-264


def fold(x, p):
    assert 0 <= x < 2 * p <= MASK
    d = (x - p) & MASK
    return x if d >> 63 else d


def shoup(a, w, p):
    assert 0 <= a <= MASK
    q = (a * ((w << 64) // p)) >> 64
    r = a * w - q * p
    assert 0 <= r < 2 * p
    return fold(r, p)


def root(p, n):
    """A primitive n-th root of unity (n a power of two)."""
    for g in range(2, 100):
        w = pow(g, (p - 1) // n, p)
        if pow(w, n // 2, p) == p - 1:
            return w
    raise AssertionError


class Column:
    """n = 2^j values at row stride m of an R = n m point column transform, in column position low < m."""

    def __init__(self, p, n, m, low):
        self.p, self.low, self.m = p, low, m
        self.w = {}
        k = n
        while k >= 2:
            self.w[k] = root(p, n * m) if k == n else pow(self.w[2 * k], 2, p)  # w of order k m
            k //= 2

    def tw(self, n, h, sign):
        return pow(self.w[n], sign * (h * self.m + self.low), self.p)

    def forward(self, x):
        """The top stages (DIF), in place order: the upper half times w^h."""
        n, p = len(x), self.p
        if n == 1:
            return list(x)
        h = n // 2
        u = [(x[i] + x[i + h]) % p for i in range(h)]
        v = [(x[i] - x[i + h]) * self.tw(n, i, 1) % p for i in range(h)]
        return self.forward(u) + self.forward(v)

    def butterfly(self, v, i, h, n):
        p = self.p
        u, t = fold(v[i], p), shoup(v[i + h], self.tw(n, i % n, -1), p)
        v[i], v[i + h] = u + t, u - t + p

    def twice_less(self, a, b):
        p = self.p
        return fold(2 * fold(a, p), p) - fold(b, p) + p

    def run(self, v, off, n, K, zt):
        """TruncatedInverse::run on v[off, off + n)."""
        p, half = self.p, n // 2
        if n == 1:
            return
        tw = lambda i, s: self.tw(n, i, s)  # noqa: E731
        if K == n:
            self.run(v, off, half, half, False)
            self.run(v, off + half, half, half, False)
            for q in range(half):
                u, t = fold(v[off + q], p), shoup(v[off + q + half], tw(q, -1), p)
                v[off + q], v[off + q + half] = u + t, u - t + p
        elif K > half:
            K1 = K - half
            self.run(v, off, half, half, False)
            for q in range(K1, half):
                u, x = v[off + q], v[off + q + half]
                d = u if zt else fold(u, p) - fold(x, p) + p
                v[off + q + half] = shoup(d, tw(q, 1), p)
                v[off + q] = 2 * fold(u, p) if zt else self.twice_less(u, x)
            self.run(v, off + half, half, K1, False)
            for q in range(K1):
                u, t = fold(v[off + q], p), shoup(v[off + q + half], tw(q, -1), p)
                v[off + q], v[off + q + half] = u + t, u - t + p
        else:
            assert not zt
            for q in range(K, half):
                s = fold(fold(v[off + q], p) + fold(v[off + q + half], p), p)
                v[off + q] = (s + (p if s & 1 else 0)) >> 1
            self.run(v, off, half, K, False)
            for q in range(K):
                v[off + q] = self.twice_less(v[off + q], v[off + q + half])
        assert all(0 <= x < 2 * p for x in v[off: off + K])


@pytest.mark.parametrize("p", PS)
@pytest.mark.parametrize("n,K", [(16, k) for k in range(9, 17)] + [(8, 5), (8, 6), (8, 7), (8, 8), (4, 3), (4, 4)])
def test_truncated_inverse_returns_the_column(p, n, K):
    rng = random.Random(n * 100 + K)
    for low, m in ((0, 2), (1, 2), (5, 16), (15, 16)):
        col = Column(p, n, m, low)
        for edge in (0, 1, p - 1, None):
            x = [rng.randrange(p) if edge is None else edge for _ in range(K)] + [0] * (n - K)
            f = col.forward(x)[:K]
            # [0, 2p) representatives of the known outputs; what sits past them is never read
            v = [y + (p if rng.random() < 0.5 else 0) for y in f] + [0xDEAD] * (n - K)
            col.run(v, 0, n, K, K < n)
            assert [y % p for y in v[:K]] == [n * y % p for y in x[:K]]
