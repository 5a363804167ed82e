"""80-bit digits (hg_common.cuh reduce80, hg_internal.h digit80 and coefs_of,
hg_carry.cuh carry80_body), modelled on the CPU with the kernels' own 64-bit
steps: forming digits from limbs, reducing them, and putting three-word
coefficients at 80-bit positions back together into limbs."""

import random

M64 = (1 << 64) - 1
CS = (197, 174, 131)  # default-moduli, src/moduli.lisp:257-264


def reduce80(lo, hi, c):
    p = (c << 55) + 1
    m = ((1 << 39) + c - 1) // c
    assert m < 1 << 32
    t = (hi << 9) | (lo >> 55)
    q = ((t * m) >> 32) >> 7
    assert q == t // c
    r = (lo - q - (((q * (c << 23)) & 0xFFFFFFFF) << 32)) & M64
    return (r + p) & M64 if r >> 63 else r


def test_reduce80():
    rng = random.Random(1)
    for c in CS:
        p = (c << 55) + 1
        vals = [0, 1, p - 1, p, p + 1, (1 << 80) - 1, (1 << 64) - 1, 1 << 64]
        vals += [k * p + d for k in (1, 2, 1000, (1 << 80) // p) for d in (-1, 0, 1)]
        vals += [(k * c << 55) + d for k in (1, 7, (1 << 25) // c) for d in (-1, 0, 1)]
        vals += [rng.randrange(1 << 80) for _ in range(20000)]
        for v in vals:
            v &= (1 << 80) - 1
            assert reduce80(v & M64, v >> 64, c) == v % p


def digits(limbs):
    n = len(limbs) - len(limbs) // 5  # coefs_of
    out = []
    for j in range(n):
        w, s = (5 * j) >> 2, (j & 3) << 4
        a = limbs[w]
        b = limbs[w + 1] if w + 1 < len(limbs) else 0
        lo = ((a >> s) | ((b << 1) << (63 - s))) & M64
        out.append(lo | (((b >> s) & 0xFFFF) << 64))
    return out


def test_digits_of_limbs():
    rng = random.Random(2)
    for n in list(range(1, 30)) + [100, 1001]:
        x = [rng.choice((0, M64, rng.getrandbits(64))) for _ in range(n)]
        v = sum(l << (64 * i) for i, l in enumerate(x))
        d = digits(x)
        assert all(0 <= y < 1 << 80 for y in d) and sum(y << (80 * j) for j, y in enumerate(d)) == v
        assert len(d) == -(-64 * n // 80)


def put_together(coefs):
    """carry80_body over one tile: pieces, sums, carries, five limbs of four digits."""
    al, ah, gen, prop, hp = [], [], [], [], 0
    pieces = [(c & ((1 << 80) - 1), (c >> 80) & ((1 << 80) - 1), c >> 160) for c in coefs]
    for i, (a, _, _) in enumerate(pieces):
        b = pieces[i - 1][1] if i >= 1 else 0
        c = pieces[i - 2][2] if i >= 2 else 0
        lo = (a & M64) + (b & M64)
        hi = (a >> 64) + (b >> 64) + (lo >> 64)
        lo = (lo & M64) + c
        hi += lo >> 64
        lo &= M64
        assert hi < 1 << 18
        z = (lo + hp) & M64
        carry = 1 if z < lo else 0
        hp = hi >> 16
        h = (hi & 0xFFFF) + carry
        al.append(z)
        ah.append(h & 0xFFFF)
        gen.append(h >> 16)
        prop.append(z == M64 and h == 0xFFFF)
        assert gen[-1] <= 1 and not (gen[-1] and prop[-1])
    cin = 0
    for k in range(len(al)):
        z = (al[k] + cin) & M64
        ah[k] = (ah[k] + (1 if z < al[k] else 0)) & 0xFFFF
        al[k] = z
        cin = gen[k] | (prop[k] & cin)
    out = []
    for q in range(0, len(al), 4):
        a, h = al[q: q + 4], ah[q: q + 4]
        out += [a[0], h[0] | (a[1] << 16) & M64, (a[1] >> 48) | (h[1] << 16) | (a[2] << 32) & M64,
                (a[2] >> 32) | (h[2] << 32) | (a[3] << 48) & M64, (a[3] >> 16) | (h[3] << 48)]
    return out, cin


def test_coefficients_to_limbs():
    rng = random.Random(3)
    top = (1 << 187) + (1 << 183)  # p0 p1 p2 = 2^187.1
    for n in (4, 8, 40):
        for kind in range(6):
            hi = min(top, (1 << (80 * 2)) * 3)
            c = [[rng.randrange(hi), (1 << 80) - 1, 0, (1 << 160) - 1, hi - 1, rng.choice((0, (1 << 80) - 1))][kind] for _ in range(n)]
            c[-2:] = [0, 0]  # a product ends within its positions
            v = sum(x << (80 * i) for i, x in enumerate(c))
            out, carry = put_together(c)
            got = sum(x << (64 * i) for i, x in enumerate(out)) + (carry << (80 * n))
            assert got == v & ((1 << (80 * n)) - 1) | (carry << (80 * n))
