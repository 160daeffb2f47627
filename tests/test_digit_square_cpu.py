"""The one-lane Montgomery square on 52-bit digits (dig_sqr1,
xmp_b200/csrc/dmont.cuh) replayed on 64-bit words: columns that start from
minus the constant of the halves they will take, cross products once and
doubled, the reduction's rows whose constant only the high words carry, and
the columns' settling; at operands and moduli on the digits' edges."""
import random

import pytest

M64, M52 = (1 << 64) - 1, (1 << 52) - 1
LO, HI = 0x433 << 52, (0x467 << 52) + (1 << 51)  # what a low / a high half's bits add to a column


def _halves(x, y):
    """Bits of the two doubles that hold x y = high 2^52 + low, -2^51 <= ... <= 2^52."""
    p = x * y
    high = p >> 52  # round towards zero of 1.5 2^104 + p, a positive number
    return (LO + p - (high << 52)) & M64, (HI + high) & M64


def _pairs(c, D):
    lo, end = max(c - D + 1, 0), (c + 1) // 2
    return 0 if c < 0 or end < lo else end - lo


def _balanced(v, D):
    out = []
    for p in range(D):
        d = v & M52
        d -= (d >> 51) << 52
        out.append(d)
        v = (v - d) >> 52
    out[-1] += v << 52
    return out


def _signed(v):
    return v - (1 << 64) if v >> 63 else v


def _square(a, n, np):
    D = len(a)
    s = [-(_pairs(c, D) * LO + _pairs(c - 1, D) * HI + (HI if c % 2 else LO) // 2) & M64 for c in range(2 * D)]
    for i in range(D):
        for j in range(i + 1, D):
            low, high = _halves(a[i], a[j])
            s[i + j] = s[i + j] + low & M64
            s[i + j + 1] = s[i + j + 1] + high & M64
    for j in range(D):
        low, high = _halves(a[j], a[j])
        s[2 * j] = 2 * s[2 * j] + low & M64
        s[2 * j + 1] = 2 * s[2 * j + 1] + high & M64
    assert sum(_signed(v) << (52 * p) for p, v in enumerate(s)) == sum(d << (52 * p) for p, d in enumerate(a)) ** 2
    k, step = 0, (LO + HI) >> 32
    assert (LO + HI) & 0xffffffff == 0
    for _ in range(D):
        x = ((((s[0] >> 32) - k & 0xffffffff) << 32 | s[0] & 0xffffffff) * np) & M52
        q = x - ((x >> 51) << 52)
        for j in range(D):
            low, high = _halves(n[j], q)
            s[j] = s[j] + low & M64
            s[j + 1] = s[j + 1] + high & M64
        c = (s[0] >> 32) - k - (LO >> 32) & 0xffffffff
        c = (c - (1 << 32) if c >> 31 else c) >> 20
        k = k + step & 0xffffffff
        s = s[1:] + [0]
        s[0] = s[0] + c & M64
    const = [(D - 1 - p) * LO + (D - p) * HI for p in range(D)]
    return sum(_signed(s[p] - const[p] & M64) << (52 * p) for p in range(D))


@pytest.mark.parametrize("limbs,D", [(6, 4), (8, 5), (12, 8), (16, 10), (24, 15), (32, 20)])
def test_square(limbs, D):
    r = random.Random(limbs)
    bits, R = 32 * limbs, 1 << (52 * D)
    edge = sum(1 << (52 * p + 51) for p in range(D)) % (1 << bits)
    for n in ((1 << bits) - 1, (1 << (bits - 1)) + 1, edge | 1, 3, r.getrandbits(bits) | 1 | 1 << (bits - 1)):
        np = -pow(n, -1, 1 << 52) % (1 << 52)
        for a in (0, 1, n - 1, -(n - 1), edge % n, r.randrange(n), -r.randrange(n)):
            v = _square(_balanced(a, D), _balanced(n, D), np)
            assert (v * R - a * a) % n == 0 and abs(v) <= n
