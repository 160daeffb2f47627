"""The 52-bit digit Montgomery product (xmp_b200/csrc/dmont.cuh) replayed with
Python integers: every quantity the kernel holds -- the halves of a digit
product with the exponent bits of their doubles, the 64-bit columns, the
quotient digits, the dropped columns' carries, the settled digits -- step by
step over the group's lanes, for the registered (lanes, digits) forms, at
operands and moduli on the digits' edges.  Checks the value, that |result| <= N,
and the bounds that make the arithmetic exact."""
import random

import pytest

MASK52, MASK64 = (1 << 52) - 1, (1 << 64) - 1
LO, HI = 0x433 << 52, (0x467 << 52) + (1 << 51)
LIMIT = (1 << 51) + (1 << 12)


def signed64(v):
    v &= MASK64
    return v - (1 << 64) if v >> 63 else v


def balanced(v, nd):
    """Digits as dig_from_limbs takes them from a non-negative number."""
    out = []
    for p in range(nd):
        d = (v >> (52 * p)) & MASK52
        below = (v >> (52 * p - 1)) & 1 if p else 0
        out.append(d - ((d >> 51) << 52) + below)
    assert sum(d << (52 * p) for p, d in enumerate(out)) == v
    return out


def halves(a, w):
    """Bits of l and h: fma_rz(a, w, 1.5 * 2^104) and the remainder on 2^52."""
    p = a * w
    assert abs(p) < 1 << 103  # 1.5 * 2^104 + p stays in one binade
    hi = p >> 52
    return LO + (p - (hi << 52)), HI + hi


def dig_mul(a, b, n, np, T, D):
    N = T * D
    col = [[0] * (D + 2) for _ in range(T)]

    def row(first, x, w):
        for g in range(T):
            for j in range(D):
                lo, hi = halves(x[g * D + j], w)
                col[g][first + j] = (col[g][first + j] + lo) & MASK64
                col[g][first + j + 1] = (col[g][first + j + 1] + hi) & MASK64

    k = 2 * LO
    row(0, a, b[0])
    for i in range(N):
        q = (col[0][0] * np) & MASK52
        q = q - (1 << 52) if q >> 51 else q  # balanced
        if i + 1 < N:
            row(1, a, b[i + 1])
        row(0, n, q)
        true = signed64(col[0][0] - k)
        assert true & MASK52 == 0 and abs(true) < 1 << 63
        # the kernel's carry: the high word less the constant, arithmetic shift
        c = ((((col[0][0] >> 32) - (k >> 32)) & 0xffffffff) ^ 0x80000000) - 0x80000000 >> 20
        assert c == true >> 52
        k = (k + 2 * (LO + HI)) & MASK64
        drop = [col[g][0] for g in range(T)]
        for g in range(T):
            col[g] = col[g][1:] + [0]
            if g + 1 < T:
                col[g][D - 1] = (col[g][D - 1] + drop[g + 1]) & MASK64
        col[0][0] = (col[0][0] + c) & MASK64
    flat = []
    for g in range(T):
        for j in range(D):
            p = g * D + j
            flat.append(signed64(col[g][j] - 2 * (N - 1 - p) * LO - 2 * (N - p) * HI))
    return settle(flat)


def settle(flat):
    """dig_settle: balanced low 52 bits, the rest once to the next digit."""
    carry = [(v + (1 << 51)) >> 52 for v in flat]
    assert all(-2048 <= c < 2048 for c in carry) and carry[-1] == 0
    return [v - (c << 52) + (carry[i - 1] if i else 0) for i, (v, c) in enumerate(zip(flat, carry))]


def value(d):
    return sum(x << (52 * p) for p, x in enumerate(d))


@pytest.mark.parametrize("T,D,bits", [(1, 5, 256), (1, 10, 512), (1, 20, 1024), (2, 5, 512), (4, 4, 768), (4, 5, 1024),
                                      (8, 8, 3072), (4, 10, 2048), (32, 10, 16384)])
def test_product_schedule(T, D, bits):
    r = random.Random(T * 100 + D)
    N, R = T * D, 1 << (52 * T * D)
    assert 52 * N >= bits + 2
    half = sum(1 << (52 * p + 51) for p in range(N)) % (1 << bits)  # every digit on the balance edge
    mods = [(1 << bits) - 1, (1 << (bits - 1)) + 1, half | 1, 3, r.getrandbits(bits) | 1 | 1 << (bits - 1)]
    for m in (mods if bits <= 3072 else mods[:1]):
        np = -pow(m, -1, 1 << 64) & MASK64
        n = balanced(m, N)
        for x, y in ((m - 1, m - 1), ((1 << bits) - 1, m - 1), (half % m, r.randrange(m)), (0, 1)):
            v = dig_mul(balanced(x, N), balanced(y, N), n, np, T, D)
            assert (value(v) * R - x * y) % m == 0 and abs(value(v)) <= m
            assert all(abs(d) <= LIMIT for d in v)
            w = dig_mul(v, v, n, np, T, D)  # a settled, signed result as both operands
            assert (value(w) * R - value(v) ** 2) % m == 0 and abs(value(w)) <= m
            assert all(abs(d) <= LIMIT for d in w)
