"""The CTA distribution's Montgomery product on 52-bit digits
(xmp_b200/csrc/cta.cuh) replayed with Python integers: the lanes of a column
pair with their terms, the chunks that a warp skips, operands stored twice, one
carry step, m without its top carry, the low half's multiple of R read off two
columns, T's upper columns left in the lanes; and Newton's iteration for
-N^-1 mod R.  Checks the value, |result| <= N and the bounds on digits and
columns, at operands and moduli on the digits' edges."""
import random

import pytest

SHAPES = {32: (20, 4), 64: (40, 8), 96: (60, 8), 128: (80, 8)}  # limbs -> digits, lanes per column pair
PAD = 8
M52 = (1 << 52) - 1


def balanced(v, nd):
    out = []
    for p in range(nd):
        d = (v >> (52 * p)) & M52
        below = (v >> (52 * p - 1)) & 1 if p else 0
        out.append(d - ((d >> 51) << 52) + below)
    assert sum(d << (52 * p) for p, d in enumerate(out)) == v
    return out


def value(d):
    return sum(x << (52 * p) for p, x in enumerate(d))


def twice(y):
    return list(y) + list(y)


def accumulate(low, high, x, y, P, mode):
    """Adds the terms of x y that the mode takes to the sums of columns c (low) and N + c (high): per column its
    low halves and its products' high halves."""
    N = len(x)
    K = -(-N // P)
    chunk = K if K <= 5 else (K + 1) // 2
    x = list(x) + [None] * PAD
    y = twice(y)
    threads = -(-N * P // 32) * 32
    for tid in range(threads):
        c, p = divmod(tid, P)
        cmin = tid // 32 * 32 // P
        cmax = cmin + 32 // P - 1
        for k0 in range(0, K, chunk):
            if chunk < K:
                if mode == "low" and P * k0 > cmax:
                    break
                if mode == "high" and P * (k0 + chunk) <= cmin + 1 and cmax < N - 3:
                    continue
            for k in range(k0, min(k0 + chunk, K)):
                i, j = p + P * k, N + c - p - P * k
                assert 0 <= i < N + PAD and -PAD <= j < 2 * N + PAD
                if c >= N:
                    continue  # a lane beyond the columns: its sums are not stored
                if i <= c:
                    to = low[c]
                elif mode != "low" and i < N:
                    to = high[c]
                else:
                    continue
                v = x[i] * y[j]
                assert abs(v) < 1 << 103
                to[0] += v & M52
                to[1] += v >> 52


def sums(N):
    return [[0, 0] for _ in range(N)]


def columns(low, high):
    """Column j: its low halves and the high halves of column j - 1."""
    s = low + high
    out = [s[j][0] + (s[j - 1][1] if j else 0) for j in range(len(s))]
    assert all(abs(v) < 1 << 62 for v in out)
    return out


def carry(v):
    c = (v + (1 << 51)) >> 52
    assert -2048 <= c < 2048
    return c


def digits(cols, first):
    """One carry step; `first`: what enters the first column."""
    out, below = [], first
    for v in cols:
        out.append(v - (carry(v) << 52) + below)
        below = carry(v)
    assert all(abs(d) <= (1 << 51) + (1 << 12) for d in out)
    return out


def low(x, y, P, add=0):
    N = len(x)
    lo, hi = sums(N), sums(N)
    accumulate(lo, hi, x, y, P, "low")
    c = columns(lo, hi)[:N]
    c[0] += add
    return digits(c, 0)


def mont(a, b, n, np, P):
    N = len(a)
    lo, hi = sums(N), sums(N)
    accumulate(lo, hi, a, b, P, "full")
    t = digits(columns(lo, hi)[:N], 0)
    m = low(t, np, P)
    accumulate(lo, hi, m, n, P, "high")
    u = columns(lo, hi)
    top = u[N - 1] + (u[N - 2] >> 52)
    return digits(u[N:], carry(top))


@pytest.mark.parametrize("limbs", [32, 64, 96, 128])
def test_product(limbs):
    N, P = SHAPES[limbs]
    bits, R = 32 * limbs, 1 << (52 * N)
    r = random.Random(limbs)
    half = sum(1 << (52 * p + 51) for p in range(N)) % (1 << bits)
    for n in ((1 << bits) - 1, (1 << (bits - 1)) + 1, half | 1, 3, r.getrandbits(bits) | 1 | 1 << (bits - 1)):
        nd = balanced(n, N)
        y = [0] * N
        y0 = -pow(n, -1, 1 << 52) % (1 << 52)
        y[0] = y0 - (1 << 52) if y0 >> 51 else y0
        k = 1
        while k < N:
            y = low(low(nd, y, P, 2), y, P)
            k *= 2
        assert (value(y) * n + 1) % R == 0
        for a, b in ((n - 1, n - 1), ((1 << bits) - 1, n - 1), (half % n, r.randrange(n)), (0, 1), (1, 1)):
            v = mont(balanced(a, N), balanced(b, N), nd, y, P)
            assert (value(v) * R - a * b) % n == 0 and abs(value(v)) <= n
            w = mont(v, v, nd, y, P)  # a signed, lazily carried result as both operands
            assert (value(w) * R - value(v) ** 2) % n == 0 and abs(value(w)) <= n
