"""Division on one thread's registers with digits from the top three limbs
(divmod_reg_kernel): every divisor class at full length with its quotient's
first group at each of its four places, digits of all ones, digits one too
large before the add-back, divisors of leading and trailing ones, in-place
quotients; and the three-by-two estimate itself replayed with Python integers."""
import random

import pytest

M32 = (1 << 32) - 1


def _reciprocal_2by1(d):
    return ((1 << 64) - 1) // d - (1 << 32)


def _reciprocal_3by2(d1, d0):
    v = _reciprocal_2by1(d1)
    p = (d1 * v + d0) & M32
    if p < d0:
        v -= 1
        if p >= d1:
            v -= 1
            p -= d1
        p = (p - d1) & M32
    t = v * d0
    p = (p + (t >> 32)) & M32
    if p < t >> 32:
        v -= 1
        if p << 32 | t & M32 >= (d1 << 32 | d0):
            v -= 1
    return v & M32


def _div_3by2(w2, w1, w0, d1, d0, v):
    m64, D, u = (1 << 64) - 1, d1 << 32 | d0, w2 << 32 | w1
    q = v * w2 + u & m64
    q1 = q >> 32
    r = ((w1 - q1 * d1 & M32) << 32 | w0) - d0 * q1 - D & m64
    q1 = q1 + 1 & M32
    if r >> 32 >= q & M32:
        q1 = q1 - 1 & M32
        r = r + D & m64
    if r >= D:
        q1 = q1 + 1 & M32
    return M32 if u >= D else q1


def test_three_by_two_estimate():
    r = random.Random(32)
    edge = [0, 1, 2, M32, M32 - 1, 1 << 31, (1 << 31) - 1, (1 << 31) + 1, 0xffff0000, 0x0000ffff]
    for _ in range(20000):
        pick = lambda: r.choice(edge) if r.random() < 0.6 else r.getrandbits(32)
        d1, d0 = pick() | 1 << 31, pick()
        D = d1 << 32 | d0
        v = _reciprocal_3by2(d1, d0)
        assert v == ((1 << 96) - 1) // D - (1 << 32)
        u = min(pick() << 32 | pick(), D)
        w0 = pick()
        want = M32 if u == D else (u << 32 | w0) // D
        assert _div_3by2(u >> 32, u & M32, w0, d1, d0, v) == want


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 7, 8, 12, 15, 16])
@pytest.mark.parametrize("more", [0, 1, 2, 3, 4, 5, 16, 19])
def test_divide_full_length_divisors(handle, nb, more):
    import xmp_b200 as xmp
    from tests.helpers import ints_from_rows, rows_from_ints
    r = random.Random(100 * nb + more)
    na, count = nb + more, 333
    top = (1 << (32 * nb)) - 1
    a, b = [], []
    for i in range(count):
        d = [top, 1 << (32 * nb - 1), top ^ M32, (1 << (32 * nb - 1)) + 1, top >> 31,
             r.getrandbits(32 * nb) | 1 << (32 * nb - 1 - i % 32), r.getrandbits(32 * nb) >> r.choice([0, 1, 33])][i % 7]
        d = d or 1
        q = [(1 << (32 * (more + 1))) - 1, r.getrandbits(32 * more + 32), 1 << 32 * more, M32][i % 4]
        n = d * q + [0, -1, d - 1, r.randrange(d)][i % 5 % 4]
        a.append(max(n, 0) if n < 1 << (32 * na) else (1 << (32 * na)) - 1 - r.choice([0, 1, d & M32]))
        b.append(d)
    A = handle.integers(32 * na, count, rows_from_ints(a, na))
    B = handle.integers(32 * nb, count, rows_from_ints(b, nb))
    Q, R = handle.integers(32 * na, count), handle.integers(32 * nb, count)
    xmp.divmod_(handle, Q, R, A, B, count)
    assert ints_from_rows(Q.export()) == [x // y for x, y in zip(a, b)]
    assert ints_from_rows(R.export()) == [x % y for x, y in zip(a, b)]
    xmp.div(handle, A, A, B, count)  # onto the dividend
    assert ints_from_rows(A.export()) == [x // y for x, y in zip(a, b)]
    for v in (A, B, Q, R):
        v.destroy()
