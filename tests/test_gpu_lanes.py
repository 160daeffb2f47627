"""Multiply and divide with operands over several lanes (mul_lanes_kernel,
divmod_lanes_kernel) at the sizes where they can go wrong, exact against
Python's integers: limb counts at and beside the lane shapes' edges, operands
of very different lengths, ragged and tiny batches, divisors with leading zero
limbs and bits beside full ones in one warp, division by zero, dividends
shorter than the divisor, quotient digits at both ends, in-place outputs and
index arrays."""
import random

import numpy as np
import pytest

import xmp_b200 as xmp
from tests.helpers import ints_from_rows, rows_from_ints

pytestmark = pytest.mark.gpu


def _values(r, limbs, count):
    top = (1 << (32 * limbs)) - 1
    edge = [0, 1, top, top - 1, 1 << (32 * limbs - 1), top ^ 0xffffffff, 0xffffffff]
    return [edge[i % 7] if i % 3 == 0 else r.getrandbits(32 * limbs) >> r.choice([0, 0, 1, 33, 32 * limbs // 2])
            for i in range(count)]


def _arr(h, limbs, vals):
    return h.integers(32 * limbs, len(vals), rows_from_ints(vals, limbs))


@pytest.mark.parametrize("na,nb", [(33, 1), (33, 33), (48, 48), (49, 17), (64, 64), (65, 64), (96, 95), (97, 12),
                                   (128, 128), (129, 3), (256, 256), (257, 130), (512, 512), (513, 2), (5, 64)])
@pytest.mark.parametrize("count", [1, 37, 5000])
def test_mul_lanes(handle, na, nb, count):
    if count == 5000 and max(na, nb) > 130:
        count = 900
    r = random.Random(na * 1000 + nb)
    a, b = _values(r, na, count), _values(r, nb, count)
    A, B = _arr(handle, na, a), _arr(handle, nb, b)
    for np_ in (na + nb, max(na, nb), na + nb + 7):  # exact, truncated, wider than the product
        P = handle.integers(32 * np_, count)
        xmp.mul(handle, P, A, B, count)
        assert ints_from_rows(P.export()) == [(x * y) % (1 << (32 * np_)) for x, y in zip(a, b)]
        P.destroy()
    for v in (A, B):
        v.destroy()


def test_mul_lanes_in_place_and_indexed(handle):
    r = random.Random(5)
    count, n = 200, 64
    a, b = _values(r, n, count), _values(r, n, count)
    mask = (1 << (32 * n)) - 1
    for first in (True, False):
        A, B = _arr(handle, n, a), _arr(handle, n, b)
        xmp.mul(handle, A if first else B, A, B, count)
        assert ints_from_rows((A if first else B).export()) == [x * y & mask for x, y in zip(a, b)]
        xmp.mul(handle, A, A, A, count)  # a square onto itself
        A.destroy()
        B.destroy()
    A, B, P = _arr(handle, n, a), _arr(handle, n, b[:7]), handle.integers(64 * n, count)
    ia, ip = np.random.default_rng(1).permutation(count), np.random.default_rng(2).permutation(count)
    pol = handle.policy()
    pol.set_indices(0, ip)
    pol.set_indices(1, ia)
    handle.set_policy(pol)
    try:
        xmp.mul(handle, P, A, B, count)
    finally:
        handle.set_policy(None)
        pol.destroy()
    got = ints_from_rows(P.export())
    assert all(got[ip[i]] == a[ia[i]] * b[i % 7] for i in range(count))
    for v in (A, B, P):
        v.destroy()


@pytest.mark.parametrize("na,nb", [(34, 17), (64, 32), (66, 33), (48, 48), (100, 49), (128, 64), (130, 65), (64, 96),
                                   (194, 97), (256, 128), (258, 129), (512, 256), (514, 257), (700, 512), (40, 512),
                                   (1, 33), (514, 513)])
@pytest.mark.parametrize("count", [1, 37, 3000])
def test_divmod_lanes(handle, na, nb, count):
    if count == 3000 and max(na, nb) > 130:
        count = 500
    r = random.Random(na * 1000 + nb)
    a, b = _values(r, na, count), _values(r, nb, count)
    for i in range(0, count, 5):  # dividends beside multiples of the divisor: digits of all ones, remainders 0, b - 1
        if b[i]:
            k = r.choice([(1 << 32) - 1, 1, r.getrandbits(32 * max(1, na - nb))])
            a[i] = max(0, b[i] * k + r.choice([0, -1, b[i] - 1])) % (1 << (32 * na))
    A, B, Q, R = _arr(handle, na, a), _arr(handle, nb, b), handle.integers(32 * na, count), \
        handle.integers(32 * (nb + 3), count)
    want_q = [x // y if y else x for x, y in zip(a, b)]
    want_r = [x % y if y else 0 for x, y in zip(a, b)]
    xmp.divmod_(handle, Q, R, A, B, count)
    assert ints_from_rows(Q.export()) == want_q and ints_from_rows(R.export()) == want_r
    xmp.div(handle, Q, A, B, count)
    assert ints_from_rows(Q.export()) == want_q
    xmp.mod(handle, B, A, B, count)  # in place
    assert ints_from_rows(B.export()) == want_r
    for v in (A, B, Q, R):
        v.destroy()
