"""The 52-bit digit kernels (xmp_b200/csrc/dmont.cuh) at the sizes and values
where they can go wrong, against Python's integers (exact): every registered
shape from six limbs a lane, operands and moduli whose digits lie on the
balance edge, ragged batches, scratch limits that leave room for one warp's
smallest table, the allocation-free entry point beyond one launch, and the
fused CRT operation on each of its digit shapes."""
import math
import random

import numpy as np
import pytest

import oracle
import xmp_b200 as xmp
from tests.helpers import ints_from_rows, rows_from_ints
from tests.test_zz_no_alloc import _deinterleave, _interleave

pytestmark = pytest.mark.gpu

SHAPES = [(t, l) for t in (1, 2, 4, 8, 16, 32) for l in (6, 8, 10, 12, 16, 24, 32)]


def _edge_values(bits, seed):
    r = random.Random(seed)
    half = sum(1 << (52 * p + 51) for p in range(bits // 52 + 1)) % (1 << bits)
    mods = [(1 << bits) - 1, (1 << (bits - 1)) + 1, half | 1, 3, 1, (1 << 52) + 1]
    mods += [r.getrandbits(bits) | 1 | 1 << (bits - 1) for _ in range(5)] + [r.getrandbits(bits // 2) | 1]
    bases = [(1 << bits) - 1, half, 0, 1, (1 << bits) - 2, half - 1] + [r.getrandbits(bits) for _ in range(6)]
    exps = [0, 1, 2, (1 << 64) - 1, 65537, 1 << 63] + [r.getrandbits(64) for _ in range(7)]
    # 13 exponents against 12 moduli and 12 bases shifted by one each round: every pairing of edges comes up
    count = 12 * 13
    return ([mods[i % 12] for i in range(count)], [bases[(i + i // 12) % 12] for i in range(count)],
            [exps[i % 13] for i in range(count)])


@pytest.mark.parametrize("tpi,limbs", SHAPES)
def test_powm_digit_shapes(handle, tpi, limbs):
    if (tpi, limbs) not in xmp.powm_kernels():
        pytest.skip("not a registered shape")
    for bits in {32 * tpi * limbs, 32 * (tpi * limbs - 1)}:  # the shape's capacity, and a limb less
        m, x, e = _edge_values(bits, bits)
        count = len(m) if bits <= 4096 else 13
        n = bits // 32
        X, M, E = (handle.integers(b, count, rows_from_ints(v[:count], b // 32))
                   for b, v in ((bits, x), (bits, m), (64, e)))
        O = handle.integers(bits, count)
        for window in (1, 3, 7):
            xmp.powm_with_config(handle, O, X, E, M, count, xmp.PowmConfig(0, tpi, limbs, window))
            got = ints_from_rows(O.export())
            assert got == [pow(a, b, c) for a, b, c in zip(x[:count], e, m)], (bits, window)
        for v in (X, M, E, O):
            v.destroy()


@pytest.mark.parametrize("bits", [256, 2048, 12288, 16384])
def test_smallest_scratch_limit(handle, bits):
    """The limit that held one 128-thread CTA of two-entry tables in limbs (1,024 bytes a limb of a lane)."""
    tpi, limbs = {256: (1, 8), 2048: (4, 16), 12288: (32, 12), 16384: (32, 16)}[bits]
    count = 40 if bits <= 2048 else 5
    m, x, e = (v[:count] for v in _edge_values(bits, 7))
    X, M, E = (handle.integers(b, count, rows_from_ints(v, b // 32)) for b, v in ((bits, x), (bits, m), (64, e)))
    O = handle.integers(bits, count)
    pol = handle.policy()
    pol.set_scratch_limit(1024 * limbs)
    handle.set_policy(pol)
    try:
        xmp.powm_with_config(handle, O, X, E, M, count, xmp.PowmConfig(0, tpi, limbs, 4))
    finally:
        handle.set_policy(None)
        pol.destroy()
    assert ints_from_rows(O.export()) == [pow(a, b, c) for a, b, c in zip(x, e, m)]
    for v in (X, M, E, O):
        v.destroy()


def test_no_alloc_beyond_one_launch():
    """A batch whose smallest digit tables exceed the fixed array and whose limb tables would not."""
    import torch

    bits, count = 2048, 30000
    n = bits // 32
    m = oracle.full_length_odd(91, count, n)
    x = oracle.below(92, m)
    e = oracle.random_limbs(93, count, 1)
    e[:, 0] &= 0xffff
    dx, dm, de = (torch.from_numpy(_interleave(v, count).view(np.int32)).cuda() for v in (x, m, e))
    out = torch.zeros_like(dx)
    rc = xmp.lib().xmpIntegersPowmNoAlloc(torch.cuda.current_stream().cuda_stream, out.data_ptr(), dx.data_ptr(),
                                          de.data_ptr(), dm.data_ptr(), bits, 32, count, count)
    assert rc == 0
    torch.cuda.synchronize()
    got = _deinterleave(out.cpu().numpy().view(np.uint32), count, n, count)
    for i in list(range(0, count, 997)) + [26213, 26214, 26215, count - 1]:
        assert oracle.to_int(got[i]) == pow(oracle.to_int(x[i]), int(e[i, 0]), oracle.to_int(m[i])), i


@pytest.mark.parametrize("half_bits,count", [(768, 3), (768, 9000), (1024, 3), (1024, 9000), (1536, 5), (1536, 4000),
                                             (2048, 5), (2048, 3000), (3072, 3), (3072, 700), (4096, 2)])
def test_crt_digit_shapes(handle, half_bits, count):
    """Any odd p, q coprime with any c, dp, dq: the counts reach both kernel shapes of each size."""
    r = random.Random(half_bits + count)
    top = 1 << (half_bits - 1)
    half = sum(1 << (52 * p + 51) for p in range(half_bits // 52 + 1)) % (1 << half_bits)
    keys = []
    for p, q in (((1 << half_bits) - 1, top + 1), (half | 1 | top, (1 << half_bits) - 3), (7, 11),
                 (r.getrandbits(half_bits) | 1 | top, r.getrandbits(half_bits - 40) | 1)):
        while math.gcd(p, q) != 1:
            q -= 2
        keys.append((p, q, r.getrandbits(64), r.getrandbits(64), pow(q, -1, p)))
    c = [r.getrandbits(2 * half_bits) for _ in range(min(count, 12))]
    c = [c[i % len(c)] for i in range(count)]
    C = handle.integers(2 * half_bits, count, rows_from_ints(c, half_bits // 16))
    bits = (half_bits, half_bits, 64, 64, half_bits)
    K = [handle.integers(b, len(keys), rows_from_ints([k[j] for k in keys], b // 32)) for j, b in enumerate(bits)]
    O = handle.integers(2 * half_bits, count)
    xmp.powm_crt(handle, O, C, *K, count)
    got = ints_from_rows(O.export())
    want = {}
    for i in range(count):
        if (i % len(keys), c[i]) not in want:
            p, q, dp, dq, qinv = keys[i % len(keys)]
            mp, mq = pow(c[i], dp, p), pow(c[i], dq, q)
            want[(i % len(keys), c[i])] = mq + q * ((mp - mq) * qinv % p)
        assert got[i] == want[(i % len(keys), c[i])], i
    for v in [C, O] + K:
        v.destroy()
