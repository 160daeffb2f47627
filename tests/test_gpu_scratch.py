"""Scratch and admission limits: what a limit lets through does not depend on
which kernel the library prefers for the batch, and the plain calls leave the
scratch arena at the size that their asynchronous forms need."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp
from tests.helpers import ints_from_rows, rows_from_ints
from tests.test_gpu_alloc import Allocator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,count", [(256, 100), (2048, 14), (2048, 256)])
def test_plain_calls_size_the_arena(bits, count):
    """After a synchronous import and export of pageable rows the asynchronous ones allocate nothing, so they can
    be captured."""
    torch.cuda.init()
    A = Allocator()
    h = xmp.Handle.__new__(xmp.Handle)
    h.h = A.handle()
    rows = np.random.default_rng(bits).integers(0, 1 << 32, (count, bits // 32), dtype=np.uint32)
    x = h.integers(bits, count)
    x.import_(rows)
    calls = A.calls
    x.import_(rows, asynchronous=True)
    assert A.calls == calls
    out = np.zeros_like(rows)
    x.export(out=out, asynchronous=True)
    assert A.calls == calls
    torch.cuda.synchronize()
    assert np.array_equal(out, rows)
    x.destroy()
    h.destroy()


def _crt(h, half, count, seed):
    """Operands and the expected results of `count` operations with short exponents."""
    r = np.random.default_rng(seed)
    draw = lambda bits, n: [int.from_bytes(r.bytes(bits // 8), "little") for _ in range(n)]
    p, q = ([v | 1 | 1 << (half - 1) for v in draw(half, count)] for _ in range(2))
    q = [v if v != u else v - 2 for u, v in zip(p, q)]
    dp, dq = draw(64, count), draw(64, count)
    qinv = [v % u for u, v in zip(p, draw(half, count))]
    c = [v % (u * w) for u, w, v in zip(p, q, draw(2 * half, count))]
    want = []
    for i in range(count):
        mp, mq = pow(c[i], dp[i], p[i]), pow(c[i], dq[i], q[i])
        want.append(mq + q[i] * ((mp - mq) * qinv[i] % p[i]))
    n = half // 32
    args = [h.integers(32 * w, count, rows_from_ints(v, w))
            for v, w in ((c, 2 * n), (p, n), (q, n), (dp, 2), (dq, 2), (qinv, n))]
    return args, want


# The limit: 128 threads' window-1 tables in limbs, four lanes an exponentiation.
@pytest.mark.parametrize("bits,count,limit", [(1024, 4096, 4096), (1536, 6144, 6144), (2048, 8192, 8192)])
@pytest.mark.parametrize("plan", [False, True])
def test_crt_within_a_small_limit(bits, count, limit, plan):
    h = xmp.Handle()
    args, want = _crt(h, bits // 2, count, bits)
    out = h.integers(bits, count)
    pol = h.policy()
    pol.set_scratch_limit(limit * 2 if plan else limit)
    h.set_policy(pol)
    if plan:
        b = xmp.BatchPlan(h, crt=[(out, *args, count)], use_graph=False)
        b.execute()
        torch.cuda.synchronize()
        b.destroy()
    else:
        xmp.powm_crt(h, out, *args, count)
    h.set_policy(None)
    assert ints_from_rows(out.export()) == want
    for v in args + [out]:
        v.destroy()
    pol.destroy()
    h.destroy()


# The limit: 128 threads' window-1 tables in limbs on the lanes of the kernel that was faster on them.
@pytest.mark.parametrize("bits,count,limit", [(256, 128, 2048), (512, 6144, 4096), (1024, 32768, 8192),
                                              (1536, 6144, 6144), (2048, 1536, 4096), (3072, 3072, 6144)])
def test_powm_within_a_small_limit(bits, count, limit):
    h = xmp.Handle()
    r = np.random.default_rng(bits)
    n = bits // 32
    x, m = (r.integers(0, 1 << 32, (count, n), dtype=np.uint32) for _ in range(2))
    e = r.integers(0, 1 << 32, (count, 1), dtype=np.uint32)
    m[:, 0] |= 1
    X, E, M, O = h.integers(bits, count, x), h.integers(32, count, e), h.integers(bits, count, m), h.integers(bits, count)
    pol = h.policy()
    pol.set_scratch_limit(limit)
    h.set_policy(pol)
    xmp.powm(h, O, X, E, M, count)
    h.set_policy(None)
    want = [pow(a, b, c) for a, b, c in zip(*(ints_from_rows(v) for v in (x, e, m)))]
    assert ints_from_rows(O.export()) == want
    for v in (X, E, M, O):
        v.destroy()
    pol.destroy()
    h.destroy()
