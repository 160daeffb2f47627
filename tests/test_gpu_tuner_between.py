"""The default kernel at counts about powers of two: one that the selector's
table holds there or in the next cells, with exact results where they differ."""
import ctypes

import numpy as np
import pytest

import oracle
import xmp_b200 as xmp
from xmp_b200 import tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [256, 512, 1024, 1536, 2048, 3072, 4096])
def test_kernel_is_a_neighbours(bits):
    handle = xmp.Handle()  # with the compiled-in selector and no tuned entries
    def lanes(count):
        c = xmp.powm_get_config(handle, bits, bits, count)
        return c.lanes if c.distribution == 0 else 0

    def cell(count):
        slot, src = ctypes.c_int32(0), ctypes.c_int32(0)
        shape = tuning.Shape(tuning.OPS["powm"], bits, bits, count)
        xmp.check(xmp.lib().xmpTuneGetChoice(handle.h, ctypes.byref(shape), ctypes.byref(slot), ctypes.byref(src)))
        return 1 << (slot.value // 6) if src.value == 2 else None

    for k in range(11, 20):
        near = [cell(1 << j) for j in (k - 2, k - 1, k, k + 1, k + 2)]
        assert None not in near
        for count in ((1 << k) - 1, 1 << k, (1 << k) + 1, 3 << (k - 1)):
            assert lanes(count) in near
    handle.destroy()


def test_results_between(handle):
    bits, count = 1536, 2001
    r = np.random.default_rng(3)
    x, e, m = (r.integers(0, 1 << 32, (count, bits // 32), dtype=np.uint32) for _ in range(3))
    e[:, 2:] = 0
    m[:, 0] |= 1
    X, E, M, O = (handle.integers(bits, count, v) for v in (x, e, m, x))
    xmp.powm(handle, O, X, E, M, count)
    want, _ = oracle.powm(x, e, m, count)
    assert np.array_equal(O.export(), want)
    for v in (X, E, M, O):
        v.destroy()
