"""Synchronous imports and exports of a few pageable rows (passed as kernel
arguments, taken through mapped memory) at and beside their size limits, with
partial limb groups, pinned and device buffers beside pageable ones,
fewer rows than the array holds, and an import while the stream is
busy."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limbs,count", [(1, 1), (1, 896), (1, 897), (3, 298), (3, 299), (4, 224), (4, 225), (5, 179),
                                         (64, 14), (64, 15), (7, 128), (896, 1), (897, 1), (64, 256), (64, 257),
                                         (1, 16384), (1, 16385), (3, 5461), (3, 5462)])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "device"])
def test_limits(handle, limbs, count, kind):
    r = np.random.default_rng(limbs * 100003 + count)
    rows = r.integers(0, 1 << 32, (count, limbs), dtype=np.uint32)
    x = handle.integers(32 * limbs, count + 3)
    x.import_(np.full((count + 3, limbs), 0xa5a5a5a5, dtype=np.uint32), count=count + 3, words=limbs)
    src = torch.from_numpy(rows.view(np.int32).copy())
    src = src.pin_memory() if kind == "pinned" else src.cuda() if kind == "device" else src
    x.import_(src, count=count, words=limbs)
    src.zero_()  # the call has read them
    got = x.export(count + 3)
    assert np.array_equal(got[:count], rows) and (got[count:] == 0xa5a5a5a5).all()
    dst = torch.zeros((count, limbs), dtype=torch.int32)
    dst = dst.pin_memory() if kind == "pinned" else dst.cuda() if kind == "device" else dst
    x.export(count, out=dst)
    assert np.array_equal(dst.cpu().numpy().view(np.uint32), rows)
    x.destroy()


def test_import_behind_queued_work(handle):
    """Rows imported while the stream still works on the array: the old values go into the queued call."""
    bits, count = 1024, 20
    r = np.random.default_rng(7)
    a, b = (r.integers(0, 1 << 32, (count, 32), dtype=np.uint32) for _ in range(2))
    m = r.integers(0, 1 << 32, (count, 32), dtype=np.uint32)
    m[:, 0] |= 1
    A, M, O, P = handle.integers(bits, count, a), handle.integers(bits, count, m), handle.integers(bits, count), \
        handle.integers(bits, count)
    xmp.powm(handle, O, A, A, M, count)
    want = O.export()
    xmp.powm(handle, P, A, A, M, count, asynchronous=True)
    A.import_(b, count=count, words=32)
    assert np.array_equal(P.export(), want) and np.array_equal(A.export(), b)
    for v in (A, M, O, P):
        v.destroy()
