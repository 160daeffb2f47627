"""The scratch arena: the plain calls leave it at the size that their
asynchronous forms need."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp
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
