"""Import and export on both sides of the sizes at which they change kernels
(per word, tiles, whole groups), exact against numpy: formats of every word
size around 2^19 words and 1 MB, native rows around 16 MB, partial limb groups,
rows of a single group, host and device buffers."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp  # noqa: F401  (the handle fixture's library)

pytestmark = pytest.mark.gpu


def _limbs(raw, order, endian, nails):
    """Wire words (count x words) -> little-endian 32-bit limbs."""
    w = raw if order == -1 else raw[:, ::-1]
    w = w.byteswap() if endian == 1 else w
    w = w & w.dtype.type((1 << (8 * w.dtype.itemsize - nails)) - 1)
    return np.ascontiguousarray(w).view(np.uint8).reshape(len(raw), -1).view("<u4")


def _words(limbs, size, order, endian, nails):
    """Little-endian 32-bit limbs -> wire words; the top `nails` bits of a stored word are clear."""
    w = np.ascontiguousarray(limbs).view(np.uint8).reshape(len(limbs), -1).view("u%d" % size)
    w = w.byteswap() if endian == 1 else w
    w = w & w.dtype.type((1 << (8 * size - nails)) - 1)
    return w if order == -1 else w[:, ::-1]


def _check(handle, bits, count, size, order, endian, nails, device):
    rng = np.random.default_rng(bits + count + size)
    words = bits // (8 * size)
    raw = rng.integers(0, 256, (count, bits // 8), dtype=np.uint8).view("u%d" % size)
    want = _limbs(raw, order, endian, nails)
    x = handle.integers(bits, count)
    buf = torch.from_numpy(raw.view(np.uint8).copy())
    buf = buf.cuda() if device else buf
    x.import_(buf, count=count, words=words, order=order, size=size, endian=endian, nails=nails)
    assert np.array_equal(x.export(count), want)
    out = torch.zeros_like(buf)
    x.export(count, order=order, size=size, endian=endian, nails=nails, out=out)
    assert np.array_equal(out.cpu().numpy().view("u%d" % size), _words(want, size, order, endian, nails))
    x.destroy()


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("bits", [32, 96, 128, 160, 1024, 1056, 2048, 4128])
@pytest.mark.parametrize("size,order,endian,nails", [(1, 1, 1, 0), (2, -1, 1, 0), (2, 1, -1, 3), (4, 1, 1, 0),
                                                     (4, -1, -1, 5), (8, 1, -1, 0), (8, -1, 1, 7)])
def test_formats_around_the_limit(handle, bits, size, order, endian, nails, device):
    if bits % (8 * size):
        pytest.skip("whole words only")
    most = min((1 << 19) // (bits // (8 * size)), (1 << 20) // (bits // 8))
    for count in (most, most + 1, most + 333):
        _check(handle, bits, count, size, order, endian, nails, device)


@pytest.mark.parametrize("bits", [32, 128, 160, 256, 1056, 2048])
def test_native_around_the_limit(handle, bits):
    most = (16 << 20) // (bits // 8)
    for count in (most, most + 1):
        _check(handle, bits, count, 4, -1, -1, 0, True)
