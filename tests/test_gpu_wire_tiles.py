"""The import and export tile kernel on the paths that only large arrays take
(foreign formats above 2^19 words or 1 MB, single-limb imports above 4 MB), exact
against numpy: single limbs in and out with a partial last group, 16-byte units
through buffers off 16-byte alignment, precisions of more than one tile's 32
groups, gathered and scattered rows, rows past a host buffer's end."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp  # noqa: F401  (the handle fixture's library)
from tests.test_gpu_wire_sizes import _limbs, _words

pytestmark = pytest.mark.gpu

FORMATS = [(1, 1, 1, 0), (2, -1, 1, 0), (2, 1, -1, 3), (4, 1, 1, 0), (4, -1, -1, 5), (8, 1, -1, 0), (8, -1, 1, 7)]


def _raw(bits, count, size):
    rng = np.random.default_rng(bits + count + size)
    return rng.integers(0, 256, (count, bits // 8), dtype=np.uint8).view("u%d" % size)


@pytest.mark.parametrize("bits", [160, 1056, 4128, 8192, 8256])
@pytest.mark.parametrize("size,order,endian,nails", FORMATS)
def test_single_limbs_and_many_groups(handle, bits, size, order, endian, nails):
    if bits % (8 * size):
        pytest.skip("whole words only")
    words = bits // (8 * size)
    count = (5 << 20) // (bits // 8) + 33
    raw = _raw(bits, count, size)
    want = _limbs(raw, order, endian, nails)
    out_want = np.ascontiguousarray(_words(want, size, order, endian, nails))
    x = handle.integers(bits, count)
    for off in (0, max(4, size)):  # bytes from 16-byte alignment; whole words all the same
        dev = torch.zeros(count * bits // 8 + 64, dtype=torch.uint8, device="cuda")
        at = dev[off:off + count * bits // 8]
        at.copy_(torch.from_numpy(raw.view(np.uint8).reshape(-1).copy()))
        x.import_(at, count=count, words=words, order=order, size=size, endian=endian, nails=nails)
        assert np.array_equal(x.export(count), want)
        dev.fill_(0x5a)
        x.export(count, order=order, size=size, endian=endian, nails=nails, out=at)
        got = dev.cpu().numpy()
        assert np.array_equal(got[off:off + count * bits // 8], out_want.view(np.uint8).reshape(-1))
        assert (got[:off] == 0x5a).all() and (got[off + count * bits // 8:] == 0x5a).all()
    x.destroy()


@pytest.mark.parametrize("bits", [96, 160, 256, 1056, 2048, 8192])
@pytest.mark.parametrize("size,order,endian,nails", [(1, 1, 1, 0), (4, 1, -1, 0), (4, -1, 1, 5), (2, -1, -1, 0)])
def test_gather_and_scatter(handle, bits, size, order, endian, nails):
    words = bits // (8 * size)
    count = (5 << 20) // (bits // 8) + 7
    raw = _raw(bits, count, size)
    limbs = _limbs(raw, order, endian, nails)
    rng = np.random.default_rng(bits)
    idx = rng.permutation(count).astype(np.uint32)
    some = idx.copy()
    some[::7] = count + 5  # past the host buffer: read as zero, dropped on export
    x = handle.integers(bits, count)
    pol = handle.policy()
    try:
        for use in (idx, some):
            pol.set_indices(0, use)
            handle.set_policy(pol)
            x.import_(raw, words=words, order=order, size=size, endian=endian, nails=nails)
            out = np.full_like(raw, 7)
            x.export(count, order=order, size=size, endian=endian, nails=nails, out=out)
            handle.set_policy(None)
            want = np.where((use < count)[:, None], limbs[np.minimum(use, count - 1)], 0).astype(np.uint32)
            assert np.array_equal(x.export(count), want)
            scattered = np.full_like(raw, 7)
            rows = _words(want, size, order, endian, nails)
            scattered[use[use < count]] = rows[use < count]
            assert np.array_equal(out, scattered)
        pol.set_indices(0, idx)
        handle.set_policy(pol)
        dev = torch.from_numpy(raw.view(np.uint8).copy()).cuda()
        x.import_(dev, count=count, words=words, order=order, size=size, endian=endian, nails=nails)
        back = torch.zeros_like(dev)
        x.export(count, order=order, size=size, endian=endian, nails=nails, out=back)
        handle.set_policy(None)
        assert np.array_equal(x.export(count), limbs[idx])
        assert np.array_equal(back.cpu().numpy().view("u%d" % size)[idx], _words(limbs[idx], size, order, endian, nails))
    finally:
        handle.set_policy(None)
        pol.destroy()
        x.destroy()
