"""Import and export through shared-memory tiles at the sizes where they can go
wrong, exact against the wire format decoded on the CPU: precisions of whole
and partial limb groups beside the tile's 32 groups, ragged instance counts,
every word size, order, byte order, nails, buffers off 16-byte alignment (host
and device), gathered and scattered rows."""
import numpy as np
import pytest
import torch

import xmp_b200 as xmp
from tests.helpers import ints_from_rows

pytestmark = pytest.mark.gpu


def _decode(raw, order, endian, size, nails):
    """Wire words (count x words) -> integers: swap bytes, mask the top `nails` bits of every word."""
    w = raw if order == -1 else raw[:, ::-1]
    if endian == 1:
        w = w.byteswap()
    w = np.ascontiguousarray(w & w.dtype.type((1 << (8 * size - nails)) - 1))
    return [int.from_bytes(r.tobytes(), "little") for r in w]


def _encode(vals, words, order, endian, size, nails):
    dt = np.dtype("u%d" % size)
    w = np.stack([np.frombuffer(v.to_bytes(words * size, "little"), dtype=dt) for v in vals])
    if endian == 1:
        w = w.byteswap()
    w = w & dt.type((1 << (8 * size - nails)) - 1)
    return np.ascontiguousarray(w if order == -1 else w[:, ::-1])


@pytest.mark.parametrize("bits", [32, 96, 128, 160, 256, 1056, 2048, 4096, 4128, 8256])
@pytest.mark.parametrize("size", [1, 2, 4, 8])
@pytest.mark.parametrize("order,endian,nails", [(-1, -1, 0), (1, 1, 0), (1, -1, 3), (-1, 1, 5)])
def test_formats(handle, bits, size, order, endian, nails):
    if bits % (8 * size):
        pytest.skip("whole words only")
    words = bits // (8 * size)
    rng = np.random.default_rng(bits + size)
    for count in (1, 33, 700):
        raw = rng.integers(0, 256, (count, bits // 8), dtype=np.uint8).view("u%d" % size)
        X = handle.integers(bits, count)
        X.import_(raw, words=words, order=order, size=size, endian=endian, nails=nails)
        vals = _decode(raw, order, endian, size, nails)
        assert ints_from_rows(X.export()) == vals
        back = X.export(order=order, size=size, endian=endian, nails=nails)
        assert np.array_equal(back, _encode(vals, words, order, endian, size, nails))
        # a device buffer off 16-byte alignment
        off = {1: 1, 2: 2, 4: 4, 8: 8}[size]
        dev = torch.zeros(count * bits // 8 + 32, dtype=torch.uint8, device="cuda")
        at = dev[off:off + count * bits // 8]
        at.copy_(torch.from_numpy(raw.view(np.uint8).reshape(-1).copy()))
        X.import_(at, count=count, words=words, order=order, size=size, endian=endian, nails=nails)
        assert ints_from_rows(X.export()) == vals
        dev.fill_(0x5a)
        X.export(count=count, order=order, size=size, endian=endian, nails=nails, out=at)
        got = dev.cpu().numpy()
        assert np.array_equal(got[off:off + count * bits // 8], back.view(np.uint8).reshape(-1))
        assert (got[:off] == 0x5a).all() and (got[off + count * bits // 8:] == 0x5a).all()
        X.destroy()


@pytest.mark.parametrize("bits", [96, 256, 2048])
def test_gather_and_scatter(handle, bits):
    count, rng = 300, np.random.default_rng(bits)
    raw = rng.integers(0, 1 << 32, (count, bits // 32), dtype=np.uint32)
    idx = rng.permutation(count).astype(np.uint32)
    some = idx.copy()
    some[::7] = count + 5  # rows past a staged host buffer: read as zero, dropped on export
    X = handle.integers(bits, count)
    pol = handle.policy()
    for use in (idx, some):
        pol.set_indices(0, use)
        handle.set_policy(pol)
        X.import_(raw, order=1)
        out = np.full_like(raw, 7)
        X.export(order=1, out=out)
        handle.set_policy(None)
        want = np.where((use < count)[:, None], raw[np.minimum(use, count - 1)], 0)
        assert np.array_equal(X.export(order=1), want)
        scattered = np.full_like(raw, 7)
        scattered[use[use < count]] = want[use < count]
        assert np.array_equal(out, scattered)
    pol.destroy()
    X.destroy()
