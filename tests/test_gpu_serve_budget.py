"""The server's arena at small budgets, and its kernels of several Montgomery
radices: every budget that creates a server serves correct results whatever
windows and kernels it left room for, a request of up to max_wave_ops
operations fits where window tables in 32-bit limbs would have held it, and
waves at every load of a class with several radices come out right."""
import numpy as np
import pytest

import oracle
import xmp_b200 as xmp

pytestmark = pytest.mark.gpu


def _request(key, m, nops, seed):
    b = oracle.below(seed, np.repeat(m[None, :], nops, axis=0))
    return key, m, b, oracle.random_limbs(seed + 1, nops, len(m))


def _plain(handle, m, b, e):
    """The same on the batch kernels; its first and last operation against GMP."""
    bits, n = 32 * len(m), len(b)
    X, E, M, O = (handle.integers(bits, len(v), v) for v in (b, e, m[None, :].copy(), b))
    xmp.powm(handle, O, X, E, M, n)
    out = O.export()
    for v in (X, E, M, O):
        v.destroy()
    ends = [0, n - 1]
    assert np.array_equal(out[ends], oracle.powm(b[ends], e[ends], np.repeat(m[None, :], 2, axis=0), 2)[0])
    return out


def _serve(handle, srv, reqs, together=False):
    outs, rids = [np.zeros_like(b) for _, _, b, _ in reqs], []
    for (key, _, b, e), o in zip(reqs, outs):
        rids.append(srv.submit(key, b, e, o))
        if not together:
            assert srv.wait(rids[-1], 60_000_000)
    for rid in rids if together else ():
        assert srv.wait(rid, 60_000_000)
    for (_, m, b, e), o in zip(reqs, outs):
        assert np.array_equal(o, _plain(handle, m, b, e))


def _limb_slot_bytes(bits, window):
    """Operands, key index, rows and a window table in 32-bit limbs, at a precision that a register kernel's
    capacity equals."""
    n = bits // 32
    return 3 * n * 4 + 4 + 3 * n * 4 + n * 4 * (1 << window)


@pytest.mark.parametrize("bits,window", [(1024, 6), (2048, 6), (3072, 7)])
def test_request_that_the_budget_holds_in_limbs(handle, bits, window):
    keys, slots = 32, 384
    budget = 2 * keys * bits // 8 + slots * _limb_slot_bytes(bits, window) + 4096
    srv = xmp.Server(handle, [bits], hbm_budget=budget, max_keys=keys, streams=2)
    m = oracle.full_length_odd(bits, 1, bits // 32)
    key = srv.add_keys(bits, m)
    _serve(handle, srv, [_request(key, m[0], slots, 5)])
    assert srv.stats()["device_bytes"] <= budget
    srv.destroy()


@pytest.mark.parametrize("bits", [1024, 3072])
def test_every_budget_that_holds_a_server(handle, bits):
    """From a budget of 2,000 slots down to the refusal: smaller windows, then one radix."""
    m = oracle.full_length_odd(bits + 1, 2, bits // 32)
    budget, made = 2000 * _limb_slot_bytes(bits, 7), 0
    while True:
        try:
            srv = xmp.Server(handle, [bits], hbm_budget=budget, max_keys=32, streams=4)
        except xmp.XmpError as e:
            assert e.name == "xmpErrorIncreaseScratchLimit"
            break
        made += 1
        assert srv.stats()["device_bytes"] <= budget
        key = srv.add_keys(bits, m)
        sizes = [1, 64, 128]
        for nops in (256, 1000):
            try:
                srv.submit(key, np.zeros((nops, bits // 32), np.uint32), np.zeros((nops, bits // 32), np.uint32),
                           np.zeros((nops, bits // 32), np.uint32))
                sizes.append(nops)
            except xmp.XmpError as e:
                assert e.name == "xmpErrorInvalidCount"
        _serve(handle, srv, [_request(key + i % 2, m[i % 2], nops, 11 * i) for i, nops in enumerate(sizes)], made % 2 == 0)
        srv.destroy()
        budget = budget * 3 // 4
    assert made >= 8


def _radix_bits(c):
    """log2 of a lane kernel's Montgomery radix: 32-bit limbs below six a lane, else 52-bit digits."""
    bits = 32 * c.lanes * c.limbs
    return bits if c.limbs < 6 else -(-(bits + 2) // (52 * c.lanes)) * 52 * c.lanes


@pytest.mark.parametrize("bits,radices", [(1056, 1), (1536, 2), (3072, 3)])
def test_waves_of_every_load(handle, bits, radices):
    """Waves of 1 to 4,096 operations: alone, and beside a wave of another class that keeps the GPU from being idle
    (a lone small wave runs one operation per CTA)."""
    own = xmp.Handle()
    configs = [xmp.powm_get_config(own, bits, bits, 1 << b) for b in range(9, 13)]
    assert len({_radix_bits(c) for c in configs}) >= radices
    own.destroy()
    srv = xmp.Server(handle, [bits, 2048], max_keys=32, max_slots=8192, hbm_budget=4 << 30)
    m, big = oracle.full_length_odd(3, 1, bits // 32), oracle.full_length_odd(4, 1, 64)
    key, other = srv.add_keys(bits, m), srv.add_keys(2048, big)
    reqs = [_request(key, m[0], 1 << b, 20 + b) for b in range(13)]
    _serve(handle, srv, reqs)
    load = _request(other, big[0], 4096, 9)
    for r in reqs[:9]:
        _serve(handle, srv, [load, r], together=True)
    srv.destroy()
