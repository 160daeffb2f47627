"""What the framework is asked to do in real use, as measurable cases.

Each case is a dict of plain values; prepare() makes what a program has in hand
before the call (operands on the GPU, or host rows where the path starts from
host data), run() is one pass through the public entry points.  Sizes are the
ones of bench.py, of the tests, or generic.
"""
import math

import numpy as np
import torch

import xmp_b200 as xmp

_handle = None


def handle():
    """One handle per process, as a program keeps it (scratch and tuner state live in it)."""
    global _handle
    if _handle is None:
        _handle = xmp.Handle()
    return _handle


class State:
    """Operands, results and plans of one case; gives the library's objects back when dropped."""

    def __init__(self, case):
        self.case = case
        self.h = handle()
        self._owned = []

    def own(self, obj):
        self._owned.append(obj)
        return obj

    def ints(self, bits, rows=None, count=None):
        """An integer array, filled from compact rows (GPU tensor or numpy) when given."""
        count = rows.shape[0] if count is None else count
        x = self.own(xmp.Integers(self.h, bits, count))
        if rows is not None:
            x.import_(rows, count=count, words=bits // 32)
        return x

    def rows(self, bits, count):
        return torch.empty((count, bits // 32), dtype=torch.int32, device="cuda")

    def __del__(self):
        for obj in reversed(self._owned):
            obj.destroy()
        self._owned = []


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _limbs(g, count, bits):
    """Uniform integers: compact little-endian rows of 32-bit limbs."""
    return torch.randint(-2**31, 2**31, (count, bits // 32), dtype=torch.int32, device="cuda", generator=g)


def _moduli(g, count, bits):
    """Odd, full length (top and bottom bits set), as RSA and DH moduli are."""
    m = _limbs(g, count, bits)
    m[:, 0] |= 1
    m[:, -1] |= -2**31
    return m


def _below_top(g, count, bits):
    """Operands below any full-length modulus (top bit clear)."""
    x = _limbs(g, count, bits)
    x[:, -1] &= 0x7FFFFFFF
    return x


def _to_ints(rows):
    a = rows.cpu().numpy() if isinstance(rows, torch.Tensor) else rows
    a = np.ascontiguousarray(a)
    return [int.from_bytes(r.tobytes(), "little") for r in a]


def _to_rows(values, bits):
    out = np.frombuffer(b"".join(v.to_bytes(bits // 8, "little") for v in values), dtype=np.int32)
    return torch.from_numpy(out.reshape(len(values), bits // 32).copy())


def _crt_keys(case, seed):
    """A few keys shared by the batch, as a signer has them: (p, q, dp, dq, qinv) rows, host numpy."""
    r = np.random.RandomState(seed % (1 << 31))
    half = case["bits"] // 2
    keys = []
    while len(keys) < case["keys"]:
        p, q = (int.from_bytes(r.bytes(half // 8), "little") | 1 | 1 << (half - 1) for _ in range(2))
        if math.gcd(p, q) != 1:
            continue
        dp, dq = (int.from_bytes(r.bytes(half // 8), "little") % (v - 1) for v in (p, q))
        keys.append((p, q, dp, dq, pow(q, -1, p)))
    return keys


def listed():
    return [
        # A program that adds a handful of values: host rows in, one op, host rows out, every call waited for.
        {"name": "add_256x100", "kind": "hostadd", "bits": 256, "count": 100},
        # A long vector of 256-bit values through the elementwise ops (the streaming end of the range).
        {"name": "chain_256x4194304", "kind": "chain", "bits": 256, "count": 1 << 22},
        # One exponentiation alone: the latency of a single signature or key agreement.
        {"name": "powm_2048x1", "kind": "powm", "bits": 2048, "ebits": 2048, "count": 1},
        # The plain batch: private exponents, every instance its own modulus.
        {"name": "powm_1024x4096", "kind": "powm", "bits": 1024, "ebits": 1024, "count": 4096},
        # The throughput workload: a full GPU of private exponentiations.
        {"name": "powm_2048x65536", "kind": "powm", "bits": 2048, "ebits": 2048, "count": 65536},
        # A ragged batch of larger moduli (3072 bits is the usual next size), neither lone nor full.
        {"name": "powm_3072x2001", "kind": "powm", "bits": 3072, "ebits": 3072, "count": 2001},
        # Signature verification: a short public exponent shared by the batch, many moduli.
        {"name": "verify_2048x50001", "kind": "powm", "bits": 2048, "ebits": 32, "count": 50001},
        # Signing with the CRT form of the private key, a few keys and many messages.
        {"name": "crt_2048x16384", "kind": "crt", "bits": 2048, "count": 16384, "keys": 64},
        # A server's mixture of sizes as one batch plan (1024/2048/3072/4096 bits at 40/30/20/10 %, and CRT items).
        {"name": "mixed_8192", "kind": "mixed", "count": 8192, "crt": 2048, "keys": 64},
        # Modular multiplication of 512-bit residues: a product and the quotient and remainder of it.
        {"name": "muldivmod_512x262144", "kind": "muldiv", "bits": 512, "mbits": 512, "count": 1 << 18, "quotient": True},
        # The same with RSA-size residues and a ragged count, the remainder alone.
        {"name": "mulmod_2048x10001", "kind": "muldiv", "bits": 2048, "mbits": 2048, "count": 10001, "quotient": False},
        # Big-endian byte strings (how keys and messages are stored) from host memory to the GPU and back.
        {"name": "wire_2048x65536", "kind": "wire", "bits": 2048, "count": 65536, "size": 1, "order": 1, "endian": 1},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bits(rng, lo, hi):
    """Precisions: the usual ones, and any other multiple of 32."""
    usual = [b for b in (128, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096) if lo <= b <= hi]
    if usual and rng.random() < 0.6:
        return rng.choice(usual)
    return max(lo // 32, min(hi // 32, _spread(rng, lo // 32, hi // 32))) * 32


def draw(rng):
    kind = rng.choice(["hostadd", "chain", "powm", "powm", "powm", "verify", "crt", "mixed", "muldiv", "muldiv", "wire"])
    if kind == "hostadd":
        return {"kind": kind, "bits": _bits(rng, 32, 2048), "count": _spread(rng, 1, 2000)}
    if kind == "chain":
        bits = _bits(rng, 32, 4096)
        return {"kind": kind, "bits": bits, "count": _spread(rng, 64, (1 << 30) // bits)}
    if kind == "powm":
        bits = _bits(rng, 128, 4096)
        ebits = bits if rng.random() < 0.7 else rng.choice([160, 224, 256])
        # no more than the throughput workload's multiply-adds
        most = max(1, min(1 << 18, int(65536 * (2048 / bits) ** 2 * 2048 / ebits)))
        return {"kind": kind, "bits": bits, "ebits": ebits, "count": _spread(rng, 1, most)}
    if kind == "verify":
        bits = rng.choice([1024, 2048, 3072, 4096])
        return {"kind": "powm", "bits": bits, "ebits": 32, "count": _spread(rng, 100, 65536 * 2048 // bits)}
    if kind == "crt":
        return {"kind": kind, "bits": rng.choice([1024, 2048, 3072, 4096]), "count": _spread(rng, 1, 16384),
                "keys": rng.choice([1, 16, 64])}
    if kind == "mixed":
        return {"kind": kind, "count": _spread(rng, 256, 8192), "crt": _spread(rng, 64, 2048), "keys": 16}
    if kind == "muldiv":
        bits = _bits(rng, 64, 4096)
        mbits = bits if rng.random() < 0.6 else _bits(rng, 32, bits)
        return {"kind": kind, "bits": bits, "mbits": mbits, "count": _spread(rng, 100, min(1 << 19, (1 << 36) // bits ** 2)),
                "quotient": rng.random() < 0.5}
    size = rng.choice([1, 2, 4, 8])
    bits = _bits(rng, 256, 4096)
    if bits % 64:
        size = min(size, 4)
    return {"kind": "wire", "bits": bits, "count": _spread(rng, 100, (1 << 27) // bits), "size": size,
            "order": rng.choice([1, -1]), "endian": rng.choice([1, -1])}


# ---- making the inputs -------------------------------------------------------------


def _powm_rows(case, seed):
    g = _gen(seed)
    bits, count = case["bits"], case["count"]
    m, x = _moduli(g, count, bits), _below_top(g, count, bits)
    if case["ebits"] == 32:
        e = torch.full((1, 1), 65537, dtype=torch.int32, device="cuda")
    else:
        e = _limbs(g, count, case["ebits"])
    return x, e, m


def _crt_rows(case, seed):
    """Rows of c, p, q, dp, dq, qinv for the whole batch."""
    keys = _crt_keys(case, seed)
    half, count = case["bits"] // 2, case["count"]
    pick = torch.arange(count, device="cuda") % len(keys)
    cols = [_to_rows([k[j] for k in keys], half).cuda()[pick] for j in range(5)]
    c = _limbs(_gen(seed + 1), count, case["bits"])
    c[:, -1] &= 0x3FFFFFFF  # below p q
    return [c] + cols


def _mixed_parts(case, seed):
    """The plan's items: powm cases and one CRT case, each with its own seed."""
    parts = [({"bits": b, "ebits": b, "count": max(1, case["count"] * share // 10)}, seed * 8 + j)
             for j, (b, share) in enumerate(((1024, 4), (2048, 3), (3072, 2), (4096, 1)))]
    return parts, ({"bits": 2048, "count": case["crt"], "keys": case["keys"]}, seed * 8 + 5)


def _host_rows(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    n, count = case["bits"] // 32, case["count"]
    return [r.randint(0, 1 << 32, (count, n), dtype=np.uint32) for _ in range(2)]


def _wire_rows(case, seed):
    """Wire words in (pinned) host memory."""
    r = np.random.RandomState(seed % (1 << 31))
    data = np.frombuffer(r.bytes(case["count"] * case["bits"] // 8), dtype=np.uint8)
    dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[case["size"]]
    return torch.from_numpy(data.copy()).view(dt).reshape(case["count"], -1).pin_memory()


def _muldiv_rows(case, seed):
    g = _gen(seed)
    a, b = _limbs(g, case["count"], case["bits"]), _limbs(g, case["count"], case["bits"])
    return a, b, _moduli(g, case["count"], case["mbits"])


def prepare(case, seed):
    s = State(case)
    kind, count = case["kind"], case["count"]
    if kind == "hostadd":
        s.a, s.b = _host_rows(case, seed)
        s.A, s.B, s.C = (s.ints(case["bits"], count=count) for _ in range(3))
    elif kind == "chain":
        g, bits = _gen(seed), case["bits"]
        s.A, s.B = s.ints(bits, _limbs(g, count, bits)), s.ints(bits, _limbs(g, count, bits))
        s.T, s.U = s.ints(bits, count=count), s.ints(bits, count=count)
        s.shift = torch.randint(-bits // 2, bits // 2, (count,), dtype=torch.int32, device="cuda", generator=g)
        s.out = s.rows(bits, count)
        s.sign = torch.empty(count, dtype=torch.int32, device="cuda")
        s.ones = torch.empty(count, dtype=torch.int32, device="cuda")
    elif kind == "powm":
        x, e, m = _powm_rows(case, seed)
        s.X, s.E, s.M = s.ints(case["bits"], x), s.ints(case["ebits"], e), s.ints(case["bits"], m)
        s.O, s.out = s.ints(case["bits"], count=count), s.rows(case["bits"], count)
    elif kind == "crt":
        rows = _crt_rows(case, seed)
        s.args = [s.ints(case["bits"] if j == 0 else case["bits"] // 2, v) for j, v in enumerate(rows)]
        s.O, s.out = s.ints(case["bits"], count=count), s.rows(case["bits"], count)
    elif kind == "mixed":
        parts, (cc, cseed) = _mixed_parts(case, seed)
        items, s.res = [], []
        for c, sd in parts:
            x, e, m = (s.ints(c["bits"], v) for v in _powm_rows(c, sd))
            o = s.ints(c["bits"], count=c["count"])
            items.append((o, x, e, m, c["count"]))
            s.res.append((o, c["count"], s.rows(c["bits"], c["count"])))
        args = [s.ints(cc["bits"] if j == 0 else cc["bits"] // 2, v) for j, v in enumerate(_crt_rows(cc, cseed))]
        o = s.ints(cc["bits"], count=cc["count"])
        s.res.append((o, cc["count"], s.rows(cc["bits"], cc["count"])))
        s.plan = s.own(xmp.BatchPlan(s.h, items, crt=[(o, *args, cc["count"])], use_graph=True))
    elif kind == "muldiv":
        a, b, m = _muldiv_rows(case, seed)
        bits, mbits = case["bits"], case["mbits"]
        s.A, s.B, s.M = s.ints(bits, a), s.ints(bits, b), s.ints(mbits, m)
        s.P, s.R, s.r = s.ints(2 * bits, count=count), s.ints(mbits, count=count), s.rows(mbits, count)
        if case["quotient"]:
            s.Q, s.q = s.ints(2 * bits, count=count), s.rows(2 * bits, count)
    else:  # wire
        s.src = _wire_rows(case, seed)
        s.dst = torch.empty_like(s.src).pin_memory()
        s.X = s.ints(case["bits"], count=count)
    return s


# ---- one pass ----------------------------------------------------------------------


def run(s):
    case, h = s.case, s.h
    kind, count = case["kind"], case["count"]
    if kind == "hostadd":
        s.A.import_(s.a)
        s.B.import_(s.b)
        xmp.add(h, s.C, s.A, s.B, count)
        return s.C.export()
    if kind == "chain":
        xmp.add(h, s.T, s.A, s.B, count, asynchronous=True)
        xmp.xor(h, s.T, s.T, s.A, count, asynchronous=True)
        xmp.shf(h, s.U, s.T, s.shift, count)
        xmp.sub(h, s.T, s.U, s.B, count, asynchronous=True)
        xmp.cmp(h, s.T, s.A, count, out=s.sign)
        xmp.popc(h, s.T, count, out=s.ones)
        s.T.export(count=count, out=s.out, asynchronous=True)
        return s.out, s.sign, s.ones
    if kind == "powm":
        xmp.powm(h, s.O, s.X, s.E, s.M, count, asynchronous=True)
        s.O.export(count=count, out=s.out, asynchronous=True)
        return s.out
    if kind == "crt":
        xmp.powm_crt(h, s.O, *s.args, count, asynchronous=True)
        s.O.export(count=count, out=s.out, asynchronous=True)
        return s.out
    if kind == "mixed":
        s.plan.execute()
        for o, n, rows in s.res:
            o.export(count=n, out=rows, asynchronous=True)
        return [rows for _, _, rows in s.res]
    if kind == "muldiv":
        xmp.mul(h, s.P, s.A, s.B, count, asynchronous=True)
        if case["quotient"]:
            xmp.divmod_(h, s.Q, s.R, s.P, s.M, count, asynchronous=True)
            s.Q.export(count=count, out=s.q, asynchronous=True)
        else:
            xmp.mod(h, s.R, s.P, s.M, count, asynchronous=True)
        s.R.export(count=count, out=s.r, asynchronous=True)
        return (s.q, s.r) if case["quotient"] else s.r
    words = case["bits"] // (8 * case["size"])
    s.X.import_(s.src, count=count, words=words, order=case["order"], size=case["size"], endian=case["endian"],
                asynchronous=True)
    return s.X.export(count=count, order=case["order"], size=case["size"], endian=case["endian"], out=s.dst)


# ---- what a pass cannot do without -------------------------------------------------


def _powm_flops(bits, ebits, ones=None):
    """Multiply-adds (two operations each) of one exponentiation: ebits squarings and a product per six bits,
    32 x 32-bit limbs, a square's cross products once, Montgomery reduction n^2 + n."""
    n = bits // 32
    mults = math.ceil(ebits / 6) if ones is None else ones
    return 2.0 * (ebits * (n * (n + 1) / 2 + n * n + n) + mults * (2 * n * n + n))


def _powm_work(c):
    b, count = c["bits"] // 8, c["count"]
    if c["ebits"] == 32:  # 65537: 16 squarings and a product
        return 3.0 * b * count, _powm_flops(c["bits"], 16, 1) * count
    return (3.0 * b + c["ebits"] / 8) * count, _powm_flops(c["bits"], c["ebits"]) * count


def _crt_work(c):
    half = c["bits"] // 2
    return (2.0 * c["bits"] + 5.0 * half) / 8 * c["count"], 2 * _powm_flops(half, half) * c["count"]


def work(case):
    kind, count = case["kind"], case["count"]
    b, n = case.get("bits", 0) / 8, case.get("bits", 0) // 32
    if kind == "hostadd":
        return {"bytes": 3 * b * count, "flops": 1.0 * n * count}
    if kind == "chain":  # each op's operands and result once, the result's rows once
        return {"bytes": (3 + 3 + 2 + 3 + 2 + 1 + 2) * b * count + 12.0 * count, "flops": 6.0 * n * count}
    if kind == "powm":
        by, fl = _powm_work(case)
        return {"bytes": by, "flops": fl}
    if kind == "crt":
        by, fl = _crt_work(case)
        return {"bytes": by, "flops": fl}
    if kind == "mixed":
        parts, (cc, _) = _mixed_parts(case, 0)
        all_ = [_powm_work(c) for c, _ in parts] + [_crt_work(cc)]
        return {"bytes": sum(v[0] for v in all_), "flops": sum(v[1] for v in all_)}
    if kind == "muldiv":
        m = case["mbits"] / 8
        by = (2 * b + 2 * b) + (2 * b + 2 * m) + (2 * b if case["quotient"] else 0) + m
        nm = case["mbits"] // 32
        return {"bytes": by * count, "flops": 2.0 * count * (n * n + (2 * n - nm + 1) * nm)}
    return {"bytes": 4 * b * count, "flops": 0.0}


# ---- the results, with plain integers ----------------------------------------------


def _exact_powm(case, seed):
    x, e, m = (_to_ints(v) for v in _powm_rows(case, seed))
    return _to_rows([pow(a, e[i % len(e)], c) for i, (a, c) in enumerate(zip(x, m))], case["bits"])


def _exact_crt(case, seed):
    c, p, q, dp, dq, qinv = (_to_ints(v) for v in _crt_rows(case, seed))
    out = []
    for i in range(case["count"]):
        mp, mq = pow(c[i], dp[i], p[i]), pow(c[i], dq[i], q[i])
        out.append(mq + q[i] * ((mp - mq) * qinv[i] % p[i]))
    return _to_rows(out, case["bits"])


def exact(case, seed):
    kind, count = case["kind"], case["count"]
    if kind in ("powm", "crt", "mixed"):
        if work(case)["flops"] > 2e10:  # Python's pow: about 1e9 of these operations a second
            return None
        if kind == "powm":
            return _exact_powm(case, seed)
        if kind == "crt":
            return _exact_crt(case, seed)
        parts, crt = _mixed_parts(case, seed)
        return [_exact_powm(c, sd) for c, sd in parts] + [_exact_crt(*crt)]
    if count * case["bits"] > 1 << 26:
        return None
    bits = case["bits"]
    top = (1 << bits) - 1
    if kind == "hostadd":
        a, b = (_to_ints(v) for v in _host_rows(case, seed))
        return _to_rows([(x + y) & top for x, y in zip(a, b)], bits).numpy().view(np.uint32)
    if kind == "chain":
        g = _gen(seed)
        a, b = _to_ints(_limbs(g, count, bits)), _to_ints(_limbs(g, count, bits))
        sh = torch.randint(-bits // 2, bits // 2, (count,), dtype=torch.int32, device="cuda", generator=g).tolist()
        out, sign, ones = [], [], []
        for x, y, k in zip(a, b, sh):
            t = ((x + y) & top) ^ x
            t = (t << k) & top if k >= 0 else t >> -k
            t = (t - y) & top
            out.append(t)
            sign.append((t > x) - (t < x))
            ones.append(t.bit_count())
        return _to_rows(out, bits), torch.tensor(sign, dtype=torch.int32), torch.tensor(ones, dtype=torch.int32)
    if kind == "muldiv":
        a, b, m = (_to_ints(v) for v in _muldiv_rows(case, seed))
        r = _to_rows([x * y % z for x, y, z in zip(a, b, m)], case["mbits"])
        if not case["quotient"]:
            return r
        return _to_rows([x * y // z for x, y, z in zip(a, b, m)], 2 * bits), r
    return _wire_rows(case, seed)
