"""What a user of the engine has it do, as measurable cases.

A case is one pass through a public entry point: a host call of `Key` on NumPy
arrays, a device call of the C-ABI (`hg_dev_*`) on torch tensors, or a graph
replay of a `Batch`.  `listed()` names the fixed ones, `draw(rng)` gives more of
the same ranges, `prepare` makes a case's inputs and loads its key, `run` is the
timed pass, `work` the bytes and operations that the path cannot do without and
`exact` the expected outputs in plain Python integers.
"""

import ctypes
import functools
import math

import numpy as np
import torch

import heu_gb300 as hg
from heu_gb300 import batch as hb
from heu_gb300 import capi

# Key pairs as a program reads them from its key file: (p, q) by key size.
_PRIMES = {
    1024: (
        int(
            "fa23cea36ffedc865d3dfb9eef46b51be9ca6c7249c4caba8ea764828d31284f4abf32a3ba90d83ad95f6df00719b1cd"
            "0e9c1086264172b63578dc7b1a693f17", 16),
        int(
            "86840e6410c9e536d2c2d71e22ab8c10188f04b5e8cd4288dec63b205e9ae130104f3c8a8bc54b96debb23acac48cf09"
            "6506d9665e9665df4a4ab8cbbc62096f", 16),
    ),
    2048: (
        int(
            "f18ca18c97de55ec3f00fa3b552ef6c4ce0366d47e60adce4ca1e3a7fce0a94288de050245f0f9b2100ae93ca508d02e"
            "a3f39bdf6f8668f4f9b9c01121a82eaf9b7536cd3c368430961e7fcba86b8dfa5fe15698d33ad156823bdad2efff1975"
            "1a4195ffb607cd4d639fadfda3d29b810f3608d9fea1e61ddc1d84e28f8b4ff3", 16),
        int(
            "964ddb46cd8747c1d570a17617190ee8433a674cfb1de80c74867a399e735b6fb2e688163ad5fae76bd7b93fba5fc1a6"
            "ce9b48b3982c6bc01b19a4d5c992e236bd74956d8ab07777955564a50faeabb9882a3c78afa2bbd47daf290e771cebcc"
            "e73e84775c07df402cbfb9dec5590d423ba98008514fb9cd747481377c7a04b3", 16),
    ),
    3072: (
        int(
            "a8b3ee78e204793757ec28fdfe80e64265fc9cb8458d12f6654cbeb02b58bfc818c7356ac86b3a918a51766b1563ffe5"
            "39412e43dd336597955433e28749eabf4bc4c687a00f875a2867e7df494d5a7a8d491a930c6ee619e7b6cbf343d0371f"
            "4c2b277b68dceea329e038998aec1af3e879497327d74fdfa34cf13631525f7c968c4be8e215efcdfd8ba577bc910646"
            "a830f9ddb26691c541c6fb8f47dd05fe624ca3f63446824bb72a44edc9e38fb1d72e1f0ebaf8ed082fd3289d30f3c9a3", 16),
        int(
            "fbe4e7e2f893609b19e5fba8a435c7b06b75369f6b1fa0f73060834aec2810549990b80851a48251eef103019a283b2b"
            "8728aacbb1f649e8e71e77b1bc34e3cb763d700468fbf844b7825b693cdc52126a0162dc28fdd43e809954ab670efb8e"
            "98f6c6a4750f0d839cbe49c056a4ddf7ecfcbdbda2f383cf4306e26ce638fe4d03a6cd70ed156671793b1b326c03ab9e"
            "ffe7c6fbca79dccdc092b25300b96c5fb62ba0ffdc908e73823c553888c711d7be2cb9e40318e9c62d79b36562e0af77", 16),
    ),
}


@functools.lru_cache(maxsize=None)
def _numbers(bits):
    """n, h_s, p, q of the key of `bits` bits: h_s = (-x^2)^n mod n^2."""
    p, q = _PRIMES[bits]
    n = p * q
    x = 0x9E3779B97F4A7C15F39CC0605CEDC835
    return n, pow(n - x * x % n, n, n * n), p, q


def listed():
    return [
        # one value encrypted in a host call: an interactive client
        {"name": "encrypt_one", "op": "encrypt", "host": True, "bits": 2048, "window": 12, "n": 1},
        # a handful of results opened in a host call: the end of a protocol round
        {"name": "decrypt_few", "op": "decrypt", "host": True, "bits": 2048, "window": 12, "n": 8},
        # a column of features or gradients encrypted on the device
        {"name": "encrypt_2048", "op": "encrypt", "host": False, "bits": 2048, "window": 16, "n": 131072},
        # the same at the long key size with the default table, a ragged length
        {"name": "encrypt_3072", "op": "encrypt", "host": False, "bits": 3072, "window": 12, "n": 20001},
        # a column of results opened on the device: the longest operation of the scheme
        {"name": "decrypt_2048", "op": "decrypt", "host": False, "bits": 2048, "window": 12, "n": 65536},
        {"name": "decrypt_3072", "op": "decrypt", "host": False, "bits": 3072, "window": 12, "n": 5001},
        # element-wise sum of two encrypted columns of a million rows
        {"name": "add_2048", "op": "add", "host": False, "bits": 2048, "window": 12, "n": 1048576},
        # an encrypted column times a signed 64-bit plaintext column
        {"name": "mul_2048", "op": "mul", "host": False, "bits": 2048, "window": 12, "n": 65537},
        # the sum of an encrypted column
        {"name": "sum_2048", "op": "sum", "host": False, "bits": 2048, "window": 12, "n": 524288},
        # gradient histograms of a boosting iteration: rows x features into 64 buckets
        {"name": "bucket_sum_2048", "op": "bucket_sum", "host": False, "bits": 2048, "window": 12, "n": 100003,
         "features": 8, "buckets": 64},
        # an encrypted matrix times a 16-bit integer matrix (linear model scoring)
        {"name": "matmul_2048", "op": "matmul", "host": False, "bits": 2048, "window": 12, "n": 256, "k": 128,
         "cols": 32, "scalar_bits": 16},
        # uneven jobs of three key sizes in one graph-replayed persistent launch
        {"name": "batch_mixed", "op": "batch", "host": False, "bits": 0, "window": 12, "n": 4096},
    ]


# Operations that draw() picks from, and the most elements of each.
_MOST = {"encrypt": 131072, "decrypt": 65536, "add": 1048576, "sub": 262144, "add_plain": 262144, "mul": 65537,
         "sum": 524288, "bucket_sum": 100003, "matmul": 256, "batch": 4096}
_HOST_MOST = 4096  # host calls of the declared range are the small ones


def _log_uniform(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    op = rng.choice(sorted(_MOST))
    host = op in ("encrypt", "decrypt", "add", "sub", "add_plain", "mul", "sum") and rng.random() < 0.3
    case = {"op": op, "host": host, "bits": rng.choice([1024, 2048, 2048, 3072]), "window": rng.choice([8, 10, 12, 14])}
    top = min(_MOST[op], _HOST_MOST) if host else _MOST[op]
    if op == "bucket_sum":
        case.update(features=rng.randint(1, 8), buckets=rng.choice([2, 10, 32, 64, 100, 256]))
    elif op == "matmul":
        case.update(k=rng.randint(1, 128), cols=rng.randint(1, 32), scalar_bits=rng.randint(2, 32))
    elif op == "batch":
        case.update(bits=0)
    case["n"] = _log_uniform(rng, 16 if op == "batch" else 1, top)
    limit = work(listed()[4])["flops"]  # decrypt_2048
    while case["n"] > 16 and work(case)["flops"] > limit:
        case["n"] = case["n"] * 2 // 3
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _p(t):
    return ctypes.c_void_p(t.data_ptr())


class _Gen:
    """Seeded random inputs on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def ints(self, shape, lo, hi):
        return torch.randint(lo, hi, shape, dtype=torch.int64, device="cuda", generator=self.g)

    def r(self, n, limbs):
        """Encryption randomness: `limbs` limbs with the top bit set, as RandomExactBits draws it."""
        v = torch.randint(-(2 ** 31), 2 ** 31, (n, limbs), dtype=torch.int32, device="cuda", generator=self.g)
        v[:, -1] |= -(2 ** 31)
        return v


def _load(ctx, bits, window):
    n, h_s, p, q = _numbers(bits)
    return ctx.load_key(bits, n, h_s, p, q, table_window=window)


def _empty_ct(key, *shape):
    return torch.empty((*shape, key.ct_limbs), dtype=torch.int32, device="cuda")


def _plain(gen, n):
    """Fixed-point feature values and gradients: signed, up to 40 bits."""
    return gen.ints((n,), -(2 ** 40), 2 ** 40)


def _encrypted(gen, key, n):
    """(m, ciphertexts) of `n` fresh encryptions."""
    m, r, ct = _plain(gen, n), gen.r(n, key.r_limbs), _empty_ct(key, n)
    torch.cuda.current_stream().synchronize()
    capi.check(key.lib.hg_dev_encrypt(key.ctx.handle, key.id, _p(m), _p(r), _p(ct), n, None))
    capi.check(key.lib.hg_dev_check(key.ctx.handle))
    return m, ct


def _host_ct(ct):
    return ct.cpu().numpy().view(np.uint32)


def _batch_jobs(n):
    """(key bits, operation, length) of the uneven jobs of a batch of size `n`."""
    return [(2048, "decrypt", n), (2048, "encrypt", 2 * n + 1), (2048, "mul", n + 3), (2048, "add", 4 * n),
            (3072, "decrypt", n // 4 + 1), (3072, "encrypt", n // 2), (3072, "add", n),
            (1024, "decrypt", n // 2 + 1), (1024, "mul", n // 3 + 1), (1024, "encrypt", n)]


def prepare(case, seed):
    gen, op, n = _Gen(seed), case["op"], case["n"]
    st = {"case": case, "stream": torch.cuda.Stream()}
    ctx = st["ctx"] = hg.Context(0)
    if op == "batch":
        keys = {b: _load(ctx, b, case["window"]) for b in (1024, 2048, 3072)}
        b = st["batch"] = hb.Batch(ctx)
        st["out"], st["held"] = [], [keys]
        for bits, what, count in _batch_jobs(n):
            key = keys[bits]
            if what == "encrypt":
                a, c = _plain(gen, count), gen.r(count, key.r_limbs)
                code = hb.ENCRYPT
            else:
                _, a = _encrypted(gen, key, count)
                c = None
                code = {"decrypt": hb.DECRYPT, "mul": hb.MUL, "add": hb.ADD}[what]
                if what == "mul":
                    c = gen.ints((count,), -(2 ** 63), 2 ** 63 - 1)
                elif what == "add":
                    _, c = _encrypted(gen, key, count)
            if what == "decrypt":
                out = torch.empty((count,), dtype=torch.int64, device="cuda")
                aux = torch.empty((count,), dtype=torch.uint8, device="cuda")
            else:
                out, aux = _empty_ct(key, count), None
            b.add(key, code, count, a, c, out, aux)
            st["held"].append((a, c))
            st["out"].append((out, aux) if aux is not None else out)
        return st
    key = st["key"] = _load(ctx, case["bits"], case["window"])
    if op == "encrypt":
        st["m"], st["r"] = _plain(gen, n), gen.r(n, key.r_limbs)
        st["out"] = _empty_ct(key, n)
    elif op == "decrypt":
        _, st["a"] = _encrypted(gen, key, n)
        st["out"] = torch.empty((n,), dtype=torch.int64, device="cuda")
        st["ovf"] = torch.empty((n,), dtype=torch.uint8, device="cuda")
    elif op in ("add", "sub"):
        (_, st["a"]), (_, st["b"]) = _encrypted(gen, key, n), _encrypted(gen, key, n)
        st["out"] = _empty_ct(key, n)
    elif op == "add_plain":
        _, st["a"] = _encrypted(gen, key, n)
        st["k"] = _plain(gen, n)
        st["out"] = _empty_ct(key, n)
    elif op == "mul":
        _, st["a"] = _encrypted(gen, key, n)
        st["k"] = gen.ints((n,), -(2 ** 63), 2 ** 63 - 1)
        st["out"] = _empty_ct(key, n)
    elif op == "sum":
        _, st["a"] = _encrypted(gen, key, n)
        st["out"] = _empty_ct(key, 1)
    elif op == "bucket_sum":
        _, st["a"] = _encrypted(gen, key, n)
        F, B = case["features"], case["buckets"]
        st["om"] = gen.ints((n, F), 0, B).to(torch.uint8)
        st["out"] = _empty_ct(key, F * B)
    elif op == "matmul":
        M, K, N = n, case["k"], case["cols"]
        _, st["a"] = _encrypted(gen, key, M * K)
        h = 2 ** (case["scalar_bits"] - 1)
        st["y"] = gen.ints((K, N), -h, h).cpu().contiguous()
        st["out"] = _empty_ct(key, M, N)
    if case["host"]:
        for name in ("a", "b"):
            if name in st:
                st[name] = _host_ct(st[name])
        for name in ("m", "k"):
            if name in st:
                st[name] = st[name].cpu().numpy()
        if "r" in st:
            st["r"] = st["r"].cpu().numpy().view(np.uint32)
        del st["out"]
    return st


# ---------------------------------------------------------------------------
# the timed pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    op, n = case["op"], case["n"]
    if op == "batch":
        st["batch"].run(stream=st["stream"], graph=True)
        return st["out"]
    key = st["key"]
    if case["host"]:
        if op == "encrypt":
            out = key.encrypt(st["m"], st["r"])
        elif op == "decrypt":
            m, ovf = key.decrypt(st["a"])
            return m, ovf
        elif op in ("add", "sub"):
            out = getattr(key, op)(st["a"], st["b"])
        elif op in ("add_plain", "mul"):
            out = getattr(key, op)(st["a"], st["k"])
        else:
            out = key.sum(st["a"])
        return out.view(np.int32)
    lib, h, kid, s, out = key.lib, key.ctx.handle, key.id, ctypes.c_void_p(st["stream"].cuda_stream), _p(st["out"])
    if op == "encrypt":
        capi.check(lib.hg_dev_encrypt(h, kid, _p(st["m"]), _p(st["r"]), out, n, s))
    elif op == "decrypt":
        capi.check(lib.hg_dev_decrypt(h, kid, _p(st["a"]), out, _p(st["ovf"]), n, s))
        return st["out"], st["ovf"]
    elif op == "add":
        capi.check(lib.hg_dev_add(h, kid, _p(st["a"]), _p(st["b"]), out, n, s))
    elif op == "sub":
        capi.check(lib.hg_dev_sub(h, kid, _p(st["a"]), _p(st["b"]), out, n, s))
    elif op == "add_plain":
        capi.check(lib.hg_dev_add_plain(h, kid, _p(st["a"]), _p(st["k"]), out, n, s))
    elif op == "mul":
        capi.check(lib.hg_dev_mul(h, kid, _p(st["a"]), _p(st["k"]), out, n, s))
    elif op == "sum":
        capi.check(lib.hg_dev_sum(h, kid, _p(st["a"]), n, out, s))
    elif op == "bucket_sum":
        capi.check(lib.hg_dev_bucket_sum(h, kid, _p(st["a"]), n, 1, _p(st["om"]), case["features"], case["buckets"], 0,
                                         out, s))
    elif op == "matmul":
        capi.check(lib.hg_dev_matmul(h, kid, _p(st["a"]), n, case["k"], _p(st["y"]), case["cols"], out, s))
    return st["out"]


# ---------------------------------------------------------------------------
# what the path cannot do without
# ---------------------------------------------------------------------------
def _mul_square(h):
    """32-bit multiply-adds of a product modulo the square of an h-limb number (two digits to that base)."""
    return 5 * h * h


def _sqr_square(h):
    return 3.5 * h * h


def _mul_any(s):
    """The same for any modulus of s limbs: the product and its reduction."""
    return 2 * s * s


def _op_work(op, bits, n, window, case=None):
    """(bytes, multiply-adds) of one operation on n elements."""
    s = bits // 16
    h, hh, ct = s // 2, s // 4, 4 * s
    if op == "encrypt":
        return n * (8 + bits // 16 + ct), n * (-(-(bits // 2) // window)) * 4 * h * h
    if op == "decrypt":
        half = bits // 2
        return n * (ct + 9), n * 2 * (half * _sqr_square(hh) + half / 7 * _mul_square(hh))
    if op == "add":
        return n * 3 * ct, n * _mul_any(s)
    if op == "sub":
        return n * 3 * ct, n * 4 * _mul_any(s)
    if op == "add_plain":
        return n * (2 * ct + 8), n * 1.25 * _mul_any(s)
    if op == "mul":
        return n * (2 * ct + 8), n * (63 * _sqr_square(h) + 18 * _mul_square(h))
    if op == "sum":
        return n * ct + ct, n * _mul_any(s)
    if op == "bucket_sum":
        f, b = case["features"], case["buckets"]
        return n * (ct + f) + f * b * ct, n * f * _mul_any(s)
    m, k, c, bit = n, case["k"], case["cols"], case["scalar_bits"]
    return (m * k + m * c) * ct + 8 * k * c, m * c * (bit * -(-k // 8) * _mul_square(h) + bit * _sqr_square(h))


def work(case):
    if case["op"] == "batch":
        parts = [_op_work(what, bits, count, case["window"]) for bits, what, count in _batch_jobs(case["n"])]
    else:
        parts = [_op_work(case["op"], case["bits"], case["n"], case["window"], case)]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": 2.0 * sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------
# expected outputs
# ---------------------------------------------------------------------------
def _to_ints(a):
    a = np.ascontiguousarray(a).view(np.uint32)
    return [int.from_bytes(row.tobytes(), "little") for row in a]


def exact(case, seed):
    op, bits, n = case["op"], case["bits"], case["n"]
    if op == "decrypt":  # what was encrypted, and no value out of the int64 range
        m = _plain(_Gen(seed), n).cpu().numpy()
        return m, np.zeros(n, np.uint8)
    if op != "encrypt" or n > 100:
        return None
    gen = _Gen(seed)
    m, r = _plain(gen, n).cpu().tolist(), _to_ints(gen.r(n, bits // 64).cpu().numpy())
    num, h_s, _, _ = _numbers(bits)
    n2 = num * num
    rows = [pow(h_s, e, n2) * (1 + v * num) * pow(2, 2 * bits, n2) % n2 for v, e in zip(m, r)]
    out = np.frombuffer(b"".join(v.to_bytes(bits // 4, "little") for v in rows), dtype=np.int32).reshape(n, -1)
    return out.copy()
