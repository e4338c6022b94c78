"""What a device call asks of its caller besides its values: the alignment of
its arrays, that calls of other threads and keys leave it alone, and what its
stream allocates."""

import ctypes
import threading

import numpy as np
import pytest
import torch

from heu_gb300 import autotune, capi

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _column(key, rng, count, dev):
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    r = rng.integers(0, 2 ** 32, (count, key.r_limbs), dtype=np.uint32)
    return m, torch.from_numpy(m).to(dev), torch.from_numpy(r.view(np.int32)).to(dev)


def _at_eight(count, limbs, dev):
    """A column of ciphertexts that starts 8 bytes past a 16-byte boundary."""
    buf = torch.zeros(count * limbs + 2, dtype=torch.int32, device=dev)
    assert buf.data_ptr() % 16 == 0
    return buf, buf[2:].view(count, limbs)


@pytest.mark.parametrize("bits,seed", [(1024, 1), (3072, 2)])
def test_few_ciphertexts_at_eight_byte_alignment(gpu_ctx, gpu_key, bits, seed):
    """Up to 12 ciphertexts a multiprocessor, encryption, re-randomization and
    decryption of these key sizes take columns of 8-byte alignment."""
    dev = torch.device("cuda", 0)
    key, _, _ = gpu_key(bits, seed)
    lib, h = key.lib, key.ctx.handle
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(bits)
    for count in (1, 5, sms, sms + 1, 12 * sms):
        m, dm, dr = _column(key, rng, count, dev)
        want = torch.empty((count, key.ct_limbs), dtype=torch.int32, device=dev)
        held, odd = _at_eight(count, key.ct_limbs, dev)
        out, ovf = torch.empty(count, dtype=torch.int64, device=dev), torch.empty(count, dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()
        capi.check(lib.hg_dev_encrypt(h, key.id, _p(dm), _p(dr), _p(want), count, None))
        capi.check(lib.hg_dev_encrypt(h, key.id, _p(dm), _p(dr), _p(odd), count, None))
        capi.check(lib.hg_dev_check(h))
        assert torch.equal(odd, want), count
        capi.check(lib.hg_dev_randomize(h, key.id, _p(want), _p(dr), count, None))
        capi.check(lib.hg_dev_randomize(h, key.id, _p(odd), _p(dr), count, None))
        capi.check(lib.hg_dev_decrypt(h, key.id, _p(odd), _p(out), _p(ovf), count, None))
        capi.check(lib.hg_dev_check(h))
        assert torch.equal(odd, want), count
        assert np.array_equal(out.cpu().numpy(), m) and not ovf.any(), count
        assert not held[:2].any()


def test_few_decryptions_of_two_keys_from_many_threads(gpu_ctx, gpu_key):
    """Two 3072-bit keys with the widest window, whose exponent programs differ
    in length and so in the shared memory that a launch for few ciphertexts asks
    for: calls of one do not take the other's limit away."""
    bits = 3072
    p, q = 2 ** (bits // 2) - 3453, 2 ** (bits // 2) - 4977  # exponents of ones: the longest programs
    n = p * q
    dense = gpu_ctx.load_key(bits, n, pow(n - 9, n, n * n), p, q, table_window=5)
    plain, _, _ = gpu_key(bits, 2)
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(1)
    saved = autotune.get_config(plain)
    work, failed = [], []
    try:
        for key in (dense, plain):
            autotune.set_config(key, dict(autotune.get_config(key), dec_window=7))
            m, dm, dr = _column(key, rng, 1, dev)
            ct = torch.empty((1, key.ct_limbs), dtype=torch.int32, device=dev)
            torch.cuda.synchronize()
            capi.check(key.lib.hg_dev_encrypt(key.ctx.handle, key.id, _p(dm), _p(dr), _p(ct), 1, None))
            capi.check(key.lib.hg_dev_check(key.ctx.handle))
            for _ in range(4):
                work.append((key, m[0], ct, torch.zeros(1, dtype=torch.int64, device=dev),
                             torch.zeros(1, dtype=torch.uint8, device=dev), torch.cuda.Stream()))
        torch.cuda.synchronize()

        def calls(key, m, ct, out, ovf, stream):
            s = ctypes.c_void_p(stream.cuda_stream)
            for _ in range(300):
                if key.lib.hg_dev_decrypt(key.ctx.handle, key.id, _p(ct), _p(out), _p(ovf), 1, s):
                    failed.append(key.lib.hg_last_error())

        threads = [threading.Thread(target=calls, args=w) for w in work]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not failed, (len(failed), failed[0])
        assert all(int(out) == m for _, m, _, out, _, _ in work)
    finally:
        autotune.set_config(plain, saved)
        dense.free()


def _held(lib):
    held = ctypes.c_size_t()
    capi.check(lib.hg_probe_set_alloc_limit(0, ctypes.byref(held)))
    return held.value


@pytest.mark.parametrize("bits,seed", [(1024, 1), (2048, 0), (3072, 2)])
def test_scratch_does_not_follow_the_length_of_the_calls(gpu_key, bits, seed):
    """A stream allocates for decryptions (and all but the inverse's tree for
    Muls) twice at most, once for short and once for any longer calls, and frees
    nothing: a long call may be captured after a short one, and what was captured
    before a longer call stays valid."""
    dev = torch.device("cuda", 0)
    key, _, _ = gpu_key(bits, seed)
    lib, h = key.lib, key.ctx.handle
    count = 30000 if bits < 3072 else 6000
    rng = np.random.default_rng(bits)
    m, dm, dr = _column(key, rng, count, dev)
    ct = torch.empty((count, key.ct_limbs), dtype=torch.int32, device=dev)
    prod, ones = torch.empty_like(ct), torch.ones(count, dtype=torch.int64, device=dev)
    out, ovf = torch.zeros(count, dtype=torch.int64, device=dev), torch.empty(count, dtype=torch.uint8, device=dev)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    capi.check(lib.hg_dev_encrypt(h, key.id, _p(dm), _p(dr), _p(ct), count, None))
    torch.cuda.synchronize()

    def decrypt(n, stream):
        s = ctypes.c_void_p(stream.cuda_stream)
        capi.check(lib.hg_dev_decrypt(h, key.id, _p(ct), _p(out), _p(ovf), n, s))

    def mul(n, stream):
        s = ctypes.c_void_p(stream.cuda_stream)
        capi.check(lib.hg_dev_mul(h, key.id, _p(ct), _p(ones), _p(prod), n, s))

    decrypt(1, streams[0])
    base = _held(lib)
    for n in (2, 3, 7):
        decrypt(n, streams[0])
        assert _held(lib) == base, n
    decrypt(2500, streams[0])
    base = _held(lib)
    for n in (5, 700, 3000, count // 2, count):
        decrypt(n, streams[0])
        assert _held(lib) == base, n
    mul(2500, streams[1])
    base = _held(lib)
    mul(count, streams[1])
    tree = (2 * count + 64) * key.ct_limbs * 4
    assert base <= _held(lib) <= base + tree
    torch.cuda.synchronize()
    assert torch.equal(prod, ct)
    # a stream that has seen one short call; the short graph runs after the long one
    decrypt(1, streams[2])
    graphs = []
    for n in (5, count):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[2]):
            decrypt(n, streams[2])
        graphs.append((n, g))
    for n, g in graphs[::-1]:
        out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out[:n].cpu().numpy(), m[:n]) and not out[n:].any()


@pytest.mark.parametrize("bits,seed", [(1024, 1), (2048, 0), (3072, 2)])
def test_the_tuner_chooses_windows_alone(gpu_key, bits, seed):
    """Layouts follow the number of elements of each call, so one length's timing
    must not take a layout away from the others: a key's layout variants are what
    they were before."""
    key, _, _ = gpu_key(bits, seed)
    saved = autotune.get_config(key)
    try:
        for calib in (64, 300, 1000, 3000):
            for variant in (0, 1):
                autotune.set_config(key, dict(saved, variant=variant, dec_variant=variant))
                cfg, rates = autotune.tune(key, calib=calib)
                assert cfg["variant"] == variant and cfg["dec_variant"] == variant, calib
                assert all(v > 0 for v in rates.values())
    finally:
        autotune.set_config(key, saved)
