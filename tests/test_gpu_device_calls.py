"""What a device call asks of its caller besides its values: the alignment of
its arrays."""

import ctypes

import numpy as np
import pytest
import torch

from heu_gb300 import capi

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
