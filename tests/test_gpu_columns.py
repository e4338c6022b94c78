"""The Montgomery core at the edges of its carries: operands of all-ones and
all-zero limbs, 0, 1 and the modulus less one, for ordinary keys and for keys
whose primes (and so n and n^2) have nothing but ones in their top limbs."""

import numpy as np
import pytest
import torch

import heu_gb300 as hg
from heu_gb300 import autotune

pytestmark = pytest.mark.gpu

# the two largest primes below 2^(bits / 2), by their distance from it
DENSE = {1024: (569, 629), 2048: (105, 179), 3072: (3453, 4977)}


@pytest.fixture(scope="module")
def edge_key(gpu_ctx, gpu_key):
    made = {}

    def get(bits, dense):
        if not dense:
            key, pk, sk = gpu_key(bits, {1024: 1, 2048: 0, 3072: 2}[bits])
            return key, pk.n, pk.h_s, sk.p, sk.q
        if bits not in made:
            p, q = (2 ** (bits // 2) - t for t in DENSE[bits])
            n = p * q
            h_s = pow(n - 9, n, n * n)
            made[bits] = (gpu_ctx.load_key(bits, n, h_s, p, q, table_window=5), n, h_s, p, q)
        return made[bits]

    return get


def edge_values(n2, limbs):
    ones = 2 ** (32 * limbs) - 1
    every_other = sum(0xFFFFFFFF << (64 * i) for i in range(limbs // 2))
    low, high = 2 ** (16 * limbs) - 1, ones - (2 ** (16 * limbs) - 1)
    vals = [0, 1, 2, n2 - 1, n2 - 2, n2 // 2, ones % n2, every_other % n2, (ones - every_other) % n2, low, high % n2,
            2 ** (32 * limbs - 1) % n2, n2 - low]
    return [v for v in vals if v < n2]


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_products_at_carry_edges(edge_key, bits, dense):
    key, n, _, _, _ = edge_key(bits, dense)
    n2, S = n * n, key.ct_limbs
    vals = edge_values(n2, S)
    a = [x for x in vals for _ in vals]
    b = vals * len(vals)
    rinv = pow(2, -32 * S, n2)
    la, lb = hg.ints_to_limbs(a, S), hg.ints_to_limbs(b, S)
    assert hg.limbs_to_ints(key.add(la, lb)) == [x * y * rinv % n2 for x, y in zip(a, b)]
    assert hg.limbs_to_ints(key.from_mont(la)) == [x * rinv % n2 for x in a]
    assert hg.limbs_to_ints(key.to_mont(la)) == [x * pow(2, 32 * S, n2) % n2 for x in a]
    # the products of a sum's tree: everything but the zeros
    c = [x for x in a if x] + [n2 - 1]
    prod = c[0]
    for x in c[1:]:
        prod = prod * x * rinv % n2
    assert hg.limbs_to_ints(key.sum(hg.ints_to_limbs(c, S))) == [prod]


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_decrypt_in_every_layout(edge_key, bits, dense):
    """Lengths on both sides of the points where the decryption takes another
    layout (lanes per chain), ragged against the ciphertexts of a warp."""
    key, n, _, _, _ = edge_key(bits, dense)
    rng = np.random.default_rng(bits + dense)
    count = 11001 if bits < 3072 else 5003
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    m[:4] = [0, -1, 2 ** 63 - 1, -(2 ** 63)]
    r = rng.integers(0, 2 ** 32, (count, key.r_limbs), dtype=np.uint32)
    ct = key.encrypt(m, r)
    cfg = autotune.get_config(key)
    for variant in (0, 1):
        autotune.set_config(key, dict(cfg, dec_variant=variant))
        for length in (1, 2, 15, 17, 33, 500, 1000, 1601, 3001, count):
            got, ovf = key.decrypt(ct[:length])
            assert np.array_equal(got, m[:length]) and not ovf.any(), (variant, length)
    for window in (2, 7):
        autotune.set_config(key, dict(cfg, dec_window=window))
        assert np.array_equal(key.decrypt(ct[:33])[0], m[:33]), window
    autotune.set_config(key, cfg)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_decrypt_full_range_and_non_units(edge_key, bits, dense):
    """Plaintexts up to +-n/2, and numbers that share a prime with n (never a
    ciphertext): L(0) is taken as (2^(32 H) - 1) / p mod 2^(32 H)."""
    key, n, h_s, p, q = edge_key(bits, dense)
    n2, S, H = n * n, key.ct_limbs, key.ct_limbs // 4
    R = 2 ** (32 * S)
    ms = [n // 2, -(n // 2), n // 2 - 1, 1 - n // 2, 2 ** (bits // 2), 1, 0, -1]
    zs = [pow(h_s, 12345 + i, n2) * (1 + m * n) % n2 for i, m in enumerate(ms)]
    assert key.decrypt_bn(hg.ints_to_limbs([z * R % n2 for z in zs], S)) == ms

    def side(c, pr):
        y = pow(c, pr - 1, pr * pr)
        hv = pow((pow(n + 1, pr - 1, pr * pr) - 1) // pr, -1, pr)
        lv = ((y - 1) % 2 ** (32 * H)) * pow(pr, -1, 2 ** (32 * H)) % 2 ** (32 * H)
        return lv * hv % pr

    odd = [0, p, q, p * p, 5 * q * q, p * q, 7 * p]
    want = []
    for c in odd:
        mp, mq = side(c, p), side(c, q)
        m = mp + p * ((mq - mp) * pow(p, -1, q) % q)
        want.append(m - n if m > n // 2 else m)
    assert key.decrypt_bn(hg.ints_to_limbs([c * R % n2 for c in odd], S)) == want


def _randomness(key, rng, count):
    r = rng.integers(0, 2 ** 32, (count, key.r_limbs), dtype=np.uint32)
    r[0], r[1], r[2] = 0, 2 ** 32 - 1, 0
    r[2, 0] = 1
    r[3, :-1] = 0
    return r


@pytest.mark.parametrize("window", [1, 5, 8, 13])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_encrypt_modes(gpu_ctx, edge_key, bits, dense, window):
    """Encrypt, EncryptZero and Randomize byte for byte, over plaintexts up to
    +-n/2 and randomness with zero, full and single digits."""
    if window == 13 and bits != 2048:
        pytest.skip("one wide window is enough")
    _, n, h_s, _, _ = edge_key(bits, dense)
    key = gpu_ctx.load_key(bits, n, h_s, table_window=window)
    n2, S = n * n, key.ct_limbs
    R = pow(2, 32 * S, n2)
    rng = np.random.default_rng(window)
    ms = [0, 1, -1, 2 ** 63 - 1, -(2 ** 63), n // 2, -(n // 2), 12345]
    r = _randomness(key, rng, len(ms))
    hr = [pow(h_s, v, n2) for v in hg.limbs_to_ints(r)]
    want = [(1 + m * n) * h % n2 * R % n2 for m, h in zip(ms, hr)]
    assert hg.limbs_to_ints(key.encrypt_bn(ms, r)) == want
    assert hg.limbs_to_ints(key.encrypt(np.array(ms[:5]), r[:5])) == want[:5]
    assert hg.limbs_to_ints(key.encrypt_zero(r)) == [h * R % n2 for h in hr]
    edges = edge_values(n2, S)[:len(ms)]
    got = key.randomize(hg.ints_to_limbs(edges, S), r)
    assert hg.limbs_to_ints(got) == [c * h % n2 for c, h in zip(edges, hr)]
    with pytest.raises(hg.HgError):
        key.encrypt_bn([n // 2 + 1], r[:1])
    with pytest.raises(hg.HgError):
        key.randomize(hg.ints_to_limbs([n2], S), r[:1])
    key.free()


@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_encrypt_in_every_layout(edge_key, bits):
    """A ciphertext does not depend on how many are encrypted with it: lengths
    on both sides of the points where another layout runs."""
    key, n, h_s, _, _ = edge_key(bits, True)
    n2 = n * n
    rng = np.random.default_rng(bits)
    count = 21001
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    r = _randomness(key, rng, count)
    ct = key.encrypt(m, r)
    for i in (0, 1, 2, 3, 77, count - 1):
        v = hg.limbs_to_ints(r[i])[0]
        assert hg.limbs_to_ints(ct[i])[0] == pow(h_s, v, n2) * (1 + int(m[i]) * n) * pow(2, 2 * bits, n2) % n2
    cfg = autotune.get_config(key)
    for variant in (0, 1):
        autotune.set_config(key, dict(cfg, variant=variant))
        for length in (1, 3, 304, 305, 608, 609, 1217, 2500, 5001, 9729):
            assert np.array_equal(key.encrypt(m[:length], r[:length]), ct[:length]), (variant, length)
            assert np.array_equal(key.encrypt(m[-length:], r[-length:]), ct[-length:]), (variant, length)
    autotune.set_config(key, cfg)


def test_encrypt_with_a_base_that_is_no_unit(gpu_ctx, edge_key):
    """h_s sharing a factor with n (never a key's) still encrypts by definition."""
    _, n, h_s, p, q = edge_key(1024, False)
    n2 = n * n
    key = gpu_ctx.load_key(1024, n, h_s * p % n2, p, q, table_window=6)
    r = _randomness(key, np.random.default_rng(0), 6)
    ms = [0, 1, -1, 77, -5, 2 ** 40]
    want = [pow(h_s * p, v, n2) * (1 + m * n) * pow(2, 2048, n2) % n2 for m, v in zip(ms, hg.limbs_to_ints(r))]
    assert hg.limbs_to_ints(key.encrypt(np.array(ms), r)) == want
    key.free()


def _scalars(rng, count):
    k = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    k[: min(count, 14)] = [0, 1, -1, 2, -2, 2 ** 63 - 1, -(2 ** 63), 15, 16, 17, -16, 2 ** 32, 2 ** 60, -3][:count]
    return k


@pytest.mark.parametrize("window", [2, 4, 6])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_mul_windows(edge_key, bits, dense, window):
    """Scalars of every length (a warp's windows follow its longest) on edge
    ciphertexts, byte for byte; 15 of them leave a ragged warp and an odd node
    on every level of the inverse's tree."""
    key, n, h_s, _, _ = edge_key(bits, dense)
    n2, S = n * n, key.ct_limbs
    R = pow(2, 32 * S, n2)
    rng = np.random.default_rng(window)
    k = _scalars(rng, 15)
    units = [pow(h_s, 3 + i, n2) * R % n2 for i in range(len(k) - 4)] + [1, 2, n2 - 1, n2 - 2]
    cfg = autotune.get_config(key)
    autotune.set_config(key, dict(cfg, mul_window=window))
    got = hg.limbs_to_ints(key.mul(hg.ints_to_limbs(units, S), k))
    small = hg.limbs_to_ints(key.mul(hg.ints_to_limbs(units, S), k % 5))
    autotune.set_config(key, cfg)
    rinv = pow(R, -1, n2)
    assert got == [pow(c * rinv % n2, int(e), n2) * R % n2 for c, e in zip(units, k)]
    assert small == [pow(c * rinv % n2, int(e), n2) * R % n2 for c, e in zip(units, k % 5)]
    # numbers that are no units, and no ciphertexts at all
    none = [v for v in edge_values(n2, S)]
    pos = np.abs(k[: len(none)] // 2)
    assert hg.limbs_to_ints(key.mul(hg.ints_to_limbs(none, S), pos)) == [
        pow(c * rinv % n2, int(e), n2) * R % n2 for c, e in zip(none, pos)]
    with pytest.raises(hg.HgError):
        key.mul(hg.ints_to_limbs([n2], S), [3])


@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_mul_in_every_layout(edge_key, bits):
    """A product does not depend on how many there are: lengths on both sides
    of the points where another layout runs, with signed scalars (every length
    another inverse tree)."""
    key, n, h_s, _, _ = edge_key(bits, False)
    n2, S = n * n, key.ct_limbs
    R = pow(2, 32 * S, n2)
    rinv = pow(R, -1, n2)
    rng = np.random.default_rng(bits)
    count = 10007
    k = _scalars(rng, count)
    ct = key.encrypt(rng.integers(-(2 ** 40), 2 ** 40, count), _randomness(key, rng, count))
    whole = key.mul(ct, k)
    for i in (0, 6, 7, 20, 5000, count - 1):
        c = hg.limbs_to_ints(ct[i])[0] * rinv % n2
        assert hg.limbs_to_ints(whole[i])[0] == pow(c, int(k[i]), n2) * R % n2
    cfg = autotune.get_config(key)
    for variant in (0, 1):
        autotune.set_config(key, dict(cfg, variant=variant))
        for length in (1, 2, 3, 9, 301, 609, 1217, 2433, 4865, count):
            assert np.array_equal(key.mul(ct[:length], k[:length]), whole[:length]), (variant, length)
    autotune.set_config(key, cfg)


@pytest.mark.parametrize("M,K,N,lo,hi", [
    (1, 1, 1, 0, 2),  # one bit plane, one chunk
    (2, 3, 1, -4, 4),
    (3, 9, 2, 0, 1),  # all exponents 0
    (1, 17, 24, -(2 ** 15), 2 ** 15),  # wide chunks, a ragged last one
    (2, 5, 3, -(2 ** 63), 2 ** 63 - 1),  # 64 planes: the sum is taken below n on the way
    (70, 2, 2, 0, 2 ** 20),  # no offset
])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_matmul_shapes(edge_key, bits, dense, M, K, N, lo, hi):
    key, n, h_s, _, _ = edge_key(bits, dense)
    n2, S = n * n, key.ct_limbs
    R = pow(2, 32 * S, n2)
    rng = np.random.default_rng(M * 100 + K)
    x = [pow(h_s, 5 + i, n2) * (1 + i * n) % n2 for i in range(M * K)]
    if K > 2:
        x[1], x[2] = 1, n2 - 1
    y = rng.integers(lo, hi, (K, N))
    y[0, 0] = lo
    got = key.matmul(hg.ints_to_limbs([v * R % n2 for v in x], S).reshape(M, K, S), y)
    for i in range(0, M, max(1, M // 3)):
        for j in range(N):
            want = 1
            for k in range(K):
                want = want * pow(x[i * K + k], int(y[k, j]), n2) % n2
            assert hg.limbs_to_ints(got[i, j])[0] == want * R % n2, (i, j)


@pytest.mark.parametrize("bits", [1024, 2048])
def test_matmul_with_bases_that_are_no_units(edge_key, bits):
    """Zero and multiples of a prime have no inverse modulo n; their powers are
    still defined for exponents >= 0, and an exponent below 0 is an error."""
    key, n, h_s, p, q = edge_key(bits, False)
    n2, S = n * n, key.ct_limbs
    R = pow(2, 32 * S, n2)
    x = [0, p, 7 * q, pow(h_s, 3, n2), n, 1]
    y = np.array([[0, 1], [3, 0], [0, 2], [5, 9], [1, 0], [2, 3]])
    limbs = hg.ints_to_limbs([v * R % n2 for v in x], S).reshape(1, 6, S)
    got = hg.limbs_to_ints(key.matmul(limbs, y).reshape(2, S))
    for j in range(2):
        want = 1
        for v, e in zip(x, y[:, j]):
            want = want * pow(v, int(e), n2) % n2
        assert got[j] == want * R % n2
    with pytest.raises(hg.HgError):
        key.matmul(limbs, -y)
    with pytest.raises(hg.HgError):
        key.matmul(hg.ints_to_limbs([n2] * 6, S).reshape(1, 6, S), y)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_decrypt_few_and_many_agree(edge_key, bits, dense):
    """Lengths on both sides of the one from which decryption no longer takes a
    block per ciphertext and prime, with ciphertexts that are multiples of a
    prime or not below n^2."""
    key, n, _, p, _ = edge_key(bits, dense)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3 * bits + dense)
    count = 4 * sms + 1
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    r = rng.integers(0, 2 ** 32, (count, key.r_limbs), dtype=np.uint32)
    ct = key.encrypt(m, r)
    ct[0] = hg.ints_to_limbs([p * 12345], ct.shape[1])[0]
    ct[1] = hg.ints_to_limbs([1], ct.shape[1])[0]
    ct[2] = hg.ints_to_limbs([n * n - 1], ct.shape[1])[0]
    want, want_ovf = key.decrypt(ct)
    assert np.array_equal(want[3:], m[3:]) and not want_ovf[3:].any()
    for length in (1, 2, 3, sms // 2 + 1, sms, sms + 1):
        got, ovf = key.decrypt(ct[:length])
        assert np.array_equal(got, want[:length]) and np.array_equal(ovf, want_ovf[:length]), length
    ct[0] = hg.ints_to_limbs([n * n], ct.shape[1])[0]
    for length in (1, sms + 1):
        with pytest.raises(hg.HgError):
            key.decrypt(ct[:length])


@pytest.mark.parametrize("window", [5, 12])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_encrypt_few_and_many_agree(gpu_ctx, edge_key, bits, window):
    """Lengths on both sides of those from which an encryption is shared by
    fewer blocks, against the same values in a longer call."""
    _, n, h_s, p, q = edge_key(bits, True)
    key = gpu_ctx.load_key(bits, n, h_s, p, q, table_window=window)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(bits + window)
    count = 16 * sms + 1
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, count)
    r = _randomness(key, rng, count)
    ct, zero = key.encrypt(m, r), key.encrypt_zero(r)
    again = key.randomize(ct, r[::-1].copy())
    for length in (1, 2, sms // 4, sms // 4 + 1, sms // 2, sms // 2 + 1, 2 * sms, 2 * sms + 1):
        assert np.array_equal(key.encrypt(m[:length], r[:length]), ct[:length]), length
        assert np.array_equal(key.encrypt_zero(r[-length:]), zero[-length:]), length
        assert np.array_equal(key.randomize(ct[:length], r[::-1][:length].copy()), again[:length]), length
    key.free()
