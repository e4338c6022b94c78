"""The Montgomery core at the edges of its carries: operands of all-ones and
all-zero limbs, 0, 1 and the modulus less one, for ordinary keys and for keys
whose primes (and so n and n^2) have nothing but ones in their top limbs."""

import pytest

import heu_gb300 as hg

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
