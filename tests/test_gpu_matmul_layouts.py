"""MatMul at the numbers of outputs and of bases where its kernels take another
layout (lanes a chain of the planes; the narrow layouts of the product tree's
large levels, from 2,432 nodes on)."""

import numpy as np
import pytest

import heu_gb300 as hg

pytestmark = pytest.mark.gpu

# the two largest primes below 2^(bits / 2), by their distance from it
DENSE = {1024: (569, 629), 2048: (105, 179), 3072: (3453, 4977)}


# M x K bases (odd, and above 2 * 2,432 but for the first) and M x N outputs on
# both sides of each change of layout
@pytest.mark.parametrize("M,K,N,lo,hi", [
    (433, 9, 3, 0, 2 ** 9),  # 1,299 outputs
    (667, 9, 3, -(2 ** 6), 2 ** 6),  # 2,001
    (1001, 7, 4, 0, 4),  # 4,004
    (2731, 3, 3, -9, 9),  # 8,193
    (6001, 1, 2, 0, 2 ** 3),  # 12,002
])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bits", [1024, 2048, 3072])
def test_matmul_in_every_layout(gpu_ctx, gpu_key, bits, dense, M, K, N, lo, hi):
    """An output does not depend on how many there are: the first, middle and
    last rows byte for byte as calls of a few rows give them, and single
    outputs as Python integers do."""
    if dense:
        p, q = (2 ** (bits // 2) - t for t in DENSE[bits])
        n = p * q
        h_s = pow(n - 9, n, n * n)
        key = gpu_ctx.load_key(bits, n, h_s, table_window=5)
    else:
        key, pk, _ = gpu_key(bits, {1024: 1, 2048: 0, 3072: 2}[bits])
        n = pk.n
    n2, S = n * n, key.ct_limbs
    rng = np.random.default_rng(M + bits)
    m = rng.integers(-(2 ** 63), 2 ** 63 - 1, M * K)
    r = rng.integers(0, 2 ** 32, (M * K, key.r_limbs), dtype=np.uint32)
    x = key.encrypt(m, r).reshape(M, K, S)
    y = rng.integers(lo, hi, (K, N))
    y[0, 0] = lo
    got = key.matmul(x, y)
    assert got.shape == (M, N, S)
    for first in (0, M // 2, M - 7):
        few = key.matmul(np.ascontiguousarray(x[first:first + 7]), y)
        assert np.array_equal(got[first:first + 7], few), first
    rinv = pow(2, -32 * S, n2)
    for i, j in ((0, 0), (M // 3, N - 1), (M - 1, N // 2), (M - 1, N - 1)):
        want = 1
        for k in range(K):
            want = want * pow(hg.limbs_to_ints(x[i, k])[0] * rinv % n2, int(y[k, j]), n2) % n2
        assert hg.limbs_to_ints(got[i, j])[0] * rinv % n2 == want, (i, j)
    if dense:
        key.free()
