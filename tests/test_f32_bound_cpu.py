"""The bound that the tests of the float32 products use: numpy's float32 sums meet it, operands with the 10 bits of mantissa of a
reduced-precision tensor-core mode do not."""

import numpy as np
import pytest

import test_f32_kernels_gpu as products


def ten_bits(x):
    """float32 numbers rounded to 10 bits of mantissa."""
    bits = x.view(np.uint32).astype(np.uint64)
    return ((bits + 0xFFF + ((bits >> 13) & 1)) & ~np.uint64(0x1FFF)).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("M,N,K", [(16, 257, 768), (8, 5, 3076), (3, 48, 1024), (64, 64, 48), (128, 128, 16), (1, 17, 132)])
def test_bound(M, N, K):
    g = np.random.default_rng(M + N + K)
    a, w = g.standard_normal((M, K)).astype(np.float32), (g.standard_normal((N, K)) / K ** 0.5).astype(np.float32)
    want = a.astype(np.float64) @ w.astype(np.float64).T
    limit = products.bound(K) * max(1.0, np.abs(want).max())
    one_by_one = np.zeros((M, N), dtype=np.float32)
    for k in range(K):
        one_by_one += a[:, k:k + 1] * w[:, k][None]
    assert np.abs(one_by_one - want).max() < limit
    reduced = ten_bits(a).astype(np.float64) @ ten_bits(w).astype(np.float64).T
    assert np.abs(reduced - want).max() > 2 * limit
