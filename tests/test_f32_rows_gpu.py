"""float32 products of at most 16 rows (csrc/gemm_simt.cu) on both sides of the rules that choose their form."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M", [1, 2, 3, 5, 9, 16])
@pytest.mark.parametrize("N", [592, 594, 1184, 1186, 4739])
@pytest.mark.parametrize("K", [768, 772, 1024, 1028, 2052, 4096, 4100])
def test_forms_have_the_same_sums(M, N, K):
    """One CTA a group of columns or CTAs that walk over the groups, any number of steps on their way together: the bits are those of a
    product of a few columns, with every epilogue, and nothing beside the result is written."""
    from test_f32_kernels_gpu import bound, ops_for, product, size_of

    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a, w, vector, base = (torch.randn(shape, generator=g).to(DEV) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    few = torch.empty(M, 60, device=DEV)
    ops.linear_f32_rows(a, w[N - 60:], None, few)
    for accumulate, act in ((0, None), (1, "gelu_tanh"), (3, None)):
        room = torch.full((M + 1, N + 4), 7.0, device=DEV)
        room[:M, :N] = base if accumulate & 1 else 7.0
        ops.linear_f32_rows(a, w, vector if accumulate else None, room[:M, :N], act=act, accumulate=accumulate)
        assert bool((room[M:] == 7.0).all()) and bool((room[:, N:] == 7.0).all())
        want = product(a, w, vector if accumulate == 1 else None, act, vector if accumulate == 3 else None, base if accumulate else None)
        assert float((room[:M, :N].double() - want).abs().max()) < bound(K) * size_of(want), accumulate
        if not accumulate:
            assert torch.equal(room[:M, N - 60:N], few)
