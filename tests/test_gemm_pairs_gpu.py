"""The tcgen05 product on pairs of CTAs (256 rows a tile) against 64 bits and against the one-CTA tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def operands(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    return a, w, torch.randn(N, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (65, 64, 64), (128, 256, 64), (129, 264, 136), (256, 256, 64), (257, 1003, 96), (385, 520, 328),
                                   (1024, 2304, 768), (511, 770, 3072), (2600, 2600, 136)])
def test_pairs(M, N, K):
    from pagedserve_b200.kernels.ops import Ops

    ops, (a, w, bias, base) = Ops(torch.bfloat16), operands(M, N, K)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = a.double() @ w.double().T
    # float32 sums in another order than 64 bits has them; bfloat16 results round at 2^-9
    for out_dtype, vector, accumulate, tol in ((torch.float32, bias, 0, 2e-5), (torch.float32, None, 1, 2e-5), (torch.bfloat16, bias, 0, 6e-3),
                                               (torch.float32, bias, 3, 2e-5)):
        expect = want if vector is None else want * vector if accumulate & 2 else want + vector
        expect = expect + base if accumulate & 1 else expect
        outs = []
        for width in (512, 128):
            out = base.clone().to(out_dtype)
            ops.linear_tc(a, w, vector, out, accumulate=accumulate, status=status, bn=width)
            assert float((out.double() - expect).abs().max()) < tol * float(expect.abs().max()), (out_dtype, accumulate, width)
            outs.append(out)
        assert torch.equal(outs[0], outs[1])                    # the same sums in the same order
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,N,K", [(3000, 1000, 64), (2048, 2304, 768), (4099, 2048, 1032), (2500, 1288, 1032), (5000, 640, 1096)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_chosen_tiles(M, N, K, out_dtype):
    """Shapes for which the rule takes tiles of 128, 192 and 256 columns and pairs: the sums of 128-wide tiles."""
    from pagedserve_b200.kernels.ops import Ops

    ops, (a, w, _, _) = Ops(torch.bfloat16), operands(M, N, K)
    chosen, plain = (torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV) for _ in range(2))
    ops.linear_tc(a, w, None, chosen, act="gelu_tanh")
    ops.linear_tc(a, w, None, plain, act="gelu_tanh", bn=128)
    assert torch.equal(chosen, plain) and int(ops.status_flag(DEV).item()) == 0
