"""The tcgen05 product on pairs of CTAs (256 rows a tile) against 64 bits and against the one-CTA tiles."""

from types import SimpleNamespace

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


@pytest.mark.parametrize("M", [1, 128, 129, 256, 300, 513])
@pytest.mark.parametrize("heads,kv_heads,head_dim,K", [(4, 4, 64, 64), (8, 2, 16, 200), (3, 1, 128, 1032), (5, 5, 64, 320)])
def test_keys_and_values_into_the_pages(M, heads, kv_heads, head_dim, K):
    """The q|k|v product on pairs: queries to the output, keys and values to pages in no order, of several requests, one position of them
    without a page; a pair's second CTA may have no rows.  The bits of one-CTA tiles, and the sums of 64 bits."""
    from pagedserve_b200.kernels.ops import Ops

    page, q_width, kv_width = 16, heads * head_dim, kv_heads * head_dim
    N = q_width + 2 * kv_width
    ops, (a, w, bias, _) = Ops(torch.bfloat16), operands(M, N, K)
    g = torch.Generator().manual_seed(M)
    per = -(-M // page) + 1
    table = torch.randperm(2 * per, generator=g).view(2, per).to(torch.int32)
    table[1, 0] = -1
    row = (torch.arange(M) % 3 == 2).to(torch.int32)                   # every third token belongs to the second request
    positions = torch.empty(M, dtype=torch.int32)
    for r in (0, 1):
        positions[row == r] = torch.arange(int((row == r).sum()), dtype=torch.int32)
    ctx = SimpleNamespace(token_slot=row.to(DEV), positions=positions.to(DEV))
    outs, pools = [], []
    for bn in (512, 128):
        pool = torch.full((2 * per, 2, kv_heads, page, head_dim), 7.0, dtype=torch.bfloat16, device=DEV)
        layer = SimpleNamespace(k_pool=pool[:, 0], v_pool=pool[:, 1], page_stride=pool.stride(0), page_size=page, block_table=table.to(DEV))
        out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.linear_tc_qkv(a, w, bias, out, ctx, layer, q_width, kv_width, head_dim, bn=bn)
        outs.append(out)
        pools.append(pool)
    assert torch.equal(outs[0], outs[1]) and torch.equal(pools[0], pools[1])
    want = a.double() @ w.double().T + bias
    tol = 6e-3 * float(want.abs().max())
    assert float((outs[0][:, :q_width].double() - want[:, :q_width]).abs().max()) < tol
    assert bool((outs[0][:, q_width:] == 7.0).all())
    pages = table[row.long(), positions.long() // page].long()
    kept = pages >= 0
    got = pools[0][pages[kept].to(DEV), :, :, (positions[kept].long() % page).to(DEV)]                     # [tokens, 2, kv_heads, head_dim]
    assert float((got.reshape(-1, 2 * kv_width).double() - want[kept.to(DEV), q_width:]).abs().max()) < tol
    written = torch.zeros(2 * per, page, dtype=torch.bool)
    written[pages[kept], positions[kept].long() % page] = True
    assert bool((pools[0].permute(0, 3, 1, 2, 4)[~written.to(DEV)] == 7.0).all())
    assert int(ops.status_flag(DEV).item()) == 0
