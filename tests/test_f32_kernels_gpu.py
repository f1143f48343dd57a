"""The float32 kernels of csrc/gemm_simt.cu and csrc/attention_f32.cu against 64 bits, at the edges of their tiles, and against
the general kernels whose calls they take over."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops_for():
    from pagedserve_b200.kernels.ops import Ops

    return Ops(torch.float32)


def product(a, w, bias, act, factor, base):
    y = a.double() @ w.double().T
    if factor is not None:
        y = y * factor.double()
    if bias is not None:
        y = y + bias.double()
    if act == "gelu_tanh":
        y = torch.nn.functional.gelu(y, approximate="tanh")
    return y if base is None else y + base.double()


# float32 sums of K products of numbers of order one over sqrt(K): each addition rounds by at most 2^-24 of a partial sum that
# is of the size of the result; K + 40 of them in a row is the longest chain
def sum_bound(K):
    return (K + 40) * 2.0 ** -24


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(1, 4), (3, 128), (17, 132), (48, 1024), (30, 1028), (5, 3076), (257, 768)])
def test_few_rows(M, N, K):
    ops, g = ops_for(), torch.Generator().manual_seed(M * 1000 + N + K)
    a, w, bias, base = (torch.randn(shape, generator=g) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    a_d, w_d, bias_d = a.to(DEV), w.to(DEV), bias.to(DEV)
    for act, how in ((None, "store"), ("gelu_tanh", "store"), (None, "add"), (None, "factor")):
        out = base.clone().to(DEV)
        ops.linear_f32_rows(a_d, w_d, bias_d, out, act=act, accumulate={"store": 0, "add": 1, "factor": 3}[how])
        want = product(a, w, None if how == "factor" else bias, act, bias if how == "factor" else None,
                       None if how == "store" else base)
        assert float((out.cpu().double() - want).abs().max()) < sum_bound(K) * 8 * float(want.abs().max()), (act, how)
    # a row alone and a row among others, rows that lie apart
    wide = torch.randn(M, K + 8, generator=g).to(DEV)
    wide[:, :K] = a_d
    alone, among = torch.empty(1, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.linear_f32_rows(wide[M - 1:, :K], w_d, None, alone)
    ops.linear_f32_rows(wide[:, :K], w_d, None, among)
    assert torch.equal(alone[0], among[M - 1])


@pytest.mark.parametrize("M,N,K", [(17, 16, 32), (33, 31, 36), (64, 65, 31), (100, 200, 96), (129, 127, 33), (700, 300, 64),
                                   (300, 2100, 40), (1500, 1030, 20), (128, 768, 3072),
                                   (128, 128, 16), (1030, 2051, 48), (2049, 1155, 160)])
def test_tiles(M, N, K):
    """Every tile shape of the many-rows kernel, tails in M, N and K, rows on and off 16-byte boundaries."""
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a, w, bias, base = (torch.randn(shape, generator=g) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    wide = torch.randn(M, K + 3, generator=g).to(DEV)
    wide[:, :K] = a.to(DEV)
    outs = []
    for rows in (a.to(DEV), wide[:, :K]):
        out = base.clone().to(DEV)
        ops.linear_simt(rows, w.to(DEV), bias.to(DEV), out, accumulate=True)
        want = product(a, w, bias, None, None, base)
        assert float((out.cpu().double() - want).abs().max()) < sum_bound(K) * 8 * float(want.abs().max())
        outs.append(out)
    assert torch.equal(outs[0], outs[1])                         # however the rows lie: the same sums in the same order
