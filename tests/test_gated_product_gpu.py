"""The product that forms a gated activation in its epilogue, against 64 bits: every form, tails in rows and columns, rows of weight
zero, experts by tile, one CTA and pairs of CTAs per tile."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
CLAMPED = ("clamped_swish", 1.5, 1.0, 1.702)


def formed(g, u, w, form, limit):
    if form == "silu":
        return g * torch.sigmoid(g) * u * w
    if form == "gelu_tanh":
        return torch.nn.functional.gelu(g, approximate="tanh") * u * w
    g, u = (g * w).clamp(max=limit), (u * w).clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


@pytest.mark.parametrize("form", ["silu", "gelu_tanh", CLAMPED])
@pytest.mark.parametrize("M,F,K", [(65, 8, 8), (128, 128, 64), (129, 136, 72), (300, 72, 200), (257, 264, 1024), (2600, 1160, 136)])
@pytest.mark.parametrize("weighted", [False, True])
def test_gated(form, M, F, K, weighted):
    from pagedserve_b200.kernels.ops import Ops

    ops, g = Ops(torch.bfloat16), torch.Generator().manual_seed(M + F + K)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * F, K, generator=g) * 2 / math.sqrt(K)).to(torch.bfloat16).to(DEV)
    weight = torch.rand(M, generator=g).to(DEV) if weighted else None
    if weighted:
        weight[::7] = 0.0
        a[::7] = float("inf")                                   # rows of no token give zeros whatever stands in them
    inner = torch.full((M, F + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.linear_gated(a, w, inner[:, :F], form=form, row_weight=weight)
    y = a.double() @ w.double().T
    want = formed(y[:, :F], y[:, F:], 1.0 if weight is None else weight[:, None].double(), form, 1.0)
    if weighted:
        want[::7] = 0.0
    # bfloat16 results round at 2^-9; the sums and the exponentials are float32's
    assert float((inner[:, :F].double() - want).abs().max()) < 6e-3 * float(want.abs().max())
    assert bool(torch.isnan(inner[:, F:]).all()) and int(ops.status_flag(DEV).item()) == 0


@pytest.mark.parametrize("form", ["silu", CLAMPED])
@pytest.mark.parametrize("M", [65, 129, 257, 385, 512])
@pytest.mark.parametrize("F,K", [(8, 64), (136, 200), (264, 1032)])
@pytest.mark.parametrize("weighted", [False, True])
def test_pairs_of_ctas(form, M, F, K, weighted):
    """One CTA of the pair has the gates, the other the ups; the second one's rows may all lie past the last, its columns end inside a
    tile.  The bits of one CTA per tile, and the sums of 64 bits."""
    from pagedserve_b200.kernels.ops import Ops

    ops, g = Ops(torch.bfloat16), torch.Generator().manual_seed(M + F + K)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * F, K, generator=g) * 2 / math.sqrt(K)).to(torch.bfloat16).to(DEV)
    weight = torch.rand(M, generator=g).to(DEV) if weighted else None
    if weighted:
        weight[::7] = 0.0
        a[::7] = float("inf")
    room = torch.full((2, M + 1, F + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    for inner, bn in zip(room, (256, 512)):
        ops.linear_gated(a, w, inner[:M, :F], form=form, row_weight=weight, bn=bn)
    assert torch.equal(room[0], room[1]) and bool((room[:, M:] == 7.0).all()) and bool((room[:, :, F:] == 7.0).all())
    y = a.double() @ w.double().T
    want = formed(y[:, :F], y[:, F:], 1.0 if weight is None else weight[:, None].double(), form, 1.0)
    if weighted:
        want[::7] = 0.0
    assert float((room[1, :M, :F].double() - want).abs().max()) < 6e-3 * float(want.abs().max())
    assert int(ops.status_flag(DEV).item()) == 0


@pytest.mark.parametrize("F,K", [(72, 64), (256, 136)])
def test_experts(F, K):
    from pagedserve_b200.kernels.ops import Ops

    ops, g, E = Ops(torch.bfloat16), torch.Generator().manual_seed(F), 3
    tile_expert = torch.tensor([2, 0, -1, 1, 0], dtype=torch.int32, device=DEV)
    M = 5 * 128
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E * 2 * F, K, generator=g) * 2 / math.sqrt(K)).to(torch.bfloat16).to(DEV)
    weight = torch.rand(M, generator=g).to(DEV)
    inner = torch.zeros(M, F, dtype=torch.bfloat16, device=DEV)
    ops.linear_gated(a, w, inner, form=CLAMPED, row_weight=weight, tile_expert=tile_expert, experts=E)
    for tile, expert in enumerate(tile_expert.tolist()):
        rows = slice(128 * tile, 128 * tile + 128)
        if expert < 0:
            assert bool((inner[rows] == 0).all())
            continue
        y = a[rows].double() @ w[2 * F * expert:2 * F * (expert + 1)].double().T
        want = formed(y[:, :F], y[:, F:], weight[rows, None].double(), CLAMPED, 1.5)
        assert float((inner[rows].double() - want).abs().max()) < 6e-3 * float(want.abs().max()), tile


def milliseconds(call):
    """The least of ten runs of a graph of twenty calls."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(20):
            call()
    times = []
    for _ in range(10):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times[2:])


@pytest.mark.parametrize("bn", [256, 512])
@pytest.mark.parametrize("M,F,K", [(129, 1024, 1024), (3969, 1024, 1024), (3969, 688, 256)])
def test_rows_that_do_not_fill_a_tile_cost_what_a_full_tile_does(M, F, K, bn):
    """The rows past the last one have sums of zero; the epilogue spends no more on them than on others.  On one CTA and pairs of
    CTAs per tile.  They once took the slow path of the division: 1.6 times the time at 129 rows."""
    from pagedserve_b200.kernels.ops import Ops

    ops, full = Ops(torch.bfloat16), -(-M // 256) * 256
    a = torch.randn(full, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device=DEV) / math.sqrt(K)).to(torch.bfloat16)
    inner = torch.empty(full, F, dtype=torch.bfloat16, device=DEV)

    def least(rows):
        return milliseconds(lambda: ops.linear_gated(a[:rows], w, inner[:rows], form="silu", bn=bn))

    assert least(M) < 1.2 * least(full)


@pytest.mark.parametrize("M,F,K", [(3000, 4096, 1024), (8192, 2048, 1024), (1024, 1024, 1024), (1536, 4096, 2048)])
def test_the_better_of_one_cta_and_pairs_is_taken(M, F, K):
    """With the numbers of the plain product's rule, pairs were taken at K of 1,024, where they lose by up to 18 %."""
    from pagedserve_b200.kernels.ops import Ops

    ops = Ops(torch.bfloat16)
    a = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device=DEV) / math.sqrt(K)).to(torch.bfloat16)
    inner = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    runs = [[milliseconds(lambda: ops.linear_gated(a, w, inner, bn=bn)) for bn in (0, 256, 512)] for _ in range(4)]
    chosen, one, pairs = (min(times) for times in zip(*runs))             # (in turn: the clocks follow the load)
    assert chosen < 1.07 * min(one, pairs), runs
