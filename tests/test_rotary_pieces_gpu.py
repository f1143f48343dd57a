"""The rotary cache write by pieces of 16 bytes beside the one by pairs."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops_for(dtype=torch.bfloat16):
    from pagedserve_b200.kernels.ops import Ops

    return Ops(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,heads,kv_heads,dim,rot", [(1, 4, 2, 64, 32), (37, 16, 16, 128, 64), (700, 3, 1, 72, 72), (33, 2, 2, 16, 0)])
@pytest.mark.parametrize("own_values", [False, True])
def test_rotary_by_pieces(dtype, T, heads, kv_heads, dim, rot, own_values):
    """Rows on 16-byte boundaries against the same rows two numbers further on, which run pair by pair: the same bits."""
    ops, g, page = ops_for(dtype), torch.Generator().manual_seed(T + dim), 8
    wide = torch.randn(T, (heads + 2 * kv_heads) * dim + 16, generator=g).to(dtype).to(DEV)
    inv = (10000.0 ** (-torch.arange(max(rot // 2, 1), dtype=torch.float32) * 2 / max(rot, 1))).to(DEV)
    ctx = SimpleNamespace(token_slot=torch.zeros(T, dtype=torch.int32, device=DEV), positions=torch.arange(T, dtype=torch.int32, device=DEV))
    count = -(-T // page)
    got = []
    for shift in (0, 2):
        rows = torch.zeros_like(wide)
        used = (heads + 2 * kv_heads) * dim
        rows[:, shift:shift + used] = wide[:, :used]
        pool = torch.zeros(count, 2, kv_heads, page, dim, dtype=dtype, device=DEV)
        layer = SimpleNamespace(k_pool=pool[:, 0], v_pool=pool[:, 1], page_stride=pool.stride(0), page_size=page,
                                block_table=torch.arange(count, dtype=torch.int32, device=DEV)[None])
        part = lambda at, n: rows[:, shift + at * dim:shift + (at + n) * dim]
        ops.rotary_cache_write(part(0, heads), part(heads, kv_heads), part(heads + kv_heads, kv_heads) if own_values else None, inv, rot,
                               True, ctx, layer, heads, kv_heads, dim)
        got.append((part(0, heads).clone(), pool))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool((got[0][1][0] != 0).any())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,heads,kv_heads,dim,rot", [(700, 4, 4, 64, 32), (103, 16, 16, 128, 64), (1500, 3, 1, 72, 72), (5000, 2, 2, 16, 0)])
@pytest.mark.parametrize("own_values", [False, True])
def test_many_tokens(dtype, T, heads, kv_heads, dim, rot, own_values):
    """Enough numbers for the kernel to go by pieces."""
    assert T * (heads * rot + 2 * kv_heads * dim) * torch.empty(0, dtype=dtype).element_size() >= 512 * 1024
    test_rotary_by_pieces(dtype, T, heads, kv_heads, dim, rot, own_values)


@pytest.mark.parametrize("T", [1, 8, 32])
def test_few_tokens_are_as_fast_as_pair_by_pair(T):
    """Rows on 16-byte boundaries take no longer than rows two numbers further on, which can only go pair by pair."""
    ops, heads, kv_heads, dim = ops_for(), 16, 4, 64
    ctx = SimpleNamespace(token_slot=torch.zeros(T, dtype=torch.int32, device=DEV), positions=torch.arange(T, dtype=torch.int32, device=DEV))
    pool = torch.zeros(T, 2, kv_heads, 16, dim, dtype=torch.bfloat16, device=DEV)
    layer = SimpleNamespace(k_pool=pool[:, 0], v_pool=pool[:, 1], page_stride=pool.stride(0), page_size=16,
                            block_table=torch.arange(T, dtype=torch.int32, device=DEV)[None])
    inv, times = torch.rand(dim // 2, device=DEV), []
    for shift in (0, 2):
        rows = torch.randn(T, (heads + 2 * kv_heads) * dim + 16, device=DEV).to(torch.bfloat16)
        part = lambda at, n: rows[:, shift + at * dim:shift + (at + n) * dim]
        call = lambda: ops.rotary_cache_write(part(0, heads), part(heads, kv_heads), part(heads + kv_heads, kv_heads), inv, dim, True, ctx,
                                              layer, heads, kv_heads, dim)
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(200):
                call()
        least = []
        for _ in range(12):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            least.append(start.elapsed_time(end))
        times.append(min(least[2:]))
    assert times[0] < 1.05 * times[1]
