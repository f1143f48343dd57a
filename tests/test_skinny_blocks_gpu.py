"""The weight-streaming product with its rows in blocks: against 64 bits at the edges of the blocks, with every epilogue, and the
norm-fused form against the norm and the product as kernels of their own."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops_for():
    from pagedserve_b200.kernels.ops import Ops

    return Ops(torch.bfloat16)


@pytest.mark.parametrize("M", [9, 16, 17, 24, 25, 33, 41, 63, 64])
@pytest.mark.parametrize("N,K", [(768, 768), (2304, 768), (3080, 1024), (1600, 1600), (770, 3072), (48, 64)])
def test_blocks(M, N, K):
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    bias, base = torch.randn(N, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)
    want = a.double() @ w.double().T
    for out_dtype, accumulate, tol in ((torch.float32, 0, 2e-5), (torch.float32, 1, 2e-5), (torch.bfloat16, 0, 6e-3), (torch.float32, 3, 2e-5)):
        expect = want * bias if accumulate & 2 else want + bias
        expect = expect + base if accumulate & 1 else expect
        out = base.clone().to(out_dtype)
        ops.linear_skinny(a, w, bias, out, accumulate=accumulate)
        assert float((out.double() - expect).abs().max()) < tol * float(expect.abs().max()), (out_dtype, accumulate)


@pytest.mark.parametrize("M", [17, 32])
@pytest.mark.parametrize("scatter", [False, True])
def test_fused_norm_in_blocks(M, scatter):
    """N of 2,304 runs in blocks of 16 rows, 3,072 with all rows in a CTA; a q|k|v product sends keys and values to the pages."""
    from pagedserve_b200.config.gpt2 import GPT2Config
    from pagedserve_b200.config.engine_config import EngineConfig
    from pagedserve_b200.engine.batch import StepEntry
    from pagedserve_b200.engine.engine import Engine

    config = GPT2Config(n_layer=1, n_embd=768, n_head=12, n_inner=3072, vocab_size=64, n_positions=64, layer_norm_epsilon=1e-5,
                        activation_function="gelu_new")
    engine = Engine.random(config, 1, EngineConfig(dtype="bfloat16", num_blocks=M, max_num_seqs=M))
    ctx = engine.runner.prepare([StepEntry(i, [i % 64]) for i in range(M)])
    engine.runner.begin(ctx)
    block, ops, group = engine.model.blocks[0], engine.ops, engine.cache.groups[0]
    k_pool, v_pool = group.layer_views(0)
    layer = SimpleNamespace(k_pool=k_pool, v_pool=v_pool, page_stride=group.page_stride, page_size=group.page_size,
                            block_table=ctx.block_tables[0])
    x = torch.randn(M + 3, 768, generator=torch.Generator().manual_seed(M)).to(DEV)
    norm, weight, bias = block.norms["pre_mixer"], block.mixer.w_qkv, block.mixer.b_qkv
    rows = torch.randperm(M, generator=torch.Generator().manual_seed(M)).to(torch.int32).to(DEV)
    for picked in (None,) if scatter else (None, rows):
        normed = norm.forward(x[:M] if picked is None else x, rows=picked)
        want = torch.empty(M, 2304, dtype=torch.bfloat16, device=DEV)
        ops.linear_tc(normed, weight, bias, want)
        out = torch.full_like(want, float("nan"))
        ops.linear_skinny_fused(norm.defer(x[:M] if picked is None else x, rows=picked), weight, bias, out,
                                kv=(ctx, layer, 768, 768, 64) if scatter else None)
        if scatter:
            pages = ctx.block_tables[0][ctx.token_slot.long(), 0].long()
            for pool, at in ((k_pool, 768), (v_pool, 1536)):
                out[:, at:at + 768] = pool[pages, :, 0].reshape(M, 768)
        # rounded bfloat16 results of float32 sums in two orders: half a step of the largest at most, and then one
        assert float((out.float() - want.float()).abs().max()) <= 2.0 ** -7 * float(want.float().abs().max())
    engine.cache.check_invariants()


@pytest.mark.parametrize("M", [8, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(768, 1024), (2400, 1024), (768, 2048), (768, 2080), (2384, 2080)])
def test_fused_norm_at_depths(M, N, K):
    """Depths on both sides of where an SM holds two CTAs and one, widths on both sides of where blocks of 16 rows are resident."""
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    x, gamma, beta = torch.randn(M, K, generator=g) * 2 + 0.5, torch.randn(K, generator=g) * 0.2 + 1, torch.randn(K, generator=g) * 0.2
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    x, gamma, beta, w = (t.to(DEV) for t in (x, gamma, beta, w))
    prologue = SimpleNamespace(weight=gamma, bias=beta, eps=1e-5, has_mean=True)
    rows = SimpleNamespace(x=x, rows=None, shape=x.shape, norm=SimpleNamespace(fused_prologue=lambda: prologue))
    out = torch.empty(M, N, device=DEV)
    ops.linear_skinny_fused(rows, w, None, out)
    normed = torch.nn.functional.layer_norm(x.double(), (K,), gamma.double(), beta.double(), 1e-5).to(torch.bfloat16)
    want = normed.double() @ w.double().T
    # a normed number that lies between two bfloat16 values may round either way: one step of 2^-8 of it, in one of K terms
    assert float((out.double() - want).abs().max()) < 2.0 ** -8 * 4 / K ** 0.5 * 4 + 2e-5 * float(want.abs().max())


def milliseconds(calls):
    for call in calls:
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for call in calls:
            call()
    times = []
    for _ in range(8):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times[2:])


@pytest.mark.parametrize("M,N,K", [(33, 3072, 768), (48, 3072, 1024), (64, 3072, 1024), (48, 4096, 1024), (40, 1600, 1600)])
def test_blocks_are_taken_where_they_win(M, N, K):
    """Weights that come from memory: the product takes blocks only where they beat the few-rows tcgen05 kernel and one CTA for all
    rows.  With registers for fewer CTAs on an SM than the rule counts on, they lost by 8 to 28 % at these sizes."""
    ops = ops_for()
    a = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    weights = [(torch.randn(N, K, device=DEV) / K ** 0.5).to(torch.bfloat16) for _ in range(1 + int(260e6) // (2 * N * K))]
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    chosen = milliseconds([lambda w=w: ops.linear(a, w, None, out) for w in weights])
    few = milliseconds([lambda w=w: ops.linear_rows_tc(a, w, None, out) for w in weights])
    assert chosen < 1.03 * few
