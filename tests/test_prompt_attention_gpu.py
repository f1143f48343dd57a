"""Prompt attention on tcgen05 (csrc/attention_prefill_tc.cu) where it takes one way or another by its data: capped scores by
multiply-adds or by special functions, whatever lies beside them; more portions than a warp has lanes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("head_dim,row_threads", [(64, 1), (64, 2), (128, 1), (128, 2)])
@pytest.mark.parametrize("scale", [0.05, 0.37, 2.0, 6.0])
@pytest.mark.parametrize("softcap,window", [(50.0, None), (50.0, 70), (30.0, 200), (1500.0, None)])
def test_scores_small_and_large_of_many_portions(head_dim, row_threads, scale, softcap, window):
    """Scores from well within the cap to far beyond it (and a cap so large that the last coefficient could vanish), whose maximum rises in
    small and in large steps from key tile to key tile.  The bound is that of probabilities rounded to bfloat16 (2^-8 each)."""
    from test_kernels_gpu import PagedCase, rel_err
    from test_tefopel_gpu import ops_for, plain_attention_rows, run_attention_kernel

    lengths = [16 + (37 * i) % 120 for i in range(38)] + [1, 128, 129, 256, 700, 131]
    case = PagedCase(ops_for(torch.bfloat16), torch.bfloat16, lengths, 4, 2, head_dim, 16, seed=head_dim)
    sink = torch.tensor([4.0, -30.0, 0.5, -1.0])
    got = run_attention_kernel("tcgen05-two" if row_threads == 2 else "tcgen05", ops_for(torch.bfloat16), case, lengths, window, scale,
                               softcap, sink.to(DEV))
    assert torch.isfinite(got.float()).all()
    want = plain_attention_rows(case, scale, softcap, window or 10 ** 6, sink)
    assert rel_err(got, want) < 8e-3


def capped_portions(entries, behind, garbage, head_dim, row_threads, softcap, window, seed=3):
    """Bits of the portions ``entries`` (kv length, new tokens), with entries of queries ``behind`` times as large after them in the step,
    and ``garbage`` in every place of the pool that holds no key of theirs."""
    from test_kernels_gpu import ops_for

    heads, kv_heads, page, ops = 4, 2, 16, ops_for(torch.bfloat16)
    g = torch.Generator().manual_seed(seed)
    keys = [torch.randn(kv, kv_heads, 2, head_dim, generator=g).to(torch.bfloat16) for kv, _ in entries]
    queries = [torch.randn(new, heads * head_dim, generator=g).to(torch.bfloat16) for _, new in entries]
    all_entries = list(entries)
    if behind:
        for kv, new in ((60, 40), (200, 130)):
            all_entries.append((kv, new))
            keys.append(torch.randn(kv, kv_heads, 2, head_dim, generator=g).to(torch.bfloat16) * behind)
            queries.append(torch.randn(new, heads * head_dim, generator=g).to(torch.bfloat16) * behind)
    widest = max(-(-kv // page) for kv, _ in all_entries)
    pool = torch.full((widest * len(all_entries) + 8, 1, 2, kv_heads, page, head_dim), garbage, dtype=torch.bfloat16)
    table = torch.zeros(len(all_entries), widest + 8, dtype=torch.int32)             # (page 0 holds garbage alone)
    for item, rows in enumerate(keys):
        for i in range(-(-len(rows) // page)):
            table[item, i] = number = 1 + item * widest + i
            part = rows[i * page:(i + 1) * page]
            pool[number, 0, :, :, :len(part)] = part.permute(2, 1, 0, 3)
    q = torch.cat(queries).to(DEV)
    out = torch.full_like(q, float("nan"))
    starts = torch.tensor([sum(new for _, new in all_entries[:i]) for i in range(len(all_entries) + 1)], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.prefill_attention_tc(q, out, pool.to(DEV), 0, starts, torch.tensor([kv for kv, _ in all_entries], dtype=torch.int32, device=DEV),
                             table.to(DEV), 0, len(all_entries), sum(-(-new // 128) for _, new in all_entries), heads, kv_heads, head_dim,
                             page, window, head_dim ** -0.5, status=status, row_threads=row_threads, softcap=softcap)
    assert int(status.item()) == 0
    return out[:sum(new for _, new in entries)]


@pytest.mark.parametrize("head_dim,row_threads", [(64, 1), (64, 2), (128, 1), (128, 2)])
@pytest.mark.parametrize("softcap", [8.0, 4.0])
@pytest.mark.parametrize("window", [None, 50])
def test_capped_portions_do_not_depend_on_what_they_do_not_see(head_dim, row_threads, softcap, window):
    """Neither on left-over rows of their pages and of shared memory nor on the queries behind theirs in the step.  Scores are about 1 in size,
    so that some of them are beyond the half of the cap, up to which multiply-adds form it, and most are not."""
    entries = [(40, 40), (100, 100), (130, 130), (333, 20), (461, 200)]
    first = capped_portions(entries, 0, 0.0, head_dim, row_threads, softcap, window)
    assert bool(torch.isfinite(first).all())
    for behind, garbage in ((0, 40.0), (0, -3000.0), (1, 0.0), (30, 40.0), (30, float("nan")), (0, 0.0)):
        assert torch.equal(first, capped_portions(entries, behind, garbage, head_dim, row_threads, softcap, window)), (behind, garbage)


@pytest.mark.parametrize("head_dim,row_threads", [(64, 1), (64, 2), (128, 1), (128, 2)])
def test_capped_prompts_in_portions_are_the_bits_of_the_whole(head_dim, row_threads):
    """Each score's cap is formed by its size alone, whoever shares its warp."""
    from test_kernels_gpu import ops_for

    whole = capped_portions([(300, 300)], 0, 0.0, head_dim, row_threads, 6.0, None)
    heads, kv_heads, page, ops, g = 4, 2, 16, ops_for(torch.bfloat16), torch.Generator().manual_seed(3)
    keys = torch.randn(300, kv_heads, 2, head_dim, generator=g).to(torch.bfloat16)
    q = torch.randn(300, heads * head_dim, generator=g).to(torch.bfloat16).to(DEV)
    pool = torch.zeros(19, 1, 2, kv_heads, page, head_dim, dtype=torch.bfloat16)
    for i in range(19):
        part = keys[i * page:(i + 1) * page]
        pool[i, 0, :, :, :len(part)] = part.permute(2, 1, 0, 3)
    table, pool = torch.arange(19, dtype=torch.int32, device=DEV)[None].contiguous(), pool.to(DEV)
    for cuts in ((0, 17, 150, 300), (0, 129, 260, 300)):
        for begin, end in zip(cuts, cuts[1:]):
            out = torch.full((end - begin, heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
            ops.prefill_attention_tc(q[begin:end].contiguous(), out, pool, 0, torch.tensor([0, end - begin], dtype=torch.int32, device=DEV),
                                     torch.tensor([end], dtype=torch.int32, device=DEV), table, 0, 1, -(-(end - begin) // 128), heads, kv_heads,
                                     head_dim, page, None, head_dim ** -0.5, row_threads=row_threads, softcap=6.0)
            assert torch.equal(out, whole[begin:end]), (begin, end)


@pytest.mark.parametrize("head_dim,row_threads", [(64, 1), (64, 2), (128, 1), (128, 2)])
@pytest.mark.parametrize("scale,softcap", [(1.0, 1e-6), (1e-3, 1e-9), (1.0, 3e-4), (0.1, 1e-4), (1.0, 1e-2)])
def test_caps_far_below_the_scores(head_dim, row_threads, scale, softcap):
    """Every score at the cap, but for those of queries of zeros, which are zero: the coefficients of the cap's polynomial reach no infinity."""
    from test_kernels_gpu import PagedCase, rel_err
    from test_tefopel_gpu import ops_for, plain_attention_rows, run_attention_kernel

    lengths, sink = [20, 140], torch.tensor([0.5, -30.0, -1.0, 0.0])
    case = PagedCase(ops_for(torch.bfloat16), torch.bfloat16, lengths, 4, 2, head_dim, 16, seed=head_dim)
    case.q[:140] = 0.0
    got = run_attention_kernel("tcgen05-two" if row_threads == 2 else "tcgen05", ops_for(torch.bfloat16), case, lengths, None, scale,
                               softcap, sink.to(DEV))
    assert bool(torch.isfinite(got.float()).all())
    assert rel_err(got, plain_attention_rows(case, scale, softcap, 10 ** 6, sink)) < 8e-3
