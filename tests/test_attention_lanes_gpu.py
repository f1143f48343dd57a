"""Attention of single tokens on CUDA cores (csrc/attention_lanes.cu) against 64 bits and the split-key kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("heads,kv_heads,head_dim,page", [(12, 12, 64, 16), (6, 2, 48, 8), (3, 1, 40, 64), (4, 2, 128, 32), (2, 2, 104, 4)])
@pytest.mark.parametrize("warps", [0, 4, 8, 16])
@pytest.mark.parametrize("window,softcap,with_sink", [(None, None, False), (70, 5.0, True), (-128, None, True)])
def test_rounds_masks_and_fresh_keys(heads, kv_heads, head_dim, page, warps, window, softcap, with_sink):
    """Contexts at the edges of a round's keys (64 to 256 at 64 numbers a head, half of that above), portions of several tokens, the newest
    keys written right before the launch while the older ones are fetched ahead of the wait."""
    from test_kernels_gpu import PagedCase, ops_for, rel_err

    ops = ops_for(torch.bfloat16)
    lengths, fresh = [1, 2, 63, 64, 65, 128, 129, 255, 256, 257, 600, 1100], [1, 2, 1, 1, 3, 1, 1, 15, 1, 1, 1, 1]
    case = PagedCase(ops, torch.bfloat16, lengths, heads, kv_heads, head_dim, page, seed=head_dim)
    sink = torch.randn(heads, generator=torch.Generator().manual_seed(1)) if with_sink else None
    scale, rows, item_of, q_start, start, want = head_dim ** -0.5, [], [], [0], 0, []
    for item, (length, new) in enumerate(zip(lengths, fresh)):
        rows += list(range(start + length - new, start + length))
        item_of += [item] * new
        q_start.append(q_start[-1] + new)
        at = torch.arange(length - new, length)[:, None]
        key = torch.arange(length)[None]
        seen = key <= at
        if window is not None:
            seen &= (at - key < window) if window > 0 else (at // -window == key // -window)
        q = case.q[start + length - new:start + length].double().reshape(new, heads, head_dim)
        k, v = (x[start:start + length].double().reshape(length, kv_heads, head_dim).repeat_interleave(heads // kv_heads, 1)
                for x in (case.k, case.v))
        s = torch.einsum("ihd,jhd->hij", q, k) * scale
        s = softcap * torch.tanh(s / softcap) if softcap else s
        s = s.masked_fill(~seen, float("-inf"))
        s = torch.cat([s, sink.double()[:, None, None].expand(heads, new, 1)], -1) if with_sink else s
        want.append(torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :length], v).reshape(new, -1))
        start += length
    rows_dev, ints = torch.tensor(rows, device=DEV), lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q, item, positions = case.q.to(DEV)[rows_dev].contiguous(), ints(item_of), case.positions[rows_dev].contiguous()
    k_new, v_new = case.k.to(DEV)[rows_dev].contiguous(), case.v.to(DEV)[rows_dev].contiguous()
    poison = torch.full_like(k_new, float("nan"))
    for dtype in (torch.bfloat16, torch.float32):
        ops.kv_append(poison, poison, item, positions, case.table, case.k_pool, case.v_pool, case.page_stride, kv_heads, head_dim, page)
        torch.cuda.synchronize()
        out = torch.full((len(rows), heads * head_dim), float("nan"), dtype=dtype, device=DEV)
        ops.kv_append(k_new, v_new, item, positions, case.table, case.k_pool, case.v_pool, case.page_stride, kv_heads, head_dim, page)
        ops.attention_lanes(q, out, case.k_pool, case.v_pool, case.page_stride, item, positions, case.table, heads, kv_heads, head_dim, page,
                            window, scale, max(lengths), q_start=ints(q_start), kv_len=ints(lengths), softcap=softcap,
                            sink=None if sink is None else sink.to(DEV), warps=warps)
        # results rounded to bfloat16 (2^-9 each), or float32 sums of up to 1,100 weights by approximate powers of two (2^-22 each)
        assert rel_err(out, torch.cat(want)) < (4e-3 if dtype == torch.bfloat16 else 2e-6)


def test_every_value_head():
    from test_kernels_gpu import PagedCase, ops_for, rel_err

    ops, heads, kv_heads, head_dim, page, lengths = ops_for(torch.bfloat16), 4, 2, 64, 16, [5, 300]
    case = PagedCase(ops, torch.bfloat16, lengths, heads, kv_heads, head_dim, page, seed=2)
    out, other = (torch.full((305, heads * kv_heads * head_dim), float("nan"), dtype=torch.float32, device=DEV) for _ in range(2))
    arguments = (case.k_pool, case.v_pool, case.page_stride, case.token_item, case.positions, case.table, heads, kv_heads, head_dim, page, None, 0.125)
    ops.attention_lanes(case.q.to(DEV), out, *arguments, 300, all_values=True)
    ops.paged_attention_simt(case.q.to(DEV), other, *arguments, all_values=True)
    assert rel_err(out, other.double()) < 2e-6


def test_which_tokens_run_on_it():
    """By sizes and alignment: contexts that one CTA walks through, or many pairs; rows of whole 16-byte pieces."""
    from test_kernels_gpu import ops_for

    ops, pool = ops_for(torch.bfloat16), torch.empty(64, 2, 8, 16, 64, dtype=torch.bfloat16, device=DEV)
    q = torch.empty(64, 512, dtype=torch.bfloat16, device=DEV)
    ok = lambda tokens, head_dim, columns, longest, stride=16384, rows=q: ops.attention_lanes_ok(rows, tokens, pool[:, 0], pool[:, 1], stride,
                                                                                               head_dim, columns, longest)
    assert ok(1, 64, 8, 1280) and ok(64, 64, 8, 8192) and ok(16, 128, 8, 1024)
    assert not ok(1, 64, 8, 1281) and not ok(1, 128, 8, 1024) and not ok(64, 32, 8, 1024) and not ok(64, 96, 8, 1024)
    assert not ok(1, 64, 8, 1024, stride=16388) and not ok(1, 64, 8, 1024, stride=2 ** 31) and not ok(1, 64, 8, 1024, rows=q[:, 4:])


@pytest.mark.parametrize("head_dim", [64, 48, 128])
@pytest.mark.parametrize("warps", [4, 8, 16])
@pytest.mark.parametrize("with_sink", [False, True])
def test_numbers_that_are_not_finite(head_dim, warps, with_sink):
    """A NaN in the query or in a key that it sees, infinite scores of either sign and infinite values give what the split-key kernel and the
    equations give: NaN in every column, in one column, or an infinity; and other heads, tokens and unseen keys are not touched."""
    from test_kernels_gpu import PagedCase, ops_for, rel_err

    ops, heads, kv_heads, page = ops_for(torch.bfloat16), 4, 2, 16
    lengths = [5, 90, 300, 301, 302, 303, 700]
    case = PagedCase(ops, torch.bfloat16, lengths, heads, kv_heads, head_dim, page, seed=warps)
    items = torch.arange(len(lengths), dtype=torch.int32, device=DEV)
    last = torch.tensor(lengths, device=DEV) - 1
    q = torch.randn(len(lengths), heads * head_dim, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).to(DEV)
    q[1:, 3] = q[1:, head_dim + 3] = 1.0                         # (heads 0 and 1 read key head 0, heads 2 and 3 key head 1)
    q[4, head_dim + 3] = -1.0
    place = lambda item, key: (int(case.table[item, key // page]), 0, key % page)
    q[0, 2 * head_dim + 1] = float("nan")                        # item 0, head 2
    case.k_pool[place(1, 17)][3] = float("nan")                  # item 1, heads 0 and 1
    case.k_pool[place(2, 290)][3] = float("inf")                 # scores of +infinity
    case.v_pool[place(3, 64)][5] = float("inf")                  # one column
    case.k_pool[place(4, 100)][3] = float("-inf")                # -infinity for head 0 (a weight of zero), +infinity for head 1
    case.k_pool[place(5, 7)][3], case.v_pool[place(5, 7)][9] = float("-inf"), float("inf")        # zero times infinity
    sink = torch.randn(heads, generator=torch.Generator().manual_seed(1)).to(DEV) if with_sink else None
    arguments = (case.k_pool, case.v_pool, case.page_stride, items, last.to(torch.int32), case.table, heads, kv_heads, head_dim, page, None,
                 head_dim ** -0.5, max(lengths))
    out, other = (torch.full((len(lengths), heads * head_dim), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops.attention_lanes(q, out, *arguments, sink=sink, warps=warps)
    ops.paged_attention_decode(q, other, *arguments, sink=sink)
    assert torch.equal(out.isnan(), other.isnan()) and torch.equal(out.isinf(), other.isinf())
    there = out.isfinite()
    assert rel_err(torch.where(there, out, 0), torch.where(there, other, 0)) < 8e-3
    rows = out.reshape(len(lengths), heads, head_dim)
    assert bool(rows[0, 2].isnan().all()) and bool(rows[1, :2].isnan().all()) and bool(rows[2, :2].isnan().all()) and bool(rows[4, 1].isnan().all())
    assert bool(rows[3, :2, 5].isinf().all()) and bool(rows[5, :2, 9].isnan().all())
    assert int((~there).sum()) == head_dim * (1 + 2 + 2 + 1) + 2 + 2


def test_contexts_of_different_lengths():
    """Which kernel and how many warps run where one context may be far longer than the others: heads of 128 with 149 to 296 pairs
    leave it beyond 512 keys, and 297 and more pairs take 8 warps where contexts may be long (a number of warps has bits of its own)."""
    from test_kernels_gpu import PagedCase, ops_for

    ops, pool = ops_for(torch.bfloat16), torch.empty(8, 2, 8, 16, 128, dtype=torch.bfloat16, device=DEV)
    ok = lambda tokens, longest: ops.attention_lanes_ok(torch.empty(tokens, 1024, dtype=torch.bfloat16, device=DEV), tokens, pool[:, 0], pool[:, 1],
                                                        16384, 128, 8, longest)
    assert ok(18, 1024) and not ok(19, 1024) and not ok(37, 513) and ok(19, 512) and ok(37, 512) and ok(38, 1280) and ok(38, 8192) and not ok(37, 8192)
    for heads, head_dim, longest, warps in ((1, 64, 1024, (16, 8, 8, 8, 8, 4, 4, 4)), (1, 64, 512, (16, 8, 8, 8, 8, 4, 4, 4)), (1, 64, 256, (16, 8, 8, 4, 4, 4, 4, 4)),
                                            (1, 64, 2048, (16, 8, 8, 8, 8, 8, 8, 4)), (1, 128, 512, (16, 8, 8, 8, 8, 8, 8, 4))):
        lengths = [500] + [20] * 9
        case = PagedCase(ops, torch.bfloat16, lengths, heads, 1, head_dim, 16, seed=1)
        for tokens, expected in zip((148, 149, 296, 297, 444, 445, 592, 593), warps):
            item = torch.arange(tokens, dtype=torch.int32, device=DEV) % len(lengths)
            positions = torch.tensor(lengths, dtype=torch.int32, device=DEV)[item.long()] - 1
            q = torch.randn(tokens, head_dim, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(DEV)
            outs = []
            for count in (0, expected) + tuple({4, 8, 16} - {expected}):
                outs.append(torch.empty(tokens, head_dim, dtype=torch.float32, device=DEV))
                ops.attention_lanes(q, outs[-1], case.k_pool, case.v_pool, case.page_stride, item, positions, case.table, heads, 1, head_dim, 16,
                                    None, head_dim ** -0.5, longest, warps=count)
            assert torch.equal(outs[0], outs[1]) and not torch.equal(outs[0], outs[2]) and not torch.equal(outs[0], outs[3]), (longest, tokens)
