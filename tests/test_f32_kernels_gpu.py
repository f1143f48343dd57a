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


class Step:
    """Requests with pages in no order, each with some keys cached and some queries at its end; the short ones come first."""

    def __init__(self, entries, n_heads, n_kv_heads, head_dim, page, seed):
        g = torch.Generator().manual_seed(seed)
        entries = sorted(entries, key=lambda entry: entry[1] >= 16)
        self.lengths = [length for length, _ in entries]
        pages = [-(-length // page) for length in self.lengths]
        order = torch.randperm(sum(pages) + 2, generator=g).tolist()
        table = torch.full((len(entries) + 1, max(pages)), -1, dtype=torch.int32)
        rows = torch.randperm(len(entries) + 1, generator=g)[:len(entries)]
        pool = torch.full((sum(pages) + 2, 2, n_kv_heads, page, head_dim), float("nan"))
        self.k = [torch.randn(length, n_kv_heads, head_dim, generator=g) for length in self.lengths]
        self.v = [torch.randn(length, n_kv_heads, head_dim, generator=g) for length in self.lengths]
        for r, count in enumerate(pages):
            for i in range(count):
                p = order.pop()
                table[rows[r], i] = p
                here = self.k[r][i * page:(i + 1) * page], self.v[r][i * page:(i + 1) * page]
                for which in (0, 1):
                    pool[p, which, :, :len(here[which])] = here[which].transpose(0, 1)
        pool = pool.to(DEV)
        counts = [count for _, count in entries]
        self.q = [torch.randn(count, n_heads, head_dim, generator=g) for count in counts]
        as_ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
        starts = [sum(counts[:i]) for i in range(len(counts) + 1)]
        short = sum(count < 16 for count in counts)
        self.ctx = SimpleNamespace(
            num_items=len(counts), num_short_items=short, num_short_tokens=starts[short],
            num_long_blocks=sum(-(-count // 64) for count in counts[short:]) + 2, q_start=as_ints(starts),
            kv_len=as_ints(self.lengths), item_slot=as_ints(rows.tolist()),
            token_slot=as_ints([int(rows[r]) for r, count in enumerate(counts) for _ in range(count)]),
            positions=as_ints([length - count + i for length, count in entries for i in range(count)]))
        self.layer = SimpleNamespace(k_pool=pool[:, 0], v_pool=pool[:, 1], page_stride=pool.stride(0), page_size=page,
                                     block_table=table.to(DEV))


def plain(step, scale, window, softcap, sink, all_values):
    out = []
    for q, k, v in zip(step.q, step.k, step.v):
        q, k, v = q.double(), k.double(), v.double()
        H, G = q.shape[1], k.shape[1]
        at = torch.arange(len(k) - len(q), len(k))[:, None]
        key = torch.arange(len(k))[None]
        seen = key <= at
        if window > 0:
            seen &= at - key < window
        elif window < 0:
            seen &= at // -window == key // -window
        for_heads = []
        for h in range(H):
            s = q[:, h] @ k[:, h // (H // G)].T * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            s = s.masked_fill(~seen, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(len(q), 1)], 1)
            p = torch.softmax(s, -1)[:, :len(k)]
            for_heads += [p @ v[:, other] for other in (range(G) if all_values else [h // (H // G)])]
        out.append(torch.cat(for_heads, -1))
    return torch.cat(out)


@pytest.mark.parametrize("n_heads,n_kv_heads,head_dim", [(3, 3, 64), (4, 2, 128), (4, 1, 36), (2, 2, 4), (2, 1, 100)])
@pytest.mark.parametrize("window,softcap,with_sink,all_values", [(0, 0.0, False, False), (19, 5.0, True, False), (-40, 0.0, True, True),
                                                                 (64, 0.0, False, False)])
def test_attention(n_heads, n_kv_heads, head_dim, window, softcap, with_sink, all_values):
    entries = [(1, 1), (700, 1), (33, 5), (16, 16), (64, 64), (129, 65), (200, 17), (331, 200), (65, 1)]
    step = Step(entries, n_heads, n_kv_heads, head_dim, page=8, seed=head_dim + n_heads)
    ops, scale = ops_for(), head_dim ** -0.5
    sink = torch.randn(n_heads, generator=torch.Generator().manual_seed(3)) if with_sink else None
    q = torch.cat([rows.reshape(len(rows), -1) for rows in step.q]).to(DEV)
    columns = n_heads * (n_kv_heads if all_values else 1) * head_dim
    out = torch.full((len(q), columns), float("nan"), device=DEV)
    layer = step.layer
    assert ops.attention_f32_ok(q, out, layer.k_pool, layer.v_pool, layer.page_stride, head_dim)
    ops.attention_f32(q, out, step.ctx, layer, n_heads, n_kv_heads, head_dim, window, scale, softcap,
                      None if sink is None else sink.to(DEV), all_values)
    want = plain(step, scale, window, softcap, sink, all_values)
    # scores of order one: a score is off by at most (head_dim + 3) 2^-24 of a few, the sums of up to 700 weights by 700 * 2^-24
    assert float((out.cpu().double() - want).abs().max()) < 1e-5
    # the general kernel, which these calls ran on before
    general = torch.full_like(out, float("nan"))
    ops.paged_attention_simt(q, general, layer.k_pool, layer.v_pool, layer.page_stride, step.ctx.token_slot, step.ctx.positions,
                             layer.block_table, n_heads, n_kv_heads, head_dim, layer.page_size, window, scale, softcap,
                             None if sink is None else sink.to(DEV), all_values=all_values)
    assert float((out - general).abs().max()) < 2e-5


def test_attention_keeps_a_later_infinity_out():
    """An infinity in a later token's key and value stays out of the earlier queries of its block of queries."""
    step = Step([(80, 80)], 2, 2, 64, page=16, seed=5)
    ops, layer = ops_for(), step.layer
    q = step.q[0].reshape(80, -1).to(DEV)
    clean, out = torch.empty(80, 128, device=DEV), torch.empty(80, 128, device=DEV)
    ops.attention_f32(q, clean, step.ctx, layer, 2, 2, 64, 0, 0.125)
    page, place = int(layer.block_table[int(step.ctx.item_slot[0]), 70 // 16]), 70 % 16
    layer.v_pool[page, :, place] = float("inf")
    layer.k_pool[page, :, place] = float("nan")
    ops.attention_f32(q, out, step.ctx, layer, 2, 2, 64, 0, 0.125)
    assert torch.equal(out[:70], clean[:70]) and bool(torch.isnan(out[70:]).all())


@pytest.mark.parametrize("M", [1, 4, 5, 8, 16])
@pytest.mark.parametrize("N,K", [(9473, 4), (9501, 768), (9490, 772), (9477, 1024)])
def test_few_rows_of_a_vocabulary(M, N, K):
    """CTAs that walk over several groups of columns: every epilogue, and the sums of the form without walking."""
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a, w, bias, base = (torch.randn(shape, generator=g) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    a, w, bias, base = (t.to(DEV) for t in (a, w, bias, base))
    for accumulate in (0, 1, 3):
        out = base.clone()
        ops.linear_f32_rows(a, w, bias, out, accumulate=accumulate)
        want = product(a, w, None if accumulate == 3 else bias, None, bias if accumulate == 3 else None, base if accumulate else None)
        assert float((out.double() - want).abs().max()) < sum_bound(K) * 8 * float(want.abs().max()), accumulate
    part = torch.empty(M, 4000, device=DEV)
    whole = torch.empty(M, N, device=DEV)
    ops.linear_f32_rows(a, w[:4000], None, part)
    ops.linear_f32_rows(a, w, None, whole)
    assert torch.equal(whole[:, :4000], part)


@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 5])
def test_weights_made_by_the_kernel_in_front(tile):
    """linear_simt reads its second operand only when the kernel in front has ended, which may have made it: a product whose result is
    the weight of the next, on every kind of tile, several times in a row with other numbers."""
    M, N, K = 700, 512, 512
    ops, g = ops_for(), torch.Generator().manual_seed(tile)
    made, outs = torch.empty(N, K, device=DEV), torch.empty(6, M, N, device=DEV)
    a = torch.randn(M, K, generator=g).to(DEV)
    left, right = torch.randn(6, N, 256, generator=g).to(DEV), (torch.randn(6, K, 256, generator=g) / 16).to(DEV)
    for i in range(6):
        ops.linear_simt(left[i], right[i], None, made)
        ops.linear_simt(a, made, None, outs[i], tile=tile)
    for i in range(6):
        want = a.double() @ (left[i].double() @ right[i].double().T).T
        assert float((outs[i].double() - want).abs().max()) < 1e-5 * float(want.abs().max()), i
