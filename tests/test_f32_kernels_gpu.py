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


# The error of a float32 sum of K products of normal numbers, relative to the largest of the results: every addition rounds by at
# most 2^-24 of a partial sum of at most the size of the result, signs at random, so that sqrt(K) of them add up (a result is
# about 0.4 sqrt(K) 2^-24 off at one standard deviation); and a few roundings of what comes behind the sum.  Operands rounded to 10
# bits of mantissa are off by 2^-11 of a product, which is far beyond it (tests/test_f32_bound_cpu.py).
def bound(K):
    return 3 * (K ** 0.5 + 4) * 2.0 ** -24


def size_of(want):
    """The largest result, or one (a sum's standard deviation) where there are few and they happen to be small."""
    return max(1.0, float(want.abs().max()))


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
        assert float((out.cpu().double() - want).abs().max()) < bound(K) * size_of(want), (act, how)
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
    """The tiles that the rule takes (test_every_tile has each of them), tails in M, N and K, rows on and off 16-byte boundaries."""
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
        assert float((out.cpu().double() - want).abs().max()) < bound(K) * size_of(want)
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
        assert float((out.double() - want).abs().max()) < bound(K) * size_of(want), accumulate
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


@pytest.mark.parametrize("tile,M,N,K,aligned", [(1, 2048, 2304, 768, 1), (1, 1900, 2305, 48, 1), (2, 1030, 2051, 48, 1), (2, 2048, 2304, 768, 0),
                                                (2, 2048, 2304, 772, 1), (3, 384, 2304, 768, 1), (4, 128, 768, 768, 1), (5, 33, 31, 36, 1)])
def test_the_rule_takes_every_tile(tile, M, N, K, aligned):
    assert ops_for().core.ps_gemm_f32_tile(M, N, K, aligned) == tile


@pytest.mark.parametrize("tile", [1, 3, 4, 5])
@pytest.mark.parametrize("M", [128, 129, 255, 257])
@pytest.mark.parametrize("N,K", [(128, 16), (129, 48), (255, 784), (257, 48), (385, 16)])
def test_every_tile(tile, M, N, K):
    """Each shape of tiles has the bits of the 64 x 64 ones and the sums of 64 bits, with every epilogue: the last tiles of 128 x 128 are
    moved back inside the matrix, store nothing twice and, with an odd first column, halves of pairs; what lies beside the result
    stays."""
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a, w, vector, base = (torch.randn(shape, generator=g) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    a_d, w_d, vector_d = a.to(DEV), w.to(DEV), vector.to(DEV)
    for act, accumulate in ((None, 0), ("gelu_tanh", 0), (None, 1), (None, 2), (None, 3)):
        outs = []
        for which in (tile, 2):
            room = torch.full((M + 1, N + 3), 7.0, device=DEV)
            room[:M, :N] = base.to(DEV)
            ops.linear_simt(a_d, w_d, vector_d, room[:M, :N], act=act, accumulate=accumulate, tile=which)
            assert bool((room[M:] == 7.0).all()) and bool((room[:, N:] == 7.0).all())
            outs.append(room[:M, :N])
        assert torch.equal(outs[0], outs[1]), (act, accumulate)
        want = product(a, w, None if accumulate & 2 else vector, act, vector if accumulate & 2 else None, base if accumulate & 1 else None)
        assert float((outs[0].cpu().double() - want).abs().max()) < bound(K) * size_of(want), (act, accumulate)


@pytest.mark.parametrize("N,K", [(768, 768), (300, 3072), (50, 1028)])
def test_sums_by_rows(N, K):
    """A row's sums are the same bits in every product of at most 16 rows, and in every product of more; between the two they differ as
    float32 sums in two orders do."""
    ops, g = ops_for(), torch.Generator().manual_seed(N + K)
    a, w = torch.randn(300, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) / K ** 0.5).to(DEV)
    results = {}
    for M in (1, 3, 16, 17, 64, 300):
        results[M] = torch.empty(M, N, device=DEV)
        ops.linear(a[:M], w, None, results[M])
    for few, more in ((1, 16), (3, 16), (17, 300), (64, 300)):
        assert torch.equal(results[few], results[more][:few]), (few, more)
    assert float((results[16] - results[300][:16]).abs().max()) < bound(K) * size_of(results[16])


@pytest.mark.parametrize("head_dim", [64, 100])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_of_a_prompt_in_portions(head_dim, window):
    """A prompt of 200 tokens whole and in portions: 16 tokens and more run on the prompt kernel, with the same bits as the whole; fewer, and
    single ones, on the token kernel, whose bits too do not depend on the cut.  Between the two: float32 sums in two orders."""
    heads, kv_heads, total = 4, 2, 200
    step, ops = Step([(total, total)], heads, kv_heads, head_dim, page=16, seed=head_dim), ops_for()
    q, row = step.q[0].reshape(total, -1).to(DEV), int(step.ctx.item_slot[0])
    as_ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)

    def run(portion):
        out = torch.empty(total, heads * head_dim, device=DEV)
        for begin in range(0, total, portion):
            end = min(begin + portion, total)
            short = portion < 16
            ctx = SimpleNamespace(num_items=1, num_short_items=int(short), num_short_tokens=end - begin if short else 0,
                                  num_long_blocks=-(-(end - begin) // 64), q_start=as_ints([0, end - begin]), kv_len=as_ints([end]),
                                  item_slot=as_ints([row]), token_slot=as_ints([row] * (end - begin)), positions=as_ints(range(begin, end)))
            ops.attention_f32(q[begin:end], out[begin:end], ctx, step.layer, heads, kv_heads, head_dim, window, head_dim ** -0.5)
        return out

    whole, single = run(total), run(1)
    for portion in (16, 17, 63, 64, 130):
        assert torch.equal(run(portion), whole), portion
    for portion in (5, 15):
        assert torch.equal(run(portion), single), portion
    # weights that add up to one times values of a few, each from sums of up to 200 float32 terms
    assert float((whole - single).abs().max()) < 2e-6
