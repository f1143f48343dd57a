"""Float32 products and prompt attention on the tensor cores (csrc/gemm_f32_tc.cu, csrc/attention_f32_tc.cu) against 64 bits and against the
float32 multiply-adds they replace."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops_for():
    from pagedserve_b200.kernels.ops import Ops

    return Ops(torch.float32)


# A float32 sum of K products of normal numbers, relative to the largest of the results: sqrt(K) roundings of at most 2^-24 of the result add
# up (tests/test_f32_kernels_gpu.py derives the same bound; tests/test_f32_bound_cpu.py shows that operands of 10 bits are beyond it).
def bound(K):
    return 3 * (K ** 0.5 + 4) * 2.0 ** -24


def size_of(want):
    return max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("M", [1, 17, 127, 128, 129, 300])
@pytest.mark.parametrize("N,K", [(64, 256), (127, 260), (129, 508), (385, 516), (257, 2044), (768, 3080)])
def test_every_epilogue(M, N, K):
    """Edges of the 128 x 128 tiles, blocks of 64 k's and parts that end inside one, rows on their own pitch, K in clusters or in one CTA."""
    ops, g = ops_for(), torch.Generator().manual_seed(M + N + K)
    a, w, vector, base = (torch.randn(shape, generator=g) for shape in ((M, K), (N, K), (N,), (M, N)))
    w /= K ** 0.5
    wide = torch.full((M, K + 4), float("nan"))
    wide[:, :K] = a
    a_d, w_d, vector_d = wide.to(DEV)[:, :K], w.to(DEV), vector.to(DEV)
    parts = ops._tc_library().ps_gemm_f32_tc_parts(K)
    exact = a.double() @ w.double().T
    for act, accumulate in ((None, 0), ("gelu_tanh", 4), (None, 1), (None, 2), (None, 3 + 4)):
        outs = []
        for splits in (1, parts // 2, parts, 0):
            room = torch.full((M + 1, N + 3), 7.0, device=DEV)
            room[:M, :N] = base.to(DEV)
            ops.linear_f32_tc(a_d, w_d, vector_d, room[:M, :N], act=act, accumulate=accumulate, splits=splits)
            assert bool((room[M:] == 7.0).all()) and bool((room[:, N:] == 7.0).all())
            outs.append(room[:M, :N].clone())
        assert all(torch.equal(outs[0], other) for other in outs[1:]), (act, accumulate)
        want = exact * vector.double() if accumulate & 2 else exact + vector.double()
        if act == "gelu_tanh":
            want = torch.nn.functional.gelu(want, approximate="tanh")
        if accumulate & 1:
            want = want + base.double()
        assert float((outs[0].cpu().double() - want).abs().max()) < bound(K) * size_of(want), (act, accumulate)
    assert int(ops.status.item()) == 0


@pytest.mark.parametrize("M,N,K", [(384, 2304, 768), (2048, 768, 768), (651, 1024, 4096), (384, 768, 3072), (200, 1600, 6400), (64, 768, 256)])
@pytest.mark.parametrize("kind", ["normal", "positive", "wide"])
def test_error_is_no_larger_than_that_of_multiply_adds(M, N, K, kind):
    """Against 64 bits, beside the float32 kernel that adds one product after the other: signs at random, no signs (every cut of a sum
    in the same direction), magnitudes over many powers of two."""
    ops, g = ops_for(), torch.Generator(device=DEV).manual_seed(M + N + K)
    a, w = (torch.randn(shape, generator=g, device=DEV) for shape in ((M, K), (N, K)))
    if kind == "positive":
        a, w = a.abs(), w.abs()
    elif kind == "wide":
        a = a * torch.exp2(torch.randint(-12, 12, (M, K), generator=g, device=DEV).float())
    want = a.double() @ w.double().T
    errors = []
    for run in (ops.linear_f32_tc, ops.linear_simt):
        out = torch.empty(M, N, device=DEV)
        run(a, w, None, out)
        errors.append(float((out.double() - want).norm() / want.norm()))
    assert errors[0] <= errors[1], errors


def test_infinities_and_nans():
    ops, g = ops_for(), torch.Generator().manual_seed(1)
    a, w = torch.randn(140, 512, generator=g), torch.randn(130, 512, generator=g)
    a[3, 7], a[4, 9], a[5, 500], a[6, 0], a[6, 511] = float("inf"), float("-inf"), float("nan"), float("inf"), float("inf")
    w[11, 7], w[12, 9], w[13, 100] = 0.0, -0.0, float("inf")
    w[14] = 1.0                                                  # numbers without second pieces
    a[20], w[20] = 3.4e38, 1e-3                                  # near the largest float: no piece is rounded up to an infinity
    a[21] = 3.0e38                                               # sums beyond it
    a[22] = torch.randn(512, generator=g) * 2.0 ** -100
    want = (a.double() @ w.double().T).float()
    for splits in (0, 1, 2):
        out = torch.empty(140, 130, device=DEV)
        ops.linear_f32_tc(a.to(DEV), w.to(DEV), None, out, splits=splits)
        out = out.cpu()
        plain = torch.empty(140, 130, device=DEV)
        ops.linear_simt(a.to(DEV), w.to(DEV), None, plain)
        plain = plain.cpu()
        finite = torch.isfinite(plain)
        assert torch.equal(torch.isnan(out), torch.isnan(plain)) and torch.equal(torch.isinf(out), torch.isinf(plain))
        assert torch.equal(out[torch.isinf(plain)], plain[torch.isinf(plain)])
        rows = [r for r in range(140) if r not in (20, 21)]
        assert torch.allclose(out[rows][finite[rows]], want[rows][finite[rows]], rtol=1e-5, atol=1e-4)
        assert torch.allclose(out[20][finite[20]], plain[20][finite[20]], rtol=1e-3)


@pytest.mark.parametrize("power", [-60, -100, -108, -112, -116, -120, -124])
def test_small_numbers(power):
    """Rows whose third pieces end below the smallest bfloat16 number: no further from 64 bits than multiply-adds, rows of zeros stay zeros."""
    from test_f32_kernels_gpu import Step, plain

    ops, g = ops_for(), torch.Generator().manual_seed(1)
    a, w = torch.randn(140, 768, generator=g).to(DEV) * 2.0 ** power, torch.randn(130, 768, generator=g).to(DEV)
    a[7], a[8] = 0.0, a[8] * 2.0 ** 30
    want, errors = a.double() @ w.double().T, []
    size = want.abs().amax(1, keepdim=True).clamp_min(1e-300)
    for run in (ops.linear_f32_tc, ops.linear_simt):
        out = torch.empty(140, 130, device=DEV)
        run(a, w, None, out)
        errors.append(float(((out.double() - want) / size).norm()))
        assert bool((out[7] == 0).all())
    assert errors[0] <= errors[1], errors
    step, errors = Step([(200, 200)], 2, 2, 64, page=16, seed=7), []
    step.layer.v_pool.mul_(2.0 ** power)
    step.v = [v * 2.0 ** power for v in step.v]
    q, want = step.q[0].reshape(200, -1).to(DEV), plain(step, 0.125, 0, 0.0, None, False)
    for heads in (ops.F32_TC_HEADS, (1, 0)):
        ops.F32_TC_HEADS = heads
        out = torch.empty(200, 128, device=DEV)
        ops.attention_f32(q, out, step.ctx, step.layer, 2, 2, 64, 0, 0.125)
        errors.append(float((out.cpu().double() - want).norm() / want.norm()))
    assert errors[0] <= 1.5 * errors[1], errors


def test_products_in_a_row():
    """Products launched one behind the other, each reading what the one before wrote: the weights among it where they may be."""
    ops, g = ops_for(), torch.Generator().manual_seed(2)
    made, outs = torch.empty(512, 512, device=DEV), torch.empty(6, 300, 512, device=DEV)
    a = torch.randn(300, 512, generator=g).to(DEV)
    left, right = torch.randn(6, 512, 256, generator=g).to(DEV), (torch.randn(6, 512, 256, generator=g) / 16).to(DEV)
    for i in range(6):
        ops.linear_f32_tc(left[i], right[i], None, made)
        ops.linear_f32_tc(a, made, None, outs[i], splits=(1, 2, 4)[i % 3])
    for i in range(6):
        want = a.double() @ (left[i].double() @ right[i].double().T).T
        assert float((outs[i].double() - want).abs().max()) < 1e-5 * float(want.abs().max()), i


@pytest.mark.parametrize("factor", [False, True])
def test_vectors_that_the_kernel_in_front_makes(factor):
    """A bias or a vector of factors may be the result of the kernel in front, which writes it late (K of 8,192), weights ready or not."""
    ops, g = ops_for(), torch.Generator().manual_seed(4)
    made, outs = torch.full((1, 700), float("nan"), device=DEV), torch.empty(12, 200, 700, device=DEV)
    left, right = torch.randn(12, 1, 8192, generator=g).to(DEV), (torch.randn(700, 8192, generator=g) / 90).to(DEV)
    a, w = torch.randn(200, 768, generator=g).to(DEV), (torch.randn(700, 768, generator=g) / 28).to(DEV)
    torch.cuda.synchronize()
    for i in range(12):
        ops.linear_f32_tc(left[i], right, None, made)
        if i % 2:
            ops.linear_f32_tc(a, w, made[0], outs[i], accumulate=2 if factor else 0)
        else:
            ops.linear(a, w, None if factor else made[0], outs[i], factor=made[0] if factor else None)
    for i in range(12):
        vector = left[i].double() @ right.double().T
        want = (a.double() @ w.double().T) * vector if factor else a.double() @ w.double().T + vector
        # (the vector: a sum of 8,192 products)
        assert float((outs[i].double() - want).abs().max()) < 2 * bound(8192) * size_of(want) * size_of(vector), i


def test_refused():
    from pagedserve_b200.kernels.ops import KernelError

    ops = ops_for()
    a, w, out = torch.zeros(32, 512, device=DEV), torch.zeros(64, 512, device=DEV), torch.zeros(32, 64, device=DEV)
    with pytest.raises(KernelError):
        ops.linear_f32_tc(a, w, None, out, splits=3)
    with pytest.raises(KernelError):
        ops.linear_f32_tc(a[:, 1:], w[:, 1:], None, out)
    with pytest.raises(KernelError):
        ops.linear_f32_tc(a[:, :128], w[:, :128], None, out)


@pytest.mark.parametrize("head_dim,all_values", [(64, False), (36, True), (60, False)])
@pytest.mark.parametrize("window,softcap,with_sink", [(0, 0.0, False), (300, 5.0, True), (-200, 0.0, True)])
def test_prompt_attention(head_dim, all_values, window, softcap, with_sink):
    """Edges of the blocks of 128 queries and of the tiles of 128 keys, portions behind cached keys; no further from 64 bits than the kernel of
    multiply-adds (half as much again where both are at a rounding's size)."""
    from test_f32_kernels_gpu import Step, plain

    entries = [(16, 16), (127, 127), (128, 128), (129, 129), (700, 257), (1100, 20), (512, 128)]
    step, ops, scale = Step(entries, 4, 2, head_dim, page=16, seed=head_dim), ops_for(), head_dim ** -0.5
    sink = torch.randn(4, generator=torch.Generator().manual_seed(3)) if with_sink else None
    q = torch.cat([rows.reshape(len(rows), -1) for rows in step.q]).to(DEV)
    want = plain(step, scale, window, softcap, sink, all_values)
    errors = []
    for heads in (ops.F32_TC_HEADS, (1, 0)):
        ops.F32_TC_HEADS = heads
        out = torch.full((len(q), want.shape[1]), float("nan"), device=DEV)
        ops.attention_f32(q, out, step.ctx, step.layer, 4, 2, head_dim, window, scale, softcap, None if sink is None else sink.to(DEV), all_values)
        errors.append(float((out.cpu().double() - want).norm() / want.norm()))
    assert errors[0] <= 1.5 * errors[1] and errors[0] < 1e-6, errors
    assert int(ops.status.item()) == 0


@pytest.mark.parametrize("before", [0, 70, 128])
@pytest.mark.parametrize("softcap", [0.0, 5.0])
def test_prompt_attention_of_part_of_a_tile(before, softcap):
    """The last tile's products are formed for the keys that are there, in steps of 16: a portion that ends at each edge of a step has the
    bits of those rows of a longer one."""
    from test_f32_kernels_gpu import Step, plain

    ops, outs = ops_for(), {}
    for end in [before + 160] + [before + n for n in (16, 17, 31, 32, 33, 48, 58, 59, 64, 65, 80, 96, 112, 113, 127, 128, 129, 144)]:
        step = Step([(before + 160, 160)], 2, 1, 64, page=16, seed=9)
        count = end - before
        step.ctx.q_start[1], step.ctx.kv_len[0], step.ctx.num_long_blocks = count, end, (count + 63) // 64
        q = step.q[0].reshape(160, -1)[:count].to(DEV)
        outs[count] = torch.full((count, 128), float("nan"), device=DEV)
        ops.attention_f32(q, outs[count], step.ctx, step.layer, 2, 1, 64, 0, 0.125, softcap or None)
    want = plain(step, 0.125, 0, softcap, None, False)
    assert float((outs[160].cpu().double() - want).norm() / want.norm()) < 1e-6
    for count, out in outs.items():
        assert torch.equal(out, outs[160][:count]), count
    assert int(ops.status.item()) == 0


def test_prompt_attention_of_infinities():
    """Scores and values that are not finite reach the rows that see them, as they do term by term, and no others."""
    from test_f32_kernels_gpu import Step

    step, ops = Step([(200, 200)], 2, 2, 64, page=16, seed=7), ops_for()
    layer, q = step.layer, step.q[0].reshape(200, -1).to(DEV)
    place = lambda token: (int(layer.block_table[int(step.ctx.item_slot[0]), token // 16]), slice(None), token % 16)
    layer.k_pool[place(60)][:, 5] = float("-inf")
    layer.v_pool[place(70)][:, 3] = float("inf")
    layer.v_pool[place(150)][:, 9] = float("nan")
    layer.k_pool[place(180)][:] = 1e30
    q[100, 64:] = float("inf")
    outs = []
    for heads in (ops.F32_TC_HEADS, (1, 0)):
        ops.F32_TC_HEADS = heads
        outs.append(torch.empty(200, 128, device=DEV))
        ops.attention_f32(q, outs[-1], step.ctx, layer, 2, 2, 64, 0, 0.125)
    new, old = outs
    assert torch.equal(torch.isnan(new), torch.isnan(old)) and torch.equal(torch.isinf(new), torch.isinf(old))
    assert bool(torch.isfinite(new[:60]).all()) and bool(torch.isinf(new[70:, 3]).any()) and bool(torch.isnan(new[160, 9]))
    there = torch.isfinite(old)
    assert torch.allclose(new[there], old[there], rtol=1e-5, atol=1e-5)
