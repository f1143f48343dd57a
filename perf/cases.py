"""What a user of this engine has it do, as a list of cases that can be timed and checked.

Whole calls ("serve"): requests run through ``Engine.step`` with continuous batching, a step holding one token of every request that
is past its prompt and, up to a token budget, portions of the prompts that are not; the next tokens are given, as when a
recorded trace is replayed or a text is scored, and every step returns its logits.  Single layers: a GPT-2 block, a
feed-forward of routed experts, a state-space mixer and rotary attention with a window, each through its part's
``forward`` on the tokens of a prepared step.

``exact`` states the same in plain torch in 64 bits, from the layers' equations, with code of its own.
"""

import math
import random

import torch

from pagedserve_b200.config import tefopel, vozirax, zositar
from pagedserve_b200.config.engine_config import EngineConfig
from pagedserve_b200.config.gpt2 import GPT2Config
from pagedserve_b200.engine.batch import StepEntry
from pagedserve_b200.engine.engine import Engine
from pagedserve_b200.parts.base import LayerContext

DEVICE = "cuda:0"
VOCAB = 50257                  # GPT-2's
SMALL_VOCAB = 512              # of models that are built for one of their layers only
POSITIONS = 1024               # GPT-2's longest sequence
PAGE = 16
EPS = 1e-5
TAPS = 4                       # rows that the state-space mixer's convolution spans
ROTARY_BASE, SOFTCAP = 10000.0, 50.0
LIMIT = 7.0                    # of the clamped experts


# ------------------------------------------------------------------------------------------------ the cases
def _serve(name, dtype, requests, longest, new, width=768, heads=12, layers=12, even=False, budget=2048):
    return dict(name=name, kind="serve", dtype=dtype, requests=requests, longest=longest, new=new, width=width, heads=heads,
                layers=layers, even=even, budget=budget)


def listed():
    return [
        # one user at a prompt, GPT-2 124M: the smallest batches, where latency and launches count
        _serve("serve-1-bf16", "bfloat16", 1, 33, 16),
        # a few users, prompts of different lengths up to half the context: the batch of the engine's headline benchmark
        _serve("serve-8-bf16", "bfloat16", 8, 512, 24),
        # a busy server: steps of 64 requests, prompts coming in as portions beside them
        _serve("serve-64-bf16", "bfloat16", 64, 256, 24),
        # reading long prompts (a document to be classified, a long chat): 2,048 tokens in one step
        _serve("prompts-2048-bf16", "bfloat16", 2, 1024, 1, even=True),
        # the engine's default precision: a batch that answers, and long prompts
        _serve("serve-5-float32", "float32", 5, 130, 8),
        _serve("prompts-2048-float32", "float32", 2, 1024, 1, even=True),
        # a layer of the 1.5B model over ragged prompts, as a step of a loaded server brings them
        dict(name="block-1600-bf16", kind="block", dtype="bfloat16", width=1600, heads=25, requests=9, longest=1023),
        # a layer of the 345M model in float32, odd sizes
        dict(name="block-1024-float32", kind="block", dtype="float32", width=1024, heads=16, requests=3, longest=333),
        # routed experts with a shared one (the w1024 model's) over a prompt step
        dict(name="experts-1024-bf16", kind="experts", dtype="bfloat16", width=1024, experts=8, top=2, ff=1024, shared=2048,
             tokens=2048),
        # the w2048 model's experts over a large step
        dict(name="experts-2048-bf16", kind="experts", dtype="bfloat16", width=2048, experts=8, top=2, ff=2048, shared=4096,
             tokens=4099),
        # a state-space layer over long prompts
        dict(name="ssm-2048-bf16", kind="ssm", dtype="bfloat16", width=2048, heads=64, dim=64, state=128, requests=3,
             longest=1500),
        # windowed attention with capped scores and sinks over long prompts
        dict(name="rotary-2048-bf16", kind="rotary", dtype="bfloat16", width=2048, heads=16, kv_heads=16, dim=128, window=1024,
             requests=3, longest=2048),
    ]


def _spread(rng, low, high):
    """A whole number, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """Another case of the same ranges: the models' widths, 1 to 64 requests, prompts of 8 tokens to the model's context,
    both precisions."""
    kind = rng.choice(("serve", "serve", "serve", "block", "block", "experts", "ssm", "rotary"))
    dtype = rng.choice(("bfloat16", "bfloat16", "float32"))
    if kind == "serve":
        width, heads, layers = rng.choice(((768, 12, 12), (1024, 16, 8), (1600, 25, 4)))
        if dtype == "float32":
            requests, longest, new = _spread(rng, 1, 8), _spread(rng, 8, 160), rng.randint(1, 6)
        else:
            requests, longest, new = _spread(rng, 1, 64), _spread(rng, 8, 600), rng.randint(1, 24)
            longest = min(longest, max(8, 16384 // requests))
        case = _serve("", dtype, requests, longest, new, width, heads, layers, budget=rng.choice((512, 1024, 2048)))
        del case["name"]
        return case
    if kind == "block":
        width, heads = rng.choice(((768, 12), (1024, 16), (1600, 25)))
        most = 8192 if dtype == "bfloat16" else 2048
        requests = _spread(rng, 1, 16)
        return dict(kind=kind, dtype=dtype, width=width, heads=heads, requests=requests,
                    longest=_spread(rng, 16, min(POSITIONS, most // requests)))
    width = rng.choice((1024, 2048))
    if kind == "experts":
        return dict(kind=kind, dtype="bfloat16", width=width, experts=rng.choice((4, 8, 16)), top=rng.choice((1, 2)), ff=width,
                    shared=2 * width, tokens=_spread(rng, 128, 4096))
    requests = _spread(rng, 1, 6)
    longest = _spread(rng, 64, 4096 // requests)
    if kind == "ssm":
        return dict(kind=kind, dtype="bfloat16", width=width, heads=width // 32, dim=64, state=rng.choice((64, 128)),
                    requests=requests, longest=min(longest, 2048))
    dim = width // 16
    return dict(kind=kind, dtype="bfloat16", width=width, heads=16, kv_heads=rng.choice((4, 16)), dim=dim,
                window=rng.choice((256, 1024)), requests=requests, longest=min(longest, 2048))


# ------------------------------------------------------------------------------------------------ sizes and inputs
def _lengths(case):
    """Tokens of each prompt: the longest one and others between a quarter of it and all of it, shorter ones first (a step
    lays its short entries out ahead of the others, and a layer's rows stand in that order)."""
    longest, count = case["longest"], case["requests"]
    if case.get("even"):
        return [longest] * count
    rng = random.Random(longest * 1009 + count)
    return sorted([longest] + [rng.randint(max(1, longest // 4), longest) for _ in range(count - 1)])


def _schedule(case):
    """The steps as lists of (request, first token, one past its last, whether the last one's logits are wanted)."""
    lengths, new, budget = _lengths(case), case["new"], case["budget"]
    done = [0] * len(lengths)                              # tokens of each request that have run
    steps = []
    while any(ran < length + new - 1 for ran, length in zip(done, lengths)):
        entries, room = [], budget
        for r, length in enumerate(lengths):
            if length <= done[r] < length + new - 1:
                entries.append((r, done[r], done[r] + 1, True))
                room -= 1
        for r, length in enumerate(lengths):
            if done[r] < length and room > 0:
                end = min(length, done[r] + room)
                entries.append((r, done[r], end, end == length))
                room -= end - done[r]
        for r, _, end, _ in entries:
            done[r] = end
        steps.append(entries)
    return steps


def _generator(seed, salt):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 16 + salt)


def _normal(g, shape, std=1.0, mean=0.0):
    """Weights: every number one that bfloat16 holds, so that both precisions start from the same ones."""
    return (torch.randn(shape, generator=g, device=DEVICE) * std + mean).to(torch.bfloat16)


def _gpt2_weights(case, layers, vocab, seed):
    g, W = _generator(seed, 1), case["width"]
    weights = {"wte.weight": _normal(g, (vocab, W), 0.02), "wpe.weight": _normal(g, (POSITIONS, W), 0.01),
               "ln_f.weight": _normal(g, (W,), 0.1, 1.0), "ln_f.bias": _normal(g, (W,), 0.1)}
    for layer in range(layers):
        p = "h.%d." % layer
        for name, shape, std in (("attn.c_attn", (W, 3 * W), 0.02), ("attn.c_proj", (W, W), 0.02 / math.sqrt(2 * layers)),
                                 ("mlp.c_fc", (W, 4 * W), 0.02), ("mlp.c_proj", (4 * W, W), 0.02 / math.sqrt(2 * layers))):
            weights[p + name + ".weight"] = _normal(g, shape, std)
            weights[p + name + ".bias"] = _normal(g, shape[1:], 0.02)
        for name in ("ln_1", "ln_2"):
            weights[p + name + ".weight"] = _normal(g, (W,), 0.1, 1.0)
            weights[p + name + ".bias"] = _normal(g, (W,), 0.1)
    return weights


def _gpt2_config(case, layers, vocab):
    return GPT2Config(n_layer=layers, n_embd=case["width"], n_head=case["heads"], n_inner=4 * case["width"], vocab_size=vocab,
                      n_positions=POSITIONS, layer_norm_epsilon=EPS, activation_function="gelu_new")


def _experts_config(case):
    mlp = zositar.moe_mlp(case["experts"], case["top"], case["ff"], limit=LIMIT, shared_ff=case["shared"], shared_limit=LIMIT)
    return zositar.ZositarConfig(vocab=SMALL_VOCAB, width=case["width"], norm_eps=EPS,
                                 layers=[zositar.attention_layer(4, 4, 64, None, mlp)])


def _ssm_config(case):
    return vozirax.VoziraxConfig(vocab=SMALL_VOCAB, width=case["width"], norm_eps=EPS, logit_scale=1.0,
                                 layers=[vozirax.mamba_layer(case["heads"], case["dim"], case["state"], None, conv=TAPS)])


def _rotary_config(case):
    return tefopel.TefopelConfig(vocab=SMALL_VOCAB, width=case["width"], norm_eps=EPS, layers=[tefopel.attention_layer(
        case["heads"], case["kv_heads"], case["dim"], case["window"], None, rot_dims=(case["dim"] // 4) * 2, softcap=SOFTCAP)])


def _layer_weights(case, seed):
    """Tensors of the one-layer models, by their checkpoints' names."""
    g, W = _generator(seed, 2), case["width"]
    std = W ** -0.5
    weights = {"embed": _normal(g, (SMALL_VOCAB, W)), "final.norm": _normal(g, (W,), 0.1)}
    p = "l0."
    weights[p + "norm1"] = _normal(g, (W,), 0.1)
    if case["kind"] == "experts":
        weights["head"] = _normal(g, (SMALL_VOCAB, W), std)
        for name, rows in (("q", 256), ("k", 256), ("v", 256)):
            weights[p + "mix." + name] = _normal(g, (rows, W), std)
            weights[p + "mix." + name + ".b"] = _normal(g, (rows,), 0.3)
        weights[p + "mix.q.norm"], weights[p + "mix.k.norm"] = _normal(g, (64,), 0.1, 1.0), _normal(g, (64,), 0.1, 1.0)
        weights[p + "mix.o"] = _normal(g, (W, 256), 1 / 16)
        weights[p + "norm2"] = _normal(g, (W,), 0.1, 1.0)
        weights[p + "mlp.router"] = _normal(g, (case["experts"], W), 2 * std)
        for name, ff in [("e%d." % e, case["ff"]) for e in range(case["experts"])] + [("shared.", case["shared"])]:
            weights[p + "mlp." + name + "gate"] = _normal(g, (ff, W), 2 * std)
            weights[p + "mlp." + name + "up"] = _normal(g, (ff, W), 2 * std)
            weights[p + "mlp." + name + "down"] = _normal(g, (W, ff), ff ** -0.5)
    elif case["kind"] == "ssm":
        H, inner = case["heads"], case["heads"] * case["dim"]
        channels = inner + 2 * case["state"]
        weights["head"] = _normal(g, (SMALL_VOCAB, W), std)
        weights[p + "ls1"] = _normal(g, (W,), 0.1, 1.0)
        weights[p + "mix.in"] = _normal(g, (inner + channels + H, W), std)
        weights[p + "mix.conv"] = _normal(g, (channels, TAPS), TAPS ** -0.5)
        weights[p + "mix.conv.b"] = _normal(g, (channels,), 0.1)
        # states that remember from a few to hundreds of tokens
        weights[p + "mix.dt_bias"], weights[p + "mix.A_log"] = _normal(g, (H,), 1.0, -3.0), _normal(g, (H,))
        weights[p + "mix.D"], weights[p + "mix.norm"] = _normal(g, (H,), 0.1, 1.0), _normal(g, (inner,), 0.1, 1.0)
        weights[p + "mix.o"] = _normal(g, (W, inner), inner ** -0.5)
    else:
        inner = case["heads"] * case["dim"]
        weights[p + "mix.q"] = _normal(g, (inner, W), std)
        weights[p + "mix.k"] = _normal(g, (case["kv_heads"] * case["dim"], W), std)
        weights[p + "mix.sink"] = _normal(g, (case["heads"],))
        weights[p + "mix.o"] = _normal(g, (W, inner), inner ** -0.5)
    return weights


def _engine(case, config, weights, tokens, requests, budget):
    pages = sum(-(-count // PAGE) for count in tokens) + requests
    return Engine(config, EngineConfig(dtype=case["dtype"], block_size=PAGE, num_blocks=pages, max_num_seqs=requests,
                                       max_num_batched_tokens=budget, max_model_len=8192), tensors=weights)


def _tokens(case, seed):
    """Per request its prompt and the tokens that follow."""
    g = _generator(seed, 3)
    return [torch.randint(VOCAB, (length + case["new"] - 1,), generator=g, device=DEVICE) for length in _lengths(case)]


def _rows(case, seed):
    """What a layer is given: residual rows for a block, normed rows of the compute type for a part."""
    rows = case["tokens"] if case["kind"] == "experts" else sum(_lengths(case))
    x = torch.randn((rows, case["width"]), generator=_generator(seed, 4), device=DEVICE)
    return x if case["kind"] == "block" else x.to(getattr(torch, case["dtype"]))


# ------------------------------------------------------------------------------------------------ running them
def prepare(case, seed):
    if case["kind"] == "serve":
        sequences = [row.cpu().numpy() for row in _tokens(case, seed)]
        engine = _engine(case, _gpt2_config(case, case["layers"], VOCAB), _gpt2_weights(case, case["layers"], VOCAB, seed),
                         [len(row) for row in sequences], case["requests"], case["budget"])
        plan = [[("r%d" % r, sequences[r][begin:end], [end - begin - 1] if wanted else [])
                 for r, begin, end, wanted in step] for step in _schedule(case)]
        return dict(case=case, engine=engine, plan=plan)
    if case["kind"] == "block":
        config, weights = _gpt2_config(case, 1, SMALL_VOCAB), _gpt2_weights(case, 1, SMALL_VOCAB, seed)
    else:
        config = {"experts": _experts_config, "ssm": _ssm_config, "rotary": _rotary_config}[case["kind"]](case)
        weights = _layer_weights(case, seed)
    lengths = [case["tokens"]] if case["kind"] == "experts" else _lengths(case)
    engine = _engine(dict(case), config, weights, lengths, len(lengths), sum(lengths))
    if max(lengths) > engine.max_model_len:
        raise ValueError("a prompt is longer than the model's context")
    # a step that brings the prompts' tokens; the layer runs on its metadata and its pages
    ctx = engine.runner.prepare([StepEntry("r%d" % r, [0] * length) for r, length in enumerate(lengths)])
    engine.runner.begin(ctx)
    layer = LayerContext(0, 0, engine.model.positions, state=engine.cache.state.get(0))
    if engine.cache.groups:
        group = engine.cache.groups[0]
        layer.k_pool, layer.v_pool = group.layer_views(0)
        layer.page_stride, layer.page_size, layer.pool, layer.pool_layer = group.page_stride, group.page_size, group.pool, 0
        layer.block_table = ctx.block_tables[0]
    x = _rows(case, seed)
    return dict(case=case, engine=engine, ctx=ctx, layer=layer, x=x,
                out=torch.empty(x.shape, dtype=torch.float32, device=DEVICE))


def run(state):
    kind, engine = state["case"]["kind"], state["engine"]
    if kind == "serve":
        logits = []
        for entries in state["plan"]:
            rows = engine.step(entries)
            if len(rows):
                logits.append(rows)
        for r in range(state["case"]["requests"]):
            engine.finish("r%d" % r)
        return logits
    block, ctx, layer, x, out = engine.model.blocks[0], state["ctx"], state["layer"], state["x"], state["out"]
    engine.ops.arena.reset()                               # a step's temporary rows begin anew
    if kind == "block":
        out.copy_(x)
        block.forward(out, ctx, layer)
        return out
    out.zero_()                                            # parts add into the residual rows
    if kind == "experts":
        block.feed_forward.forward(x, out, ctx)
        return out
    if kind == "ssm":
        layer.state.zero_()                                # the sequences begin
        block.mixer.forward(x, out, ctx, layer)
        return out, layer.state
    block.mixer.forward(x, out, ctx, layer)
    return out


# ------------------------------------------------------------------------------------------------ what they cost at least
def _attended(begin, end, window=None):
    """Keys that the queries at positions begin .. end - 1 see, added up."""
    if window is None:
        return (end - begin) * (begin + end + 1) // 2
    return sum(min(position + 1, window) for position in range(begin, end))


def work(case):
    size = 2 if case["dtype"] == "bfloat16" else 4
    W = case["width"]
    if case["kind"] == "serve":
        L, flops, moved = case["layers"], 0, 0
        layer_weights = 12 * W * W
        for step in _schedule(case):
            tokens = sum(end - begin for _, begin, end, _ in step)
            rows = sum(wanted for _, _, _, wanted in step)
            flops += 2 * L * layer_weights * tokens + 2 * VOCAB * W * rows
            flops += sum(4 * L * W * _attended(begin, end) for _, begin, end, _ in step)
            # every weight once a step; the keys and values of the contexts, read and written; the logits
            moved += size * (L * layer_weights + (VOCAB * W if rows else 0) + 2 * L * W * (tokens + sum(end for _, _, end, _ in step)))
            moved += 4 * VOCAB * rows
        return dict(bytes=moved, flops=flops)
    if case["kind"] == "experts":
        T, shared, ff = case["tokens"], case["shared"], case["ff"]
        flops = 2 * T * W * (3 * shared + 3 * ff * case["top"] + case["experts"])
        weights = 3 * W * (shared + ff * min(case["experts"], T * case["top"])) + case["experts"] * W
        return dict(bytes=size * (weights + T * W) + 4 * T * W, flops=flops)
    lengths = _lengths(case)
    T = sum(lengths)
    if case["kind"] == "block":
        return dict(bytes=size * (12 * W * W + 2 * T * W) + 8 * T * W,
                    flops=24 * T * W * W + sum(4 * W * _attended(0, length) for length in lengths))
    if case["kind"] == "ssm":
        inner, N = case["heads"] * case["dim"], case["state"]
        rows = 2 * inner + 2 * N + case["heads"]
        return dict(bytes=size * (rows * W + inner * W + T * W) + 4 * T * W + 4 * len(lengths) * inner * N,
                    flops=2 * T * W * (rows + inner) + 4 * T * inner * N + 2 * TAPS * T * (inner + 2 * N))
    inner, kv = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
    return dict(bytes=size * (W * (2 * inner + kv) + T * (W + 2 * kv)) + 4 * T * W,
                flops=2 * T * W * (2 * inner + kv) + sum(4 * inner * _attended(0, n, case["window"]) for n in lengths))


def tolerance(case):
    # about four times what is seen against 64 bits: 1.4e-6 to 2.4e-6 in float32 (sums of 768 to 6,400 numbers, twelve layers of
    # them); in bfloat16 0.0012 for a block (most of its result is the float32 row that it adds to), 0.0028 to 0.0045 elsewhere
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.005 if case["kind"] == "block" else 0.015}


# ------------------------------------------------------------------------------------------------ 64 bits
def _layer_norm(x, weight, bias):
    centred = x - x.mean(-1, keepdim=True)
    return centred / torch.sqrt((centred * centred).mean(-1, keepdim=True) + EPS) * weight + bias


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _heads_softmax(q, k, v, scale, window=None, cap=None, sink=None):
    """q [T, H, d], k and v [T, G, d], one sequence: [T, H * d]."""
    T, H, _ = q.shape
    share = H // k.shape[1]
    i, j = torch.arange(T, device=q.device)[:, None], torch.arange(T, device=q.device)[None]
    unseen = (j > i) if window is None else (j > i) | (i - j >= window)
    rows = []
    for h in range(H):
        s = q[:, h] @ k[:, h // share].T * scale
        if cap is not None:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(unseen, -math.inf)
        top = s.max(-1, keepdim=True).values
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0)
        rows.append((e / total) @ v[:, h // share])
    return torch.cat(rows, -1)


def _gpt2_block(w, p, x, lengths, heads):
    """x [sum of the lengths, W]."""
    W = x.shape[1]
    h = _layer_norm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"])
    qkv = h @ w[p + "attn.c_attn.weight"] + w[p + "attn.c_attn.bias"]
    context = []
    for rows in qkv.split(lengths):
        q, k, v = (part.reshape(len(rows), heads, W // heads) for part in rows.split(W, -1))
        context.append(_heads_softmax(q, k, v, (W // heads) ** -0.5))
    x = x + torch.cat(context) @ w[p + "attn.c_proj.weight"] + w[p + "attn.c_proj.bias"]
    h = _layer_norm(x, w[p + "ln_2.weight"], w[p + "ln_2.bias"])
    return x + _gelu(h @ w[p + "mlp.c_fc.weight"] + w[p + "mlp.c_fc.bias"]) @ w[p + "mlp.c_proj.weight"] + w[p + "mlp.c_proj.bias"]


def _clamped_expert(w, p, x):
    g, u = (x @ w[p + "gate"].T).clamp(max=LIMIT), (x @ w[p + "up"].T).clamp(-LIMIT, LIMIT)
    return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].T


def _experts(case, w, x):
    p = "l0.mlp."
    scores = torch.sigmoid(x @ w[p + "router"].T)
    weight, chosen = scores.topk(case["top"], -1)
    out = _clamped_expert(w, p + "shared.", x)
    for e in range(case["experts"]):
        row, place = (chosen == e).nonzero(as_tuple=True)
        out.index_add_(0, row, _clamped_expert(w, p + "e%d." % e, x[row] * weight[row, place][:, None]))
    return out


def _ssm(case, w, x, lengths):
    H, P, N, p = case["heads"], case["dim"], case["state"], "l0.mix."
    inner, rows = H * P, []
    for part in (x @ w[p + "in"].T).split(lengths):
        T = len(part)
        z, u, dt = part.split([inner, inner + 2 * N, H], -1)
        before = torch.cat([u.new_zeros(TAPS - 1, u.shape[1]), u])
        u = sum(before[j:j + T] * w[p + "conv"][:, j] for j in range(TAPS)) + w[p + "conv.b"]
        xs, b, c = (u * torch.sigmoid(u)).split([inner, N, N], -1)
        dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
        keep, scaled = torch.exp(-torch.exp(w[p + "A_log"]) * dt), dt[:, :, None] * xs.reshape(T, H, P)
        S, y = x.new_zeros(H, P, N), []
        for t in range(T):
            S = torch.addcmul(S * keep[t][:, None, None], scaled[t][:, :, None], b[t])
            y.append(S @ c[t])
        y = torch.stack(y) + w[p + "D"][:, None] * xs.reshape(T, H, P)
        y = y.reshape(T, inner) * z * torch.sigmoid(z)
        y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + EPS) * w[p + "norm"]
        rows.append(y @ w[p + "o"].T * w["l0.ls1"])
    return torch.cat(rows)


def _rotary(case, w, x, lengths):
    H, G, d, p, rows = case["heads"], case["kv_heads"], case["dim"], "l0.mix.", []
    dims = (d // 4) * 2
    for part in x.split(lengths):
        T = len(part)
        q, v = (part @ w[p + "q"].T).reshape(T, H, d), (part @ w[p + "k"].T).reshape(T, G, d)
        angle = torch.arange(T, dtype=x.dtype, device=x.device)[:, None] * ROTARY_BASE ** (
            -torch.arange(0, dims, 2, dtype=x.dtype, device=x.device) / dims)
        cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

        def turned(a):
            out = a.clone()
            out[..., 0:dims:2] = a[..., 0:dims:2] * cos - a[..., 1:dims:2] * sin
            out[..., 1:dims:2] = a[..., 1:dims:2] * cos + a[..., 0:dims:2] * sin
            return out

        rows.append(_heads_softmax(turned(q), turned(v), v, d ** -0.5, case["window"], SOFTCAP, w[p + "sink"]) @ w[p + "o"].T)
    return torch.cat(rows)


def exact(case, seed):
    if case["kind"] == "serve":
        w = {name: value.double() for name, value in _gpt2_weights(case, case["layers"], VOCAB, seed).items()}
        sequences = _tokens(case, seed)
        lengths = [len(row) for row in sequences]
        x = torch.cat([w["wte.weight"][row] + w["wpe.weight"][:len(row)] for row in sequences])
        for layer in range(case["layers"]):
            x = _gpt2_block(w, "h.%d." % layer, x, lengths, case["heads"])
        x = _layer_norm(x, w["ln_f.weight"], w["ln_f.bias"]).split(lengths)
        steps = [[x[r][end - 1] for r, _, end, wanted in step if wanted] for step in _schedule(case)]
        return [torch.stack(rows) @ w["wte.weight"].T for rows in steps if rows]
    x = _rows(case, seed).double()
    if case["kind"] == "block":
        w = {name: value.double() for name, value in _gpt2_weights(case, 1, SMALL_VOCAB, seed).items()}
        return _gpt2_block(w, "h.0.", x, _lengths(case), case["heads"])
    w = {name: value.double() for name, value in _layer_weights(case, seed).items()}
    if case["kind"] == "experts":
        return _experts(case, w, x)
    if case["kind"] == "ssm":
        return _ssm(case, w, x, _lengths(case)), None
    return _rotary(case, w, x, _lengths(case))
