"""The state-space recurrence over more prompt entries than a grid's second dimension counts, and over more than its CTAs sort by
length."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("entries,heads", [(255, 3), (256, 2), (257, 2), (65536, 1), (70001, 1)])
def test_single_tokens_as_prompt_entries(entries, heads):
    from pagedserve_b200.kernels.ops import Ops

    N, P, g = 16, 16, torch.Generator().manual_seed(entries)
    inner = heads * P
    conv = torch.randn(entries, inner + 2 * N, generator=g).to(torch.bfloat16).to(DEV)
    raw = torch.randn(entries, 2 * inner, generator=g).to(torch.bfloat16).to(DEV)                # z, then dt
    a_log, dt_bias, d = (torch.randn(heads, generator=g).to(DEV) for _ in range(3))
    state = torch.randn(entries + 2, heads * N * P, generator=g).to(DEV)
    slots = torch.randperm(entries + 2, generator=g)[:entries].to(DEV)
    ctx = SimpleNamespace(max_q_len=1, q_start=torch.arange(entries + 1, dtype=torch.int32, device=DEV), item_slot=slots.to(torch.int32),
                          num_items=entries, num_short_items=0, num_short_tokens=0)
    x, b, c = conv[:, :inner].double().view(entries, heads, 1, P), conv[:, inner:inner + N].double(), conv[:, inner + N:].double()
    z, dt = raw[:, :inner].double(), torch.nn.functional.softplus(raw[:, inner:inner + heads].double() + dt_bias.double())
    S = state[slots].double().view(entries, heads, N, P) * torch.exp(-dt * torch.exp(a_log.double()))[:, :, None, None]
    S = S + dt[:, :, None, None] * b[:, None, :, None] * x
    y = (c[:, None, :, None] * S).sum(2) + d.double()[None, :, None] * x[:, :, 0]
    want = y.reshape(entries, inner) * z * torch.sigmoid(z)
    out = torch.empty(entries, inner, device=DEV)
    Ops(torch.bfloat16).ssd(conv, raw, (0, inner, inner + N, 0, inner), a_log, dt_bias, d, state, ctx, out, heads, 1, N, P)
    # float32 sums of 16 products, operands in pieces that hold all of their 24 bits
    assert float((out.double() - want).abs().max()) < 2e-5 * float(want.abs().max())
    assert float((state[slots].double().view_as(S) - S).abs().max()) < 5e-6 * float(S.abs().max())
