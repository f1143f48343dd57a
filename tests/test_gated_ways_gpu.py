"""The two ways to a gated activation of many rows, the product that forms it and the product with a gate kernel behind it: each
against a plain implementation, whichever the rule would take."""

import pytest
import torch

import test_zositar_gpu as zositar
from pagedserve_b200.kernels.ops import Ops

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("which,count", [("a", 300), ("b", 129), ("m", 260)])
def test_experts_either_way(monkeypatch, which, count, fused):
    calls = []
    gated, by_rows = Ops.linear_gated, Ops.moe_gate_mul_rows
    monkeypatch.setattr(Ops, "gated_pays", lambda self, rows, columns: fused)
    monkeypatch.setattr(Ops, "linear_gated", lambda self, *args, **options: calls.append(True) or gated(self, *args, **options))
    monkeypatch.setattr(Ops, "moe_gate_mul_rows", lambda self, *args, **options: calls.append(False) or by_rows(self, *args, **options))
    zositar.test_experts_with_many_tokens(which, count, "bfloat16", 1.2e-2)
    assert calls and all(call == fused for call in calls)


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 3e-6), (torch.bfloat16, 4.5e-3)])      # (bfloat16 rounds at 2^-9 of a result)
@pytest.mark.parametrize("rows,columns", [(1, 1), (7, 33), (130, 40), (65, 1024)])
def test_gate_kernel_over_rows(dtype, tol, rows, columns):
    """Every width and both types; rows of weight zero give zeros whatever stands in them."""
    ops, g = Ops(dtype), torch.Generator().manual_seed(rows + columns)
    both = (torch.randn(rows, 2 * columns, generator=g) * 2).to(dtype).to(DEV)
    weight = torch.rand(rows, generator=g).to(DEV) + 0.1
    weight[3::7] = 0.0
    both[3::7] = float("nan")
    gate, up, by = both[:, :columns].double(), both[:, columns:].double(), weight[:, None].double()
    for form, want in (("silu", gate * torch.sigmoid(gate) * up * by),
                       ("gelu_tanh", torch.nn.functional.gelu(gate, approximate="tanh") * up * by),
                       (("clamped_swish", 1.5, 1.0, 1.702), (gate * by).clamp(max=1.5) * torch.sigmoid(1.702 * (gate * by).clamp(max=1.5))
                        * ((up * by).clamp(-1.5, 1.5) + 1))):
        inner = torch.empty(rows, columns, dtype=dtype, device=DEV)
        ops.moe_gate_mul_rows(both, weight, inner, form=form)
        want = torch.where(by == 0, torch.zeros_like(want), want)
        assert float((inner.double() - want).abs().max()) <= tol * max(float(want.abs().max()), 1e-3), form
