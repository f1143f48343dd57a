"""The router of a layer of experts (csrc/moe.cu) with several tokens a CTA against one token a CTA."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [1185, 1187, 2048])
@pytest.mark.parametrize("width,experts,top,groups,keep,score,shared,norm", [
    (72, 8, 2, 0, 0, "softmax", True, True), (1024, 9, 3, 0, 0, "sigmoid", False, False), (250, 7, 7, 0, 0, "softmax", True, False),
    (512, 256, 8, 8, 3, "sigmoid", False, True), (2056, 16, 1, 4, 1, "softmax", False, False)])
def test_many_tokens_are_the_bits_of_few(dtype, tokens, width, experts, top, groups, keep, score, shared, norm):
    """More tokens than a wave of CTAs (the last CTA's tokens not all there), batches of experts that end early, rows of any width."""
    from pagedserve_b200.kernels.ops import Ops

    ops, g = Ops(dtype), torch.Generator(device=DEV).manual_seed(width + experts)
    normal = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    x, router, raw, gain = normal(tokens, width).to(dtype), (normal(experts, width) / width ** 0.5).to(dtype), normal(tokens, width), normal(width)
    gate = normal(width).to(dtype) if shared else None

    def run(begin, end):
        rows = x[begin:end].clone()
        count = end - begin
        dense, chosen = torch.full((count, experts), float("nan"), device=DEV), torch.full((count, top), -9, dtype=torch.int32, device=DEV)
        weights, shared_out = torch.full((count, top), float("nan"), device=DEV), torch.full((count,), float("nan"), device=DEV)
        ops.moe_route(rows, router, gate, dense, chosen, weights, shared_out if shared else None, top, groups, keep,
                      norm=(raw[begin:end], gain, 1e-5) if norm else None, score=score)
        return [rows, dense, chosen, weights] + ([shared_out] if shared else [])

    whole, parts = run(0, tokens), [run(begin, min(begin + 500, tokens)) for begin in range(0, tokens, 500)]
    for i, result in enumerate(whole):
        assert not result.isnan().any()
        assert torch.equal(result, torch.cat([part[i] for part in parts])), i
