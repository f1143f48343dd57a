"""Prompt attention on tcgen05 (csrc/attention_prefill_tc.cu) where it takes one way or another by its data: capped scores by
multiply-adds or by special functions, softmax bases that stay behind the maximum, more portions than a warp has lanes."""

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
