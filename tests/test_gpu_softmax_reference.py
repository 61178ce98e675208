"""W against the softmax of the scan's own scores in 64 bits, with scores so large that the rounding of
score * log2(e) matters: a reference point m has m * log2(e) rounded to 2^-24 of itself, 2.6e-6 of a weight at
m = 80, and that has to cancel between the selected entries and the normaliser."""
import pytest
import torch

from jf_testlib import Case

pytestmark = pytest.mark.gpu

# What is left per weight: the exponent fma's own rounding (half an ulp of a number below 4 for the weights
# that count: 1.2e-7 * ln 2), log2(e) as a float (1.3e-8 relative, times a difference of scores below 8),
# exp2 (2^-22.5) and the sums (a few 2^-24).
LIMIT = 8e-7


@pytest.mark.parametrize("mode,dtype", [("k3v2", torch.bfloat16), ("k3v2", torch.float16), ("k4v4", torch.bfloat16)])
@pytest.mark.parametrize("lens", [[700, 33], [20000, 12345, 7000]], ids=["short", "long"])
def test_weights_sum_with_large_scores(mode, dtype, lens):
    from jetfire_b200 import ops
    case = Case(mode, len(lens), 16, 2, max(lens), lens=lens, seed=31, dtype=dtype)
    kd, ks, vd, vs = case.device_cache()
    res = ops.fused_attn_topk(mode, case.q.cuda(), kd, ks, vd, vs, case.block_table.cuda(), case.seq_lens.cuda(), case.ctx,
                              16, 2, 16, 64, 16.0 * case.attn_scale, want_scores=True)
    p = torch.softmax(res.scores.double(), dim=-1)                       # -inf past each sequence
    want = torch.gather(p, 2, res.topk_idx.clamp_min(0)).mul(res.topk_idx >= 0).sum(-1)
    assert res.scores.amax() > 60.0
    err = ((res.W.double() - want) / want).abs().max().item()
    assert err < LIMIT, f"{err:.2e}"


@pytest.mark.parametrize("mode", ["k3v2", "k4v4"])
def test_many_weights_of_one_size(mode):
    """4096 nearly equal weights: a running sum of their 128 partial sums rounds once per term at the full size
    (1.8e-7 rms over the rows), pairwise sums seven times; with the scan's own sums 7.5e-8 is left, 2^-23 allowed."""
    from jetfire_b200 import ops
    case = Case(mode, 2, 32, 4, 8192, lens=[8192, 8000], seed=33)
    kd, ks, vd, vs = case.device_cache()
    res = ops.fused_attn_topk(mode, case.q.cuda(), kd, ks, vd, vs, case.block_table.cuda(), case.seq_lens.cuda(), case.ctx,
                              32, 4, 16, 4096, 0.02 * case.attn_scale, want_scores=True)
    p = torch.softmax(res.scores.double(), dim=-1)
    want = torch.gather(p, 2, res.topk_idx.clamp_min(0)).mul(res.topk_idx >= 0).sum(-1)
    rms = ((res.W.double() - want) / want).square().mean().sqrt().item()
    assert rms < 1.2e-7, f"{rms:.2e}"
