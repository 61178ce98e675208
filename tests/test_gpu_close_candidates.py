"""K3V2 rows that share a multiprocessor (more rows than there are): of a row's candidates only those whose scan
scores are close to another one's are re-scored, or they are cut down by their scan scores first.  Lists must still be the
oracle's where scores tie, crowd together or are so large that every candidate is re-scored, and name positions of the
row whatever the scores are."""
import numpy as np
import pytest
import torch

from oracle import native
from jf_testlib import Case, f32_values, to_bits
from test_gpu_decode_parity import k3_score_bound, run_gpu
from test_gpu_long_rows import _run, _select_us

pytestmark = pytest.mark.gpu
B, H_Q, H_KV = 5, 32, 2    # 160 rows


def _few_keys(case, distinct, jitter=0.0):
    g = torch.Generator().manual_seed(3)
    rows = case.k_full[:, torch.randperm(case.num_slots, generator=g)[:distinct]]
    k = rows[:, torch.randint(0, distinct, (case.num_slots,), generator=g)].float()
    case.k_full = (k * (1.0 + jitter * torch.randn(k.shape[:2] + (1,), generator=g))).to(case.dtype).contiguous()
    return case


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ctx,top_k", [(1600, 256), (1601, 64), (17008, 128)])
def test_lists_are_the_oracles(dtype, ctx, top_k):
    _run(Case("k3v2", B, H_Q, H_KV, ctx, lens=[ctx, ctx - 1, 513, 512, 33], seed=ctx, dtype=dtype), top_k)


@pytest.mark.parametrize("distinct,jitter", [(40, 0.0), (8, 1e-3), (700, 0.0)])
def test_ties_and_crowds(distinct, jitter):
    _run(_few_keys(Case("k3v2", B, H_Q, H_KV, 2000, seed=4), distinct, jitter), 128)


def test_scores_whose_band_spans_bins():
    case = Case("k3v2", B, H_Q, H_KV, 1500, seed=5)
    case.k_full = (case.k_full.float() * 300.0).to(case.dtype)
    res, (kd, ks, vd, vs) = run_gpu(case, 128)
    ref = native.c_decode("k3v2", f32_values(case.q), kd.cpu().numpy(), to_bits(ks), vd.cpu().numpy(), to_bits(vs),
                          case.block_table.numpy(), case.seq_lens.numpy(), case.ctx, 128, case.attn_scale, want_scores=True)
    assert np.array_equal(res.topk_idx.cpu().numpy(), ref["topk_idx"])
    for b in range(B):   # sums of terms of some thousands: fp32 orders differ by the bound that the selection goes by
        n = int(case.seq_lens[b])
        err = np.abs(res.scores.cpu().numpy()[b, :, :n] - ref["scores"][b, :, :n])
        assert (err <= k3_score_bound(case, to_bits(ks), b, n)[:, None]).all()


@pytest.mark.parametrize("few", [False, True])
def test_wide_top_k_of_a_cache_beyond_l2(few):
    """5 x 10 KV heads x 33008 positions x 88 bytes = 145 MB: candidates are cut down before their rows are read."""
    case = Case("k3v2", B, 40, 10, 33008, lens=[33008, 33007, 1025, 300, 20000], seed=12)
    _run(_few_keys(case, 5000) if few else case, 400)


def test_scores_of_another_cache_select_positions_of_the_row():
    from jetfire_b200 import ops
    calls = []
    for seed in (6, 7):
        c = Case("k3v2", B, H_Q, H_KV, 1600, seed=seed)
        calls.append(ops.DecodeCall("k3v2", c.q.cuda(), *c.device_cache(), c.block_table.cuda(), c.seq_lens.cuda(), c.ctx, H_Q, H_KV, 16,
                                    256, c.attn_scale))
    calls[0].scan()              # both calls use the stream's workspace
    calls[1].select_finish()
    idx = calls[1].out["topk_idx"].cpu()
    lens = c.seq_lens[:, None, None]
    assert ((idx >= 0) & (idx < lens)).all()


def test_rows_of_ties_take_their_time_from_the_candidates():
    """Hundreds of candidates in one bin of the ranking: 2.2 times an ordinary row (3.1 when a bin is counted one by one)."""
    ordinary, ties = (Case("k4v4", 1, H_Q, 8, 8192, lens=[8192], seed=3) for _ in range(2))
    assert _select_us(_few_keys(ties, 4), 512, reps=20) <= 2.7 * _select_us(ordinary, 512, reps=20)
