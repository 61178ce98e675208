"""Block ids inside a sequence that name no block of the cache: their positions score -inf and are never selected, whatever
the workspace held before, on every path of the selection."""
import numpy as np
import pytest
import torch

from oracle import native
from jf_testlib import Case, f32_values, to_bits

pytestmark = pytest.mark.gpu


def _holes(case, every):
    """Every `every`-th page and two neighbours are no blocks; the last page of the first sequence is one of them."""
    table = case.block_table.clone()
    table[:, 3::every] = -1
    table[:, 8:10] = case.n_blocks
    table[0, (int(case.seq_lens[0]) - 1) // 16] = 2 ** 40
    return table


CASES = [
    ("k3v2", "fp32", 1, 8, 2, 300, 64, torch.bfloat16),        # every position is a candidate
    ("k3v2", "fp32", 3, 8, 2, 2001, 64, torch.bfloat16),       # one staged chunk, narrow groups
    ("k3v2", "fp32", 3, 8, 2, 2001, 64, torch.float16),
    ("k3v2", "fp32", 2, 16, 2, 2001, 64, torch.bfloat16),      # wide groups
    ("k3v2", "fp32", 2, 16, 2, 2001, 64, torch.float16),
    ("k3v2", "fp32", 1, 8, 2, 40000, 64, torch.bfloat16),      # from page maxima
    ("k3v2", "fp32", 5, 32, 2, 1600, 64, torch.float16),       # rows share a multiprocessor: close candidates re-scored
    ("k3v2", "fp32", 6, 32, 8, 33008, 257, torch.bfloat16),    # from page maxima, every candidate re-scored
    ("k4v4", "fp32", 1, 8, 2, 2001, 64, torch.bfloat16),
    ("k4v4", "int8p", 3, 8, 2, 6007, 64, torch.bfloat16),
    ("k4v4", "int8p", 2, 16, 2, 6007, 64, torch.bfloat16),
    ("k4v4", "int8p", 2, 8, 2, 40000, 64, torch.bfloat16),
]


@pytest.mark.parametrize("mode,stage_b,B,H_q,H_kv,ctx,top_k,dtype", CASES)
def test_positions_without_a_block(mode, stage_b, B, H_q, H_kv, ctx, top_k, dtype):
    from jetfire_b200 import ops
    case = Case(mode, B, H_q, H_kv, ctx, seed=ctx, dtype=dtype)
    cache = case.device_cache()
    kd, ks, vd, vs = cache
    ref = native.c_decode(mode, f32_values(case.q), kd.cpu().numpy(), to_bits(ks), vd.cpu().numpy(), to_bits(vs), case.block_table.numpy(),
                          case.seq_lens.numpy(), ctx, top_k, case.attn_scale, want_scores=True)["scores"]
    table = _holes(case, 50 if ctx > 1000 else 7)
    pages = table.numpy()
    bad = np.repeat((pages < 0) | (pages >= case.n_blocks), 16, 1)[:, :ctx]
    tail = (table.cuda(), case.seq_lens.cuda(), ctx, H_q, H_kv, 16)
    ws = torch.full((ops.decode_workspace_bytes(mode, B, H_q, H_kv, ctx, top_k) // 4 + 64,), 1e4, device="cuda").view(torch.uint8)
    inner = ops.fused_attn_topk(mode, case.q.cuda(), *cache, *tail, top_k, case.attn_scale, workspace=ws, stage_b=stage_b)
    seen = ops.fused_attn_topk(mode, case.q.cuda(), *cache, *tail, top_k, case.attn_scale, want_scores=True, stage_b=stage_b)
    idx, slots, scores = inner.topk_idx.cpu().numpy(), inner.topk_slots.cpu().numpy(), seen.scores.cpu().numpy()
    for b in range(B):
        n = int(case.seq_lens[b])
        row = np.where(bad[b, :n], -np.inf, ref[b, :, :n])
        want = np.argsort(-row, axis=1, kind="stable")[:, :top_k]
        assert np.isfinite(np.take_along_axis(row, want, 1)).all()
        assert np.array_equal(idx[b], want)
        assert np.array_equal(slots[b], pages[b][want // 16] * 16 + want % 16)
    for b in range(B):
        n = int(case.seq_lens[b])
        assert np.isneginf(scores[b][:, bad[b]]).all() and np.isneginf(scores[b, :, n:]).all()
        assert np.isfinite(scores[b, :, :n][:, ~bad[b, :n]]).all()
    assert torch.equal(inner.topk_idx, seen.topk_idx)
    # the calls may cut their work differently: fp16 weights relative to other reference points
    for a, c in ((inner.o_hat, seen.o_hat), (inner.o_old_unnorm, seen.o_old_unnorm), (inner.W, seen.W)):
        assert torch.isfinite(a).all() and torch.allclose(a, c, atol=2e-3, rtol=1e-3)
