"""Scores past a sequence's end (-inf, written by the scan's own blocks) and the row statistics at the edges of what
their kernel holds in registers."""
import pytest
import torch

from jf_testlib import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,ctx,lens", [
    ("k3v2", 20000, [20000, 6001, 0, 1, 19999]),     # blocks shared out by length
    ("k3v2", 100, [100, 3, 0]),                      # one block a sequence
    ("k4v4", 5003, [5003, 17, 0, 4000]),
])
def test_scores_past_the_end(mode, ctx, lens):
    from jetfire_b200 import ops
    case = Case(mode, len(lens), 32, 8, ctx, lens=lens, seed=1)
    cache = case.device_cache()
    args = (case.block_table.cuda(), case.seq_lens.cuda(), ctx, 32, 8, 16)
    full = ops.fused_attn_topk(mode, case.q.cuda(), *cache, *args, 32, case.attn_scale, want_scores=True).scores
    if mode == "k3v2":
        alone = ops.int3_qk_scores_topk(case.q.cuda(), *cache[:2], *args, case.attn_scale, 32)[0]
    else:
        alone = ops.int8tc_qk_scores_topk_stats(case.q.cuda(), *cache[:2], *args, case.attn_scale, 32)[0]
    for b, n in enumerate(lens):
        for s in (full, alone):
            assert torch.isneginf(s[b, :, n:]).all() and torch.isfinite(s[b, :, :n]).all()


@pytest.mark.parametrize("max_S", [1, 511, 8191, 8192, 8193, 20001])
def test_row_statistics(max_S):
    from jetfire_b200 import _lib
    g = torch.Generator().manual_seed(max_S)
    s = (3.0 * torch.randn(3, 4, max_S, generator=g)).cuda()
    lens = torch.tensor([max_S, max_S // 2, 0], dtype=torch.int32, device="cuda")
    s[0, 1, : max_S // 3] = float("-inf")
    s[0, 2] = float("-inf")
    m, inv = torch.empty(3, 4, device="cuda"), torch.empty(3, 4, device="cuda")
    st = _lib.lib.jf_softmax_stats(s.data_ptr(), lens.data_ptr(), m.data_ptr(), inv.data_ptr(), 3, 4, max_S,
                                   torch.cuda.current_stream().cuda_stream)
    assert st == 0
    for b in range(3):
        n = int(lens[b])
        for h in range(4):
            row = s[b, h, :n].double()
            if n == 0 or bool(torch.isneginf(row).all()):
                assert m[b, h] == 0 and inv[b, h] == 0
                continue
            assert m[b, h] == row.max().float()
            # exp's bound of 2 + |x| units in fp32 and a sum of positive terms: 2e-5 for scores within 15 of the maximum's
            want = 1.0 / torch.exp(row - row.max()).sum()
            assert abs(float(inv[b, h]) - float(want)) <= 2e-5 * float(want)


@pytest.mark.parametrize("mode", ["k3v2", "k4v4"])
@pytest.mark.parametrize("B,H_q,H_kv,max_S", [(4, 8, 2, 97), (3, 8, 2, 1022), (3, 16, 2, 4003),
                                              (64, 16, 2, 131071)])   # more than 512 MB of scores: a kernel of its own
def test_tails_at_every_alignment(mode, B, H_q, H_kv, max_S):
    from jetfire_b200 import ops
    g = torch.Generator().manual_seed(B)
    lens = [max(0, n) for n in (max_S - 1, 0, 1, max_S - 5, 7, max_S // 2 + 1, max_S, 18)][:min(B, 8)]
    lens = torch.tensor((lens * B)[:B], dtype=torch.int32)
    table = torch.randint(0, 256, (B, (max_S + 15) // 16), generator=g)
    row = {"k3v2": (48, 2), "k4v4": (64, 1)}[mode]
    kd = torch.randint(0, 256, (H_kv, 4096, row[0]), dtype=torch.uint8, generator=g)
    ks = torch.rand(H_kv, 4096, row[1], generator=g).bfloat16()
    q = torch.randn(B, H_q, 128, generator=g).bfloat16()
    stage_a = ops.int3_qk_scores_topk if mode == "k3v2" else ops.int8tc_qk_scores_topk_stats
    scores = stage_a(q.cuda(), kd.cuda(), ks.cuda(), table.cuda(), lens.cuda(), max_S, H_q, H_kv, 16, 0.1, 8)[0]
    past = torch.arange(max_S, device="cuda") >= lens.cuda()[:, None]
    for b in range(B):
        assert torch.isneginf(scores[b][:, past[b]]).all() and torch.isfinite(scores[b][:, ~past[b]]).all()
