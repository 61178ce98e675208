"""K4V4 groups of at most four query heads, whose two pages of a tile share the eight columns: every group size, last pages and
tiles that a boundary of the reference's splits cuts, an odd page, short and empty sequences, both weight arithmetics."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_decode_parity import check_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage_b", ["fp32", "int8p"])
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ctx,lens", [(17, [17, 16, 0]), (1001, [1001, 993, 31]), (6007, [6007, 4097, 5000])])
def test_group_sizes(stage_b, group, ctx, lens):
    check_case(Case("k4v4", len(lens), 2 * group, 2, ctx, lens=lens, seed=group), 16, stage_b=stage_b)


@pytest.mark.parametrize("stage_b,ctx,lens", [("fp32", 2049, [2049]), ("int8p", 6007, [6007, 4097, 31]), ("int8p", 40000, [40000, 39990])])
@pytest.mark.parametrize("parts", ["all", "halves"])
def test_outputs_are_those_of_wide_groups(stage_b, ctx, lens, parts):
    """Four heads on their own and twice over in a group of eight: the same sums in the same order, to the bit."""
    from jetfire_b200 import ops
    case = Case("k4v4", len(lens), 8, 2, ctx, lens=lens, seed=ctx)
    kd, ks, vd, vs = case.device_cache()
    tail = (case.block_table.cuda(), case.seq_lens.cuda(), ctx)
    got = []
    for q in (case.q, case.q.reshape(-1, 2, 4, 128).repeat(1, 1, 2, 1).reshape(-1, 16, 128)):
        args = (*tail, q.shape[1], 2, 16)   # table, lengths, ...
        if parts == "all":
            r = ops.fused_attn_topk("k4v4", q.cuda(), kd, ks, vd, vs, *args, 32, case.attn_scale, stage_b=stage_b)
            out = (r.o_hat, r.o_old_unnorm, r.W)
        else:
            scores, idx, _, m, inv_z = ops.int8tc_qk_scores_topk_stats(q.cuda(), kd, ks, *args, case.attn_scale, 32)
            if stage_b == "int8p":
                out = ops.int8tc_softmax_v_with_pre_corr_reg_stats(scores, m, inv_z, vd, vs, *tail[:2], idx, *args[2:], 32)
            else:
                out = ops.int4_softmax_v_with_pre_corr_wvs2_scores(scores, vd, vs, *tail[:2], idx, *args[2:], 32)
        got.append([x.cpu() for x in out])
    for narrow, wide in zip(*got):
        wide = wide.reshape(wide.shape[0], 2, 8, *wide.shape[2:])[:, :, :4].reshape(narrow.shape)
        assert torch.equal(narrow, wide)
