"""K3V2 with at most four query heads per KV head, which the scan repeats on its unused columns: every group size, both
query types, ragged ends, blocks shared out by length, and the two-stage order's halves."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ctx,lens", [(700, [700, 33, 0]), (20001, [20001, 9000, 161])])
def test_group_sizes(dtype, group, ctx, lens):
    _run(Case("k3v2", len(lens), 2 * group, 2, ctx, lens=lens, seed=group, dtype=dtype), 32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_halves(dtype):
    from jetfire_b200 import ops
    case = Case("k3v2", 2, 6, 2, 1500, seed=8, dtype=dtype)
    kd, ks, vd, vs = case.device_cache()
    tail = (case.block_table.cuda(), case.seq_lens.cuda(), case.ctx, case.H_q, case.H_kv, 16)
    whole = ops.fused_attn_topk("k3v2", case.q.cuda(), kd, ks, vd, vs, *tail, 64, case.attn_scale)
    scores, idx, slots = ops.int3_qk_scores_topk(case.q.cuda(), kd, ks, *tail, case.attn_scale, 64)
    o_hat, o_old, w = ops.int2_softmax_v_with_pre_corr_wvs2(scores, vd, vs, *tail[:2], idx, *tail[2:], 64)
    assert torch.equal(idx, whole.topk_idx) and torch.equal(slots, whole.topk_slots)
    # the same weights as fp16 numbers relative to reference points that may differ: 2^-11 of each, 2e-3 of the gate
    for got, want in ((o_hat, whole.o_hat), (o_old, whole.o_old_unnorm), (w, whole.W)):
        assert torch.allclose(got, want, atol=2e-3, rtol=1e-3)
