"""What the scans leave in the workspace: partials of the heads of the group, and nothing in the places of the others."""
import pytest
import torch

from jf_testlib import Case

pytestmark = pytest.mark.gpu
FILL = 0x7B


@pytest.mark.parametrize("mode,group,parts", [("k3v2", 1, "all"), ("k3v2", 4, "all"), ("k3v2", 5, "all"), ("k3v2", 3, "v"), ("k4v4", 2, "all"),
                                              ("k4v4", 4, "v"), ("k4v4", 7, "all"), ("k3v2", 8, "all"), ("k4v4", 8, "all")])
def test_only_the_heads_of_the_group(mode, group, parts):
    from jetfire_b200 import ops
    case = Case(mode, 2, 2 * group, 2, 3000, seed=group)
    ws = torch.full((ops.decode_workspace_bytes(mode, 2, case.H_q, 2, case.ctx, 32) + 256,), FILL, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    args = (case.q.cuda(), *case.device_cache(), case.block_table.cuda(), case.seq_lens.cuda(), case.ctx, case.H_q, 2, 16, 32, case.attn_scale)
    scores = None
    if parts == "v":   # from the scores of an earlier call
        scores = ops.fused_attn_topk(mode, *args, want_scores=True).scores
    call = ops.DecodeCall(mode, *args, workspace=ws, parts=parts, scores=scores)
    call.scan()
    first = ws[256:256 + 8 * 128 * 4].view(torch.float32).reshape(8, 128)   # after the status record: the first CTA's output rows
    empty = torch.full((4,), FILL, dtype=torch.uint8).view(torch.float32).item()
    assert (first[group:] == empty).all()
    assert torch.isfinite(first[:group]).all() and (first[:group] != empty).all()
