"""Scratch of the one-shot ops under stream capture: a graph must not write to the block that later eager
calls on the stream are given (and that may go back to the allocator), and its replays give the eager bits."""
import pytest
import torch

from jf_testlib import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["k3v2", "k4v4"])
def test_a_captured_call_has_scratch_of_its_own(mode):
    from jetfire_b200 import ops
    case = Case(mode, 2, 8, 2, 3000, lens=[3000, 777], seed=12)
    kd, ks, vd, vs = case.device_cache()
    q, bt, lens = case.q.cuda(), case.block_table.cuda(), case.seq_lens.cuda()
    call = lambda: ops.int2_fused_attn_topk(q, kd, ks, None, vd, vs, bt, lens, case.ctx, 8, 2, 16, 64, case.attn_scale)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = [t.clone() for t in call()]
        table_block = ops.get_workspace(1, "cuda")
        assert table_block.numel() >= ops.decode_workspace_bytes(mode, 2, 8, 2, case.ctx, 64)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = call()
        table_block.fill_(0x5A)
        graph.replay()
        side.synchronize()
        assert bool((table_block == 0x5A).all())
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        other = torch.full_like(table_block, 0x33)       # whatever the allocator hands out now is not the graph's
        graph.replay()
        side.synchronize()
        assert bool((other == 0x33).all())
    del graph
