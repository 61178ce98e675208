"""The select kernel's blocks at the edges of their ranges: rows that just fit a chunk of either width or
one position more, and rows of mostly equal scores, whose selection is decided by position alone."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["k3v2", "k4v4"])
@pytest.mark.parametrize("ctx,top_k", [(1023, 512), (2049, 33), (16384, 64), (16385, 64), (32768, 512), (32769, 512)])
def test_chunk_edges(mode, ctx, top_k):
    _run(Case(mode, 1, 4, 2, ctx, lens=[ctx], seed=ctx), top_k)


@pytest.mark.parametrize("ctx", [5000, 20000, 40000])
def test_ties_go_to_the_lower_position(ctx):
    case = Case("k4v4", 1, 4, 2, ctx, lens=[ctx - 3], seed=9)
    g = torch.Generator().manual_seed(10)
    few = case.k_full[:, torch.randperm(case.num_slots, generator=g)[:3]]           # three distinct keys per head
    case.k_full = few[:, torch.randint(0, 3, (case.num_slots,), generator=g)].contiguous()
    _run(case, 64)
