"""Ragged batches whose rows are long enough for the scan's blocks to be shared out by length, at the edges
of that rule: empty sequences first and last, single tokens, a sequence past the first 32, one long row
among empty ones, rows of one unit less than the longest."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu

CTX = 11000   # 344 units of two pages: more than 24 for each of the 7 blocks of 40 sequences x 2 KV heads

MIXED = [0, 1, 17, 33, CTX, 4097, 32, 0] + [97 * i for i in range(1, 30)] + [CTX - 1, 16, 0]


@pytest.mark.parametrize("mode,stage_b,dtype", [
    ("k3v2", "fp32", torch.bfloat16), ("k3v2", "fp32", torch.float16),
    ("k4v4", "fp32", torch.bfloat16), ("k4v4", "int8p", torch.bfloat16),
])
@pytest.mark.parametrize("lens", [MIXED, [0] * 35 + [CTX] + [0] * 4, [CTX] * 39 + [CTX - 32], [CTX - 5] * 40, [0] * 40],
                         ids=["mixed", "one", "unit", "full", "none"])
def test_shares_by_length(mode, stage_b, dtype, lens):
    case = Case(mode, 1, 4, 2, CTX, seed=len(set(lens)), dtype=dtype)
    g = torch.Generator().manual_seed(21)
    case.B = len(lens)                                   # the sequences' rows are shuffles of the same blocks
    case.q = torch.randn(case.B, 4, 128, generator=g).to(dtype)
    n = (CTX + 15) // 16
    case.block_table = torch.stack([torch.randperm(case.n_blocks, generator=g)[:n] for _ in lens]).to(torch.int64)
    case.seq_lens = torch.tensor(lens, dtype=torch.int32)
    _run(case, 64, stage_b)
