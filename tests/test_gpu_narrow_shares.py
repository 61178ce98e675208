"""K3V2 with at most four query heads per KV head in a long ragged batch: the scan's blocks are shared out among the
sequences by their lengths, for every group size and both query types."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu
B, H_KV, CTX = 5, 8, 20000


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group", [1, 2, 3, 4])
def test_blocks_shared_out_by_length(dtype, group):
    # one wave of four blocks a multiprocessor: 24 units of two pages a block is where shares begin
    splits = 4 * torch.cuda.get_device_properties(0).multi_processor_count // (B * H_KV)
    assert -(-(CTX // 32) // splits) >= 24
    _run(Case("k3v2", B, H_KV * group, H_KV, CTX, lens=[CTX, 9001, 161, 0, 14999], seed=group, dtype=dtype), 32)
