"""K3V2, a wide top-k of long rows, more rows than multiprocessors, threshold from the scan's page maxima: candidates are cut
down by their scan scores before their rows are read.  Lists must be the oracle's where the K-th score is one of many equal
or nearly equal ones, for both query types, and where pages inside a sequence have no block."""
import pytest
import torch

import test_gpu_invalid_blocks as invalid_blocks
from jf_testlib import Case
from test_gpu_close_candidates import _few_keys
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu
B, H_Q, CTX = 5, 32, 49168


def _check_route(top_k):
    """More than 256 entries: sort buffer of 1024; page pairs enough for the threshold; rows that share a multiprocessor."""
    assert 384 <= top_k <= 512 and CTX % 16 == 0 and CTX // 32 >= 4 * top_k
    assert B * H_Q > torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H_kv,distinct,jitter", [
    (8, 0, 0.0),          # narrow groups
    (4, 0, 0.0),          # wide groups
    (4, 8000, 0.0),       # six equal scores everywhere, among them at the K-th
    (4, 8000, 4e-3),      # ... and as many whose scales lie a bf16 step or two apart
    (4, 40, 1e-3),        # crowds of hundreds: more candidates than the sort buffer holds
])
def test_lists_are_the_oracles(dtype, H_kv, distinct, jitter):
    _check_route(384)
    case = Case("k3v2", B, H_Q, H_kv, CTX, lens=[CTX, CTX - 1, 1025, 300, 20000], seed=12, dtype=dtype)
    _run(_few_keys(case, distinct, jitter) if distinct else case, 384)


def test_positions_without_a_block():
    _check_route(384)
    invalid_blocks.test_positions_without_a_block("k3v2", "fp32", B, H_Q, 8, CTX, 384, torch.bfloat16)
