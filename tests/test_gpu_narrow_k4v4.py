"""K4V4 groups of at most four query heads, whose two pages of a tile share the eight columns: every group size, last pages and
tiles that a boundary of the reference's splits cuts, an odd page, short and empty sequences, both weight arithmetics."""
import pytest

from jf_testlib import Case
from test_gpu_decode_parity import check_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage_b", ["fp32", "int8p"])
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ctx,lens", [(17, [17, 16, 0]), (1001, [1001, 993, 31]), (6007, [6007, 4097, 5000])])
def test_group_sizes(stage_b, group, ctx, lens):
    check_case(Case("k4v4", len(lens), 2 * group, 2, ctx, lens=lens, seed=group), 16, stage_b=stage_b)
