"""K4V4 with the weights of a tile rounded to 127 levels, where scores lie hundreds apart: tiles whose largest weight is
next to nothing must weigh nothing."""
import pytest
import torch

from jf_testlib import Case
from test_gpu_long_rows import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [8.0, 30.0, 100.0])
def test_weights_of_far_tiles(scale):
    case = Case("k4v4", 3, 8, 2, 6000, lens=[6000, 5003, 900], seed=2)
    case.k_full = (case.k_full.float() * scale).to(case.dtype)
    _run(case, 64, stage_b="int8p")
