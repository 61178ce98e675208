"""The native half of ``ops``: argument errors are RuntimeErrors that name the op, before any launch."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

from jetfire_b200 import ops


@pytest.mark.parametrize("call", [
    lambda t: ops.fused_quant_write_int3_sym(t, t, t, t, 64),
    lambda t: ops.fused_quant_write_kv(t, t, t, t, t, t, t, 64, 3, 2),
    lambda t: ops.fused_attn_topk("k3v2", t, t, t, t, t, t, t, 16, 8, 2, 16, 32, 1.0),
    lambda t: ops.int3_qk_scores_topk(t, t, t, t, t, 16, 8, 2, 16, 1.0, 32),
    lambda t: ops.int2_softmax_v_with_pre_corr_wvs2(t, t, t, t, t, t, 16, 8, 2, 16, 32),
    lambda t: ops.blend_unnorm_into(t, t, t, t, t),
    lambda t: ops.blend_unnorm_into(None, t, t, t, t),
])
def test_host_tensors_are_refused_by_name(call):
    with pytest.raises(RuntimeError, match=r"^[a-z0-9_]+: "):
        call(torch.zeros(1, 8, 128))


@pytest.mark.parametrize("call", [
    lambda t, n: ops.int3_qk_scores_topk(t, t, t, t, t, n(16), n(8), n(2), n(16), n(1), n(32)),
    lambda t, n: ops.int8tc_qk_scores_topk_stats(t, t, t, t, t, n(16), n(8), n(2), n(16), n(1), n(32)),
    lambda t, n: ops.fused_attn_topk("k3v2", t, t, t, t, t, t, t, 16, 8, 2, n(16), 32, n(1)),
])
@pytest.mark.parametrize("number", [float, np.float32, torch.tensor, lambda v: torch.tensor(float(v)), str],
                         ids=["float", "numpy", "tensor", "float tensor", "text"])
def test_numbers_are_what_int_and_float_take(call, number):
    """The ops that convert their sizes with int() and float() get as far as the tensors."""
    with pytest.raises(RuntimeError, match="must be CUDA"):
        call(torch.zeros(1, 8, 128), number)


def test_a_number_that_is_none_is_an_error_of_its_own():
    t = torch.zeros(1, 8, 128)
    with pytest.raises((TypeError, ValueError)):
        ops.int3_qk_scores_topk(t, t, t, t, t, "sixteen", 8, 2, 16, 1.0, 32)


@pytest.mark.parametrize("module", ["None", "types.SimpleNamespace(built_for='jetfire_b200._host for torch 0.1')"],
                         ids=["missing", "of another torch"])
def test_the_host_ops_need_only_the_library(module):
    """Without a usable ``_host.so`` the package imports, the ops of the correction workers run, and an op
    that needs the module says how to build it."""
    code = f"""
import sys, types
sys.modules["jetfire_b200._host"] = {module}
import torch, jetfire_b200
if {module} is not None: jetfire_b200._host = {module}
from jetfire_b200 import ops
assert ops.get_cpu_attn_threads() > 0 and ops.numa_node_count() >= 1
t = torch.zeros(1, 8, 128)
try:
    ops.blend_unnorm_into(t, t, t, t, t)
except ImportError as e:
    assert "jetfire_b200.build" in str(e), e
    print("refused")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout == "refused\n", r.stdout + r.stderr


def test_a_module_for_another_torch_is_not_up_to_date(monkeypatch):
    from jetfire_b200 import build
    if not build.up_to_date():
        pytest.skip("the sources are newer than the build")
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".1")
    assert not build.up_to_date()
