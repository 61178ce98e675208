"""Tensors of unusual make at the ops that are native code: an error or the right bytes, never a crash."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

BATCHED = """
import torch
from jetfire_b200 import ops
bf, u8, f32 = (dict(device="cuda", dtype=d) for d in (torch.bfloat16, torch.uint8, torch.float32))
x, slots = torch.zeros(4, 2, 128, **bf), torch.zeros(4, dtype=torch.int64, device="cuda")
kd, ks = torch.zeros(2, 64, 48, **u8), torch.zeros(2, 64, 2, **bf)
vd, vs = torch.zeros(2, 64, 32, **u8), torch.zeros(2, 64, 2, **bf)
bt, lens = torch.zeros(1, 4, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
q, o, W, out = torch.zeros(1, 4, 128, **bf), torch.zeros(1, 4, 128, **f32), torch.zeros(1, 4, **f32), torch.zeros(1, 4, 128, **bf)
for arg, call in ((x, lambda x: ops.fused_quant_write_int3_sym(x, slots, kd, ks, 64)),
                  (x, lambda x: ops.fused_quant_write_kv(x, x, slots, kd, ks, vd, vs, 64, 3, 2)),
                  (q, lambda q: ops.int2_fused_attn_topk(q, kd, ks, None, vd, vs, bt, lens, 64, 4, 2, 16, 32, 1.0)),
                  (q, lambda q: ops.int3_qk_scores_topk(q, kd, ks, bt, lens, 64, 4, 2, 16, 1.0, 32)),
                  (out, lambda out: ops.blend_unnorm_into(o, o, W, q, out))):
    try:
        torch.vmap(lambda t: (call(t), t)[1])(torch.stack([arg, arg]))
        print("no error")
    except RuntimeError as e:
        print("refused" if "storage" in str(e) else str(e))
torch.cuda.synchronize()
"""


def test_tensors_without_storage_are_refused():
    """A tensor whose address cannot be taken (here: batched by vmap) raises; with the address taken after the
    interpreter lock was released the same error ended the process."""
    r = subprocess.run([sys.executable, "-c", BATCHED], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split("\n")[:-1] == ["refused"] * 5


def test_a_lazy_copy_gets_memory_of_its_own_before_it_is_written():
    from jetfire_b200 import ops
    x = torch.randn(4, 2, 128, device="cuda").to(torch.bfloat16)
    slots = torch.arange(4, device="cuda")
    caches = [torch.full((2, 64, 48), 0xA5, dtype=torch.uint8, device="cuda"), torch.zeros(2, 64, 2, dtype=torch.bfloat16, device="cuda"),
              torch.full((2, 64, 32), 0xA5, dtype=torch.uint8, device="cuda"), torch.zeros(2, 64, 2, dtype=torch.bfloat16, device="cuda")]
    before = [t.clone() for t in caches]
    copies = [torch._lazy_clone(t) for t in caches]
    ops.fused_quant_write_kv(x, x, slots, *copies, 64, 3, 2)
    out = torch.zeros(1, 4, 128, dtype=torch.bfloat16, device="cuda")
    out_copy = torch._lazy_clone(out)
    o = torch.ones(1, 4, 128, device="cuda")
    ops.blend_unnorm_into(o, torch.zeros_like(o), torch.zeros(1, 4, device="cuda"), out, out_copy)
    torch.cuda.synchronize()
    for t, b, c in zip(caches, before, copies):
        assert torch.equal(t, b) and not torch.equal(c, b)
    assert bool((out == 0).all()) and bool((out_copy == 1).all())
