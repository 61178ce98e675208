"""Workspace sizes: what a call requires does not outgrow a workspace made for a longer row, fits the built-in
scratch wherever one wave of the scan's partials does, and what it can use covers every smaller call."""
import itertools

import pytest
import torch

from jetfire_b200 import ops
from jetfire_b200._lib import lib

GEOMETRIES = [(32, 8), (64, 8), (32, 4), (16, 2), (8, 1), (32, 2)]
BATCHES = (1, 2, 3, 4, 5, 7, 8, 12, 16, 24, 32, 64)
LENGTHS = range(16, 140000, 1040)


def _required(mode, B, H_q, H_kv, S):
    return lib.jf_decode_workspace_bytes(mode, B, H_q, H_kv, S, 256)


def _useful(mode, B, H_q, H_kv, S):
    return lib.jf_decode_workspace_useful_bytes(mode, B, H_q, H_kv, S, 256)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("H_q,H_kv", GEOMETRIES)
def test_a_workspace_for_the_longest_row_serves_the_shorter_ones(mode, H_q, H_kv):
    for B in BATCHES:
        # neighbours of a page as well: the cut may change from one to the next
        lengths = sorted(set(itertools.chain.from_iterable((s, s + 16, s + 32) for s in LENGTHS)))
        required = [_required(mode, B, H_q, H_kv, s) for s in lengths]
        useful = [_useful(mode, B, H_q, H_kv, s) for s in lengths]
        assert required == sorted(required) and useful == sorted(useful)
        assert all(r <= u for r, u in zip(required, useful))
        bigger = [_useful(mode, B + 1, H_q, H_kv, s) for s in lengths]
        assert all(a <= b for a, b in zip(useful, bigger))


def test_required_is_one_wave_of_partials():
    """128 rows of KV heads, 148 multiprocessors with four blocks each: four partials a row in one wave, while
    nine in two are faster from 300 units on.  Partials take 8 x 128 floats and 18 more; the arrays and the row of
    page maxima (one per page or pair of pages) are rounded up to 256 bytes, plus 256 for the status record."""
    up = lambda n: (n + 255) // 256 * 256
    for mode, group in ((0, 32), (1, 16)):
        for S in (4096, 9600, 9616, 20000, 131072):
            def size(partials):
                maxima = ((S + group - 1) // group + 3) // 4 * 4
                return (256 + up(partials * 4096) + 2 * up(partials * 32) + up(partials * 8) + up(16 * 32 * maxima * 4)
                        + up(16 * 32 * S * 4))
            assert _required(mode, 16, 32, 8, S) == size(4 * 128)
            assert _useful(mode, 16, 32, 8, S) == size(2 * 148 * 4)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,stage_b", [("k3v2", "fp32"), ("k4v4", "int8p")])
def test_a_call_with_the_required_workspace_alone(mode, stage_b):
    """Rows long enough for two waves of blocks in the smaller workspace: the same selection, outputs to rounding."""
    import numpy as np
    from jf_testlib import Case
    case = Case(mode, 1, 16, 8, 10400, seed=8)
    B = 16                                              # the sequences' rows are shuffles of the same blocks
    g = torch.Generator().manual_seed(9)
    n = (case.ctx + 15) // 16
    kd, ks, vd, vs = case.device_cache()
    q = torch.randn(B, 16, 128, generator=g).to(case.dtype).cuda()
    bt = torch.stack([torch.randperm(case.n_blocks, generator=g)[:n] for _ in range(B)]).cuda()
    lens = torch.tensor([case.ctx - 600 * (i % 3) for i in range(B)], dtype=torch.int32, device="cuda")
    need, useful = (f(0 if mode == "k3v2" else 1, B, 16, 8, case.ctx) for f in (_required, _useful))
    assert need < useful
    res = []
    for size in (need, useful):
        ws = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
        ws = ws[(-ws.data_ptr()) % 256:][:size]         # exactly that much
        r = ops.fused_attn_topk(mode, q, kd, ks, vd, vs, bt, lens, case.ctx, 16, 8, 16, 64, case.attn_scale, workspace=ws,
                                stage_b=stage_b)
        res.append([t.cpu().numpy() for t in (r.topk_idx, r.topk_slots, r.o_hat, r.o_old_unnorm, r.W)])
    a, b = res
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for x, y in zip(a[2:], b[2:]):
        assert np.all(np.abs(x - y) <= 2e-3 + 1e-3 * np.abs(y))
    with pytest.raises(RuntimeError, match="workspace"):
        ops.fused_attn_topk(mode, q, kd, ks, vd, vs, bt, lens, case.ctx, 16, 8, 16, 64, case.attn_scale, workspace=ws[:need - 256])
