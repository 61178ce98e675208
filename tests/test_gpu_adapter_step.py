"""The kernels at the two ends of the adapter's stream-ordered step: the forms of inputs and outputs they
address themselves, and the ones that go through a copy, all give the bits of the plain form."""
import time
from types import SimpleNamespace

import pytest
import torch

from jf_testlib import Case

pytestmark = pytest.mark.gpu


def _store(case, cfg):
    from jetfire_b200.adapter.cache_store import JetFireCacheStore
    st = JetFireCacheStore(num_blocks=case.n_blocks, num_kv_heads=case.H_kv, head_dim=128, cfg=cfg, device="cuda",
                           dtype=case.dtype, mirror_append="mapped")
    st.write_slots(case.k_full.transpose(0, 1).contiguous().cuda(), case.v_full.transpose(0, 1).contiguous().cuda(),
                   torch.arange(case.num_slots, dtype=torch.int32, device="cuda"))      # converted by the store
    return st


@pytest.mark.parametrize("B,H_q,dtype", [(1, 2, torch.bfloat16), (3, 8, torch.float16), (2, 32, torch.bfloat16)])
def test_step_takes_the_forms_a_caller_has(B, H_q, dtype):
    from jetfire_b200.adapter.config import JetFireConfig
    from jetfire_b200.adapter.decode_path import make_decode_metadata, try_jetfire_decode
    case = Case("k3v2", B, H_q, 2, 200, seed=61 + B, dtype=dtype)
    cfg = JetFireConfig(mode="SymInt3K_SymInt2V", top_k=32, group_size=64, cpu_attn_threads=2)
    st = _store(case, cfg)
    assert bool(st.slot_filled.all())
    impl = SimpleNamespace(scale=case.attn_scale, attn_type=SimpleNamespace(name="DECODER"))
    layer = SimpleNamespace(num_heads=H_q, num_kv_heads=2, head_size=128, layer_name="l0")
    bt, lens, q = case.block_table.cuda(), case.seq_lens.cuda(), case.q.cuda()
    row = H_q * 128

    def run(query, block_table, seq_lens, out):
        md = make_decode_metadata(seq_lens, block_table)
        assert try_jetfire_decode(impl=impl, layer=layer, query=query, attn_metadata=md, output=out, store=st, cfg=cfg) is out
        torch.cuda.synchronize()
        return out[:B].reshape(B, row).cuda()

    want = run(q, bt, lens, torch.zeros(B, row, dtype=dtype, device="cuda"))
    wide = torch.full((B + 2, row + 8), 3.0, dtype=dtype, device="cuda")
    odd = torch.zeros(B, row + 3, dtype=dtype, device="cuda")
    q_pad = torch.zeros(B + 1, H_q, 128, dtype=dtype, device="cuda")
    q_pad[:B] = q
    q_odd = torch.zeros(B * row + 1, dtype=dtype, device="cuda")[1:].view(B, H_q, 128)   # 2-byte aligned
    q_odd.copy_(q)
    forms = [(q.view(B, row), bt.to(torch.int32), lens.to(torch.int64), wide[:, :row]),
             (q_pad, bt, lens, torch.zeros(B, H_q, 128, dtype=dtype, device="cuda")),
             (q_odd, torch.cat([bt, bt], 1), lens, odd[:, 3:]),
             (q, bt.cpu(), lens.cpu(), torch.zeros(B, row, dtype=dtype, device="cuda")),
             (q, bt, lens.double(), torch.zeros(B, 2 * row, dtype=dtype)[:, ::2])]
    if B == 1:       # strides of a dimension of one element mean nothing; lengths without a dimension
        forms.append((q.view(H_q, 128, 1).clone().permute(2, 0, 1), bt, lens[0], torch.zeros(1, row, dtype=dtype, device="cuda")))
    for query, table, length, out in forms:
        if query.dim() == 2:
            query = query.view(B, H_q, 128)
        assert torch.equal(run(query, table, length, out), want)
    assert bool((wide[B:] == 3.0).all()) and bool((wide[:, row:] == 3.0).all())
    same = run(q, bt[:1].expand(B, -1).contiguous(), lens, torch.zeros(B, row, dtype=dtype, device="cuda"))
    assert torch.equal(run(q, bt[:1], lens, torch.zeros(B, row, dtype=dtype, device="cuda")), same)    # one table for all
    for bad in (torch.zeros(B, row, device="cuda"), torch.zeros(B, row, dtype=dtype)):
        with pytest.raises(RuntimeError, match="output"):
            run(q, bt, lens, bad)


def _one_step(top_k=32):
    """A store with one sequence and a callable that runs its step."""
    from jetfire_b200.adapter import decode_path as dp
    from jetfire_b200.adapter.config import JetFireConfig
    case = Case("k3v2", 1, 8, 2, 200, seed=71)
    cfg = JetFireConfig(mode="SymInt3K_SymInt2V", top_k=top_k, group_size=64, cpu_attn_threads=2)
    st = _store(case, cfg)
    impl = SimpleNamespace(scale=case.attn_scale)
    layer = SimpleNamespace(num_heads=8, num_kv_heads=2, head_size=128)
    md = dp.make_decode_metadata(case.seq_lens.cuda(), case.block_table.cuda())
    q = case.q.cuda()

    def run():
        out = torch.zeros(1, 8 * 128, dtype=case.dtype, device="cuda")
        assert dp.try_jetfire_decode(impl=impl, layer=layer, query=q, attn_metadata=md, output=out, store=st, cfg=cfg) is out
        torch.cuda.synchronize()
        return out
    return st, run


TAGGED = torch.tensor([0x4A46535441545553, 2], dtype=torch.int64)      # a status record that says JF_ERR_TIMEOUT


def test_a_recorded_error_is_reported_once():
    """An error in the workspace's record reaches the host with the step's end, raises from the next call
    (or from ``status()``) and from no later one; the calls after that run."""
    from jetfire_b200._lib import JetFireError
    from jetfire_b200.adapter.decode_path import stream_steps
    st, run = _one_step()
    want = run()
    step = stream_steps(st)[0]
    record = step.call.status_record().view(torch.int64)
    for read in (run, step.status):
        record.copy_(TAGGED)
        assert torch.equal(run(), want)            # carries the record to the host
        with pytest.raises(JetFireError, match="bounded wait"):
            read()
        assert torch.equal(run(), want) and torch.equal(run(), want)
        step.status()
    # a record that came over while the host did not look stays until it does
    record.copy_(TAGGED)
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        step.run(step.q.clone(), step.block_table.clone(), step.seq_lens.clone(), torch.zeros_like(want))
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    with pytest.raises(JetFireError, match="bounded wait"):
        step.status()
    graph.replay()
    torch.cuda.synchronize()
    step.status()
    del graph


@pytest.mark.parametrize("B,H_q", [(1, 4), (1, 32), (3, 11), (5, 20)], ids=["one block", "a full block", "two blocks", "four blocks"])
def test_the_wait_at_the_end_runs_out(B, H_q):
    """jf_step_end with a completion word that nobody sets: the stream goes on after the budget, the error is
    handed to the host, the record is clear again; the next call, with the word set, leaves no error.  A word
    left set by a run that was given up does not count once the trigger is raised."""
    from jetfire_b200 import ops
    from jetfire_b200._lib import JF_ERR_TIMEOUT, lib
    g = torch.Generator(device="cuda").manual_seed(3)
    o_hat, o_old = (torch.randn(B, H_q, 128, generator=g, device="cuda") for _ in range(2))
    W = torch.rand(B, H_q, generator=g, device="cuda")
    o_new = torch.randn(B, H_q, 128, generator=g, device="cuda").to(torch.float16)
    want = torch.empty_like(o_new)
    ops.blend_unnorm_into(o_hat, o_old, W, o_new, want)
    host, dev = ops.alloc_mapped_pinned_pair((64,), torch.int64)       # trigger, completion word, record's copy a line apart
    ops.zero_host(host)
    word = lambda i: dev.data_ptr() + 8 * i
    record = torch.zeros(32, dtype=torch.int64, device="cuda")

    def end(trigger):
        record.zero_()
        out = torch.zeros_like(o_new)
        t = time.perf_counter()
        st = lib.jf_step_end(o_hat.data_ptr(), o_old.data_ptr(), W.data_ptr(), o_new.data_ptr(), out.data_ptr(), H_q * 128,
                             ops._dtype_id(out), B, H_q, word(16), word(0) if trigger else None, 20, record.data_ptr(), word(32),
                             torch.cuda.current_stream().cuda_stream)
        assert st == 0
        torch.cuda.synchronize()
        assert time.perf_counter() - t < 1.0 and torch.equal(out, want)
        assert int(record[0]) == 0
        code = int(host[33]) & 0xFFFFFFFF if int(host[32]) else 0
        ops.zero_host(host[32:34])
        return code

    assert end(False) == JF_ERR_TIMEOUT
    host[16] = 1
    assert end(False) == 0 and end(False) == 0
    assert end(True) == JF_ERR_TIMEOUT and int(host[0]) == 1 and int(host[16]) == 0
    ops.free_mapped_pinned_pair(host)


def test_building_a_step_leaves_the_processors_free():
    """No thread may still be busy once a step object is built: its first run needs the processors for the
    dispatcher and the workers.  (Fifteen OpenMP threads spinning for 4 ms are 60 ms of processor time.)"""
    from jetfire_b200.adapter import decode_path as dp
    from jetfire_b200.adapter.config import JetFireConfig
    if torch.get_num_threads() < 8:
        pytest.skip("fewer than eight OpenMP threads: nothing to see")
    torch.zeros(1 << 20).add_(1.0)                               # the OpenMP threads exist
    cfg = JetFireConfig(mode="SymInt3K_SymInt2V", top_k=256, group_size=64, cpu_attn_threads=2)
    st = _store(Case("k3v2", 1, 8, 2, 4096, seed=5), cfg)
    step = dp._StreamStep(st, cfg, 4, 32, 256, 256, 4096, torch.bfloat16, torch.device("cuda"), 1.0)
    step.close()                                                 # dispatcher and allocator have been used once
    time.sleep(0.2)
    step = dp._StreamStep(st, cfg, 4, 32, 256, 256, 4096, torch.bfloat16, torch.device("cuda"), 1.0)
    busy = time.process_time()
    time.sleep(0.006)
    busy = time.process_time() - busy
    torch.cuda.synchronize()
    step.close()
    assert busy < 0.02, f"{1e3 * busy:.1f} ms of processor time in the 6 ms after the step was built"
