"""The work a user of this package has it do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges; ``prepare`` makes what
a program holds before the call, ``run`` is one pass through the public entry points, ``work`` the
bytes and operations a pass cannot do without, ``tolerance`` how far another correct
implementation may be off.

Kinds of pass (``kind``):
  append   quantise-on-append of K and V of ``tokens`` tokens into the packed paged cache
  call     the one-shot decode-attention op under the reference's name, arguments checked and outputs
           allocated by every call
  step     one layer of a decode step with a kept argument block: append of one token per sequence,
           fused attention over the packed cache, merge of a correction that is at hand; ``graph``
           replays the same calls from a CUDA graph, as serving loops do
  stages   the same attention through the reference's Stage A / Stage B ops, then the merge
  adapter  the serving adapter's layer step: ``JetFireCacheStore.write_slots`` (packed cache and host
           mirror), then ``try_jetfire_decode`` with the host correction over the mirror

Geometries are those of ``bench.py`` (32/8, 64/8 and 32/4 query/KV heads) and what tensor-parallel
sharding leaves of them on one GPU (16/2, 8/1); 32/2 is the widest group the kernels take.  K and V are
N(0, 1), K scaled per channel by log-normal(0, 0.75): a few channels are outliers.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from jetfire_b200 import ops
from jetfire_b200.adapter.cache_store import JetFireCacheStore
from jetfire_b200.adapter.config import JetFireConfig
from jetfire_b200.adapter.decode_path import make_decode_metadata, try_jetfire_decode

HEAD_DIM, BLOCK = 128, 16
MODE_BITS = {"k3v2": (3, 2, 64), "k4v4": (4, 4, 128)}          # K bits, V bits, group size
ROW_BYTES = {"k3v2": 88, "k4v4": 132}                          # packed K + V of one (token, KV head), scales included
SCHEME = {"k3v2": "SymInt3K_SymInt2V", "k4v4": "SymInt4K_SymInt4V"}
DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16}
GEOMETRIES = ((32, 8), (64, 8), (32, 4), (16, 2), (8, 1), (32, 2))
MAX_APPEND_ROWS = 32768 * 8                                    # (token, KV head) rows of the largest append
MAX_KV_ROWS = 16 * 8 * 131072                                  # (position, KV head) rows of the largest step
MAX_MIRROR_ROWS = 4 * 8 * 8192                                 # rows of the largest adapter case (mirror in host memory)


def listed():
    return [
        # one new token of each of eight sequences: the smallest launch of a serving loop
        dict(name="append_decode_tokens", kind="append", mode="k3v2", dtype="bf16", tokens=8, kv_heads=8, layout="qkv"),
        # a 32768-token prefill chunk, K and V as views into the projection's output
        dict(name="append_prefill_32k", kind="append", mode="k3v2", dtype="bf16", tokens=32768, kv_heads=8, layout="qkv"),
        # a ragged chunk of several prompts, fp16, padded at its end
        dict(name="append_prefill_ragged", kind="append", mode="k4v4", dtype="fp16", tokens=3001, kv_heads=8, layout="own"),
        # a short chat turn through the one-shot op
        dict(name="call_short_b1", kind="call", mode="k3v2", dtype="bf16", heads=32, kv_heads=8, batch=1, ctx=2048,
             top_k=256, ragged=False, paging="runs"),
        # the reference's two-stage call order, ragged lengths, tensors whose sizes divide nothing
        dict(name="stages_ragged_b3", kind="stages", mode="k4v4", dtype="fp16", heads=32, kv_heads=8, batch=3, ctx=6007,
             top_k=256, ragged=True, paging="shuffled"),
        # Llama-3.1-8B layer, batch 1 at 32k: latency of one sequence
        dict(name="step_8b_b1_32k", kind="step", mode="k3v2", dtype="bf16", heads=32, kv_heads=8, batch=1, ctx=32768,
             top_k=256, ragged=False, paging="runs", graph=True),
        # the same layer, K4V4, batch 4
        dict(name="step_8b_k4_b4_32k", kind="step", mode="k4v4", dtype="bf16", heads=32, kv_heads=8, batch=4, ctx=32768,
             top_k=256, ragged=False, paging="runs", graph=False),
        # Llama-3.3-70B layer, the benchmark's default workload
        dict(name="step_70b_b4_64k", kind="step", mode="k3v2", dtype="bf16", heads=64, kv_heads=8, batch=4, ctx=65536,
             top_k=512, ragged=False, paging="shuffled", graph=False),
        # Qwen3-30B-A3B layer, fp16, eight sequences of different lengths
        dict(name="step_30b_b8_ragged", kind="step", mode="k3v2", dtype="fp16", heads=32, kv_heads=4, batch=8, ctx=32761,
             top_k=256, ragged=True, paging="shuffled", graph=True),
        # the largest of the sweep: sixteen sequences at 128k
        dict(name="step_8b_k4_b16_128k", kind="step", mode="k4v4", dtype="fp16", heads=32, kv_heads=8, batch=16, ctx=131072,
             top_k=256, ragged=False, paging="runs", graph=False),
        # what the vLLM backend does per layer, host correction included
        dict(name="adapter_8b_b4_8k", kind="adapter", mode="k3v2", dtype="bf16", heads=32, kv_heads=8, batch=4, ctx=8192,
             top_k=256, ragged=True, paging="runs"),
        dict(name="adapter_8b_k4_b1_2k", kind="adapter", mode="k4v4", dtype="bf16", heads=32, kv_heads=8, batch=1, ctx=2048,
             top_k=128, ragged=False, paging="shuffled"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("append", "append", "call", "step", "step", "step", "stages", "adapter"))
    mode, dtype = rng.choice(("k3v2", "k4v4")), rng.choice(("bf16", "fp16"))
    if kind == "append":
        kv = rng.choice((1, 2, 4, 8))
        return dict(kind=kind, mode=mode, dtype=dtype, tokens=_log_int(rng, 1, MAX_APPEND_ROWS // kv if kv > 2 else 65536),
                    kv_heads=kv, layout=rng.choice(("qkv", "own")))
    heads, kv = rng.choice(GEOMETRIES)
    batch = _log_int(rng, 1, 16)
    rows = {"adapter": MAX_MIRROR_ROWS, "call": MAX_KV_ROWS // 64, "stages": MAX_KV_ROWS // 16, "step": MAX_KV_ROWS}[kind]
    ctx = _log_int(rng, 512, max(1024, min(131072, rows // (batch * kv))))
    case = dict(kind=kind, mode=mode, dtype=dtype, heads=heads, kv_heads=kv, batch=batch, ctx=ctx,
                top_k=rng.choice((64, 128, 256, 256, 512)), ragged=rng.random() < 0.5, paging=rng.choice(("runs", "shuffled")))
    if kind == "step":
        case["graph"] = rng.random() < 0.5
    return case


def _lens(case):
    """Sequence lengths: all ``ctx``, or falling from it to about a third of it in uneven steps."""
    b, ctx = case["batch"], case["ctx"]
    if not case["ragged"]:
        return [ctx] * b
    return [max(1, ctx - (2 * ctx * i) // (3 * b) - 7 * i) for i in range(b)]


def _stage_b(case):
    # the reference's plan: K4V4 with more than one sequence rounds the weights per tile
    return "int8p" if case["mode"] == "k4v4" and case["batch"] > 1 else "fp32"


def _tokens(g, n, kv, dtype, scale, layout="own"):
    """K and V of ``n`` tokens, (n, kv, 128): tensors of their own, or views into a projection's output."""
    if layout == "qkv":
        x = torch.randn(n, 3 * kv, HEAD_DIM, generator=g, device="cuda")
        x[:, kv:2 * kv] *= scale
        x = x.to(dtype)
        return x[:, kv:2 * kv], x[:, 2 * kv:]
    k = torch.randn(n, kv, HEAD_DIM, generator=g, device="cuda") * scale
    v = torch.randn(n, kv, HEAD_DIM, generator=g, device="cuda")
    return k.to(dtype), v.to(dtype)


def _cache(mode, kv, slots):
    kb, vb, gs = MODE_BITS[mode]
    u8 = dict(dtype=torch.uint8, device="cuda")
    bf = dict(dtype=torch.bfloat16, device="cuda")
    return (torch.zeros(kv, slots, 16 * kb, **u8), torch.zeros(kv, slots, HEAD_DIM // gs, **bf),
            torch.zeros(kv, slots, 16 * vb, **u8), torch.zeros(kv, slots, HEAD_DIM // gs, **bf))


def _channel_scale(g, kv):
    return torch.exp(0.75 * torch.randn(1, kv, HEAD_DIM, generator=g, device="cuda"))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPE[case["dtype"]]
    s = SimpleNamespace(kind=case["kind"], mode=case["mode"])
    s.kb, s.vb, s.gs = MODE_BITS[case["mode"]]
    kv = case["kv_heads"]
    scale = _channel_scale(g, kv)
    if s.kind == "append":
        n = case["tokens"]
        s.key, s.value = _tokens(g, n, kv, dtype, scale, case["layout"])
        blocks = (n + BLOCK - 1) // BLOCK + 1
        if n <= 64:      # one token of each sequence: anywhere in the cache
            s.slots = torch.randperm(64 * BLOCK, generator=g, device="cuda")[:n]
            blocks = 64
        else:            # whole prompts: their blocks in any order, the chunk's last rows padding
            order = torch.randperm(blocks, generator=g, device="cuda")
            s.slots = (order[:, None] * BLOCK + torch.arange(BLOCK, device="cuda")).reshape(-1)[:n].contiguous()
            if n % 8:
                s.slots[n - n % 8:] = -1
        s.cache = _cache(s.mode, kv, blocks * BLOCK)
        return s

    batch, ctx, heads = case["batch"], case["ctx"], case["heads"]
    lens = _lens(case)
    per_seq = (ctx + BLOCK - 1) // BLOCK
    n_blocks = batch * per_seq + 1
    if case["paging"] == "shuffled":
        table = torch.randperm(n_blocks, generator=g, device="cuda")[:batch * per_seq].reshape(batch, per_seq)
    else:
        table = torch.arange(batch * per_seq, device="cuda").reshape(batch, per_seq)
    s.block_table = table.to(torch.int64).contiguous()
    s.seq_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    s.max_s, s.heads, s.kv, s.top_k, s.attn = per_seq * BLOCK, heads, kv, case["top_k"], HEAD_DIM ** -0.5
    s.q = torch.randn(batch, heads, HEAD_DIM, generator=g, device="cuda").to(dtype)
    if s.kind == "adapter":
        cfg = JetFireConfig(mode=SCHEME[s.mode], top_k=s.top_k, group_size=s.gs, max_batch_size=batch)
        s.store = JetFireCacheStore(num_blocks=n_blocks, num_kv_heads=kv, head_dim=HEAD_DIM, cfg=cfg, device="cuda", dtype=dtype)
        s.cfg = cfg
        write = s.store.write_slots
    else:
        s.cache = _cache(s.mode, kv, n_blocks * BLOCK)

        def write(k, v, slots):
            ops.fused_quant_write_kv(k, v, slots, *s.cache, s.gs, s.kb, s.vb)
    for b, n in enumerate(lens):
        k, v = _tokens(g, n, kv, dtype, scale)
        pos = torch.arange(n, device="cuda")
        write(k, v, s.block_table[b, pos // BLOCK] * BLOCK + pos % BLOCK)
    # the token of this step: each sequence's last
    last = torch.tensor([n - 1 for n in lens], device="cuda")
    s.slots = s.block_table.gather(1, (last // BLOCK)[:, None])[:, 0] * BLOCK + last % BLOCK
    s.key, s.value = _tokens(g, batch, kv, dtype, scale, "qkv")
    if s.kind == "adapter":
        s.impl = SimpleNamespace(scale=s.attn)
        s.layer = SimpleNamespace(num_heads=heads, num_kv_heads=kv, head_size=HEAD_DIM)
        s.meta = make_decode_metadata(s.seq_lens, s.block_table.to(torch.int32))
        s.query = s.q.reshape(batch, heads, HEAD_DIM)
        s.out = torch.zeros(batch, heads * HEAD_DIM, dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        return s
    s.o_new = torch.randn(batch, heads, HEAD_DIM, generator=g, device="cuda").to(dtype)
    s.out = torch.empty(batch, heads, HEAD_DIM, dtype=dtype, device="cuda")
    if s.kind == "step":
        s.call = ops.DecodeCall(s.mode, s.q, *s.cache, s.block_table, s.seq_lens, s.max_s, heads, kv, BLOCK, s.top_k, s.attn,
                                stage_b=_stage_b(case))
        s.graph = None
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _step(s)
            torch.cuda.current_stream().wait_stream(side)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                _step(s)
            s.graph = graph
    elif s.kind == "stages":
        s.k3 = s.mode == "k3v2"
        s.int8p = _stage_b(case) == "int8p"
    return s


def _step(s):
    ops.fused_quant_write_kv(s.key, s.value, s.slots, *s.cache, s.gs, s.kb, s.vb)
    s.call.fused()
    r = s.call.out
    ops.blend_unnorm_into(r["o_hat"], r["o_old_unnorm"], r["W"], s.o_new, s.out)


def run(s):
    if s.kind == "append":
        ops.fused_quant_write_kv(s.key, s.value, s.slots, *s.cache, s.gs, s.kb, s.vb)
        return s.cache
    if s.kind == "adapter":
        s.store.write_slots(s.key, s.value, s.slots)
        out = try_jetfire_decode(impl=s.impl, layer=s.layer, query=s.query, attn_metadata=s.meta, output=s.out,
                                 store=s.store, cfg=s.cfg)
        return (out, s.store.k_data, s.store.k_scales, s.store.v_data, s.store.v_scales, s.store.slot_filled,
                s.store.k_shadow, s.store.v_shadow)
    if s.kind == "step":
        if s.graph is not None:
            s.graph.replay()
        else:
            _step(s)
        r = s.call.out
        return (s.out, r["o_hat"], r["o_old_unnorm"], r["W"], r["topk_idx"], r["topk_slots"]) + s.cache
    k_data, k_scales, v_data, v_scales = s.cache
    if s.kind == "call":
        o_hat, slots, o_old, w = ops.int2_fused_attn_topk(s.q, k_data, k_scales, None, v_data, v_scales, s.block_table,
                                                          s.seq_lens, s.max_s, s.heads, s.kv, BLOCK, s.top_k, s.attn)
        ops.blend_unnorm_into(o_hat, o_old, w, s.o_new, s.out)
        return s.out, o_hat, o_old, w, slots
    tail = (s.block_table, s.seq_lens, s.max_s, s.heads, s.kv, BLOCK)
    if s.k3:
        scores, idx, slots = ops.int3_qk_scores_topk(s.q, k_data, k_scales, *tail, s.attn, s.top_k)
        stats = ()
        o_hat, o_old, w = ops.int2_softmax_v_with_pre_corr_wvs2(scores, v_data, v_scales, *tail[:2], idx, *tail[2:], s.top_k)
    else:
        scores, idx, slots, m, inv_z = ops.int8tc_qk_scores_topk_stats(s.q, k_data, k_scales, *tail, s.attn, s.top_k)
        stats = (m, inv_z)
        if s.int8p:
            o_hat, o_old, w = ops.int8tc_softmax_v_with_pre_corr_reg_stats(scores, m, inv_z, v_data, v_scales, *tail[:2], idx,
                                                                           *tail[2:], s.top_k)
        else:
            o_hat, o_old, w = ops.int4_softmax_v_with_pre_corr_wvs2_scores(scores, v_data, v_scales, *tail[:2], idx,
                                                                           *tail[2:], s.top_k)
    ops.blend_unnorm_into(o_hat, o_old, w, s.o_new, s.out)
    return (s.out, scores, idx, slots, o_hat, o_old, w) + stats


def work(case):
    kv, row = case["kv_heads"], ROW_BYTES[case["mode"]]
    if case["kind"] == "append":
        live = case["tokens"] - (case["tokens"] % 8 if case["tokens"] > 64 else 0)
        return {"bytes": live * (kv * (2 * 2 * HEAD_DIM + row)) + 8 * case["tokens"], "flops": 4 * live * kv * HEAD_DIM}
    batch, heads, k = case["batch"], case["heads"], case["top_k"]
    positions = sum(_lens(case))
    rows = batch * heads
    nbytes = positions * kv * row + 4 * positions // BLOCK * 2 + rows * HEAD_DIM * 2      # packed cache, block table, query
    flops = 4 * positions * heads * HEAD_DIM
    if case["kind"] in ("step", "adapter"):
        nbytes += batch * kv * (2 * 2 * HEAD_DIM + row)                                   # the new tokens
    if case["kind"] == "adapter":
        sel = sum(min(n, k) for n in _lens(case)) * heads
        nbytes += batch * kv * 2 * 2 * HEAD_DIM + sel * 2 * 2 * HEAD_DIM + rows * HEAD_DIM * 2   # mirror rows written and gathered, output
        return {"bytes": nbytes, "flops": flops + 4 * sel * HEAD_DIM}
    nbytes += rows * (HEAD_DIM * (4 + 4 + 2 + 2) + 4) + rows * k * 8                       # outputs, correction, merged output, slots
    if case["kind"] in ("step", "stages"):
        nbytes += rows * k * 8                                                            # positions
    if case["kind"] == "stages":
        nbytes += rows * ((case["ctx"] + 15) // 16 * 16) * 4                              # scores, an output here
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "append":
        return "exact"          # packed bytes and scales
    # Slots and positions are exact.  Attention outputs: the softmax weights meet V as 16-bit floats
    # (2^-11 each, relative to a reference point that an implementation may choose), sums in fp32, the
    # merged output is stored in the model's 16-bit type (bf16: 2^-9).
    return {"rel": 4e-3, "max": 0.05} if case["kind"] == "adapter" else {"rel": 2e-3, "max": 0.05}
