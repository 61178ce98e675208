"""K4V4 with a tile's weights rounded to 127 levels of the largest (stage_b "int8p"): the levels are those of correctly
rounded fp32 arithmetic, whatever the V scales.  With a query of zeros every softmax weight is 1 exactly, so a tile's
weights are its V scales; V codes that are 1 in the token's own channel and 0 elsewhere hand each weight out by itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOKENS, MAX_S, H_KV = 32, 256, 8       # max_S / 8 positions a split of the reference: one tile a sequence


def tile_weights(scales: np.ndarray, group: int) -> np.ndarray:
    """Weight by weight what tiles of 32 tokens with these V scales (tiles, 32) bring to the output."""
    from jetfire_b200 import ops
    B = scales.shape[0] // H_KV
    slots = B * TOKENS
    vd = torch.full((H_KV, slots, 64), 0x88, dtype=torch.uint8)
    t = torch.arange(slots) % TOKENS
    vd[:, torch.arange(slots), t // 2] = torch.where(t % 2 == 0, 0x98, 0x89).to(torch.uint8)   # code + 8; even channels in the high half
    vs = torch.from_numpy(scales.reshape(B, H_KV, TOKENS)).transpose(0, 1).reshape(H_KV, slots, 1).to(torch.bfloat16)
    table = torch.zeros(B, MAX_S // 16, dtype=torch.int64)
    table[:, :2] = torch.arange(2 * B).reshape(B, 2)
    kd = torch.randint(0, 256, (H_KV, slots, 64), dtype=torch.uint8)
    ks = torch.ones(H_KV, slots, 1, dtype=torch.bfloat16)
    q = torch.zeros(B, H_KV * group, 128, dtype=torch.bfloat16)
    res = ops.fused_attn_topk("k4v4", q.cuda(), kd.cuda(), ks.cuda(), vd.cuda(), vs.cuda(), table.cuda(),
                              torch.full((B,), TOKENS, dtype=torch.int32, device="cuda"), MAX_S, H_KV * group, H_KV, 16, 8, 1.0,
                              stage_b="int8p")
    o = res.o_hat.cpu().numpy().reshape(B, H_KV, group, 128)
    assert not o[..., TOKENS:].any()
    assert np.array_equal(o, np.broadcast_to(o[:, :, :1], o.shape), equal_nan=True)   # the heads of a group have the same weights
    return o[:, :, 0, :TOKENS].reshape(-1, TOKENS) * np.float32(TOKENS)


def levels(scales: np.ndarray):
    s = scales.astype(np.float32)
    unit = s.max(1, keepdims=True) * np.float32(1.0 / 127.0)
    inv = np.float32(1.0) / unit
    return np.rint(s.astype(np.float64) * inv.astype(np.float64)), unit   # 8 x 24 bits: the product is exact


def bf16_scales(octaves: int) -> np.ndarray:
    """(tiles, 32): every bf16 significand as the largest scale of a tile against every bf16 number down to 2^-octaves."""
    sig = 1.0 + np.arange(128) / 128.0
    low = (sig[None] * 0.5 ** np.arange(octaves)[:, None]).ravel()
    low = np.pad(low, (0, -len(low) % (TOKENS - 1)), constant_values=low[-1]).reshape(-1, TOKENS - 1)
    rows = [np.concatenate([np.full((len(low), 1), a), np.minimum(low, a)], 1) for a in sig]
    return np.concatenate(rows).astype(np.float32)


@pytest.mark.parametrize("group", [4, 8])
def test_every_pair_of_scales(group):
    s = bf16_scales(9)
    want, unit = levels(s)
    got = tile_weights(s, group) / unit
    # a weight is a level times the unit as an fp16 number (127 * 2^-12 of a unit) and comes out of a sum of 8 * 32 * 127 units
    # at most in fp32 (2^-8): well within the half that tells two levels apart
    assert np.array_equal(np.rint(got), want)
    assert np.abs(got - want).max() < 0.1


@pytest.mark.parametrize("group", [4, 8])
def test_signed_scales(group):
    s = bf16_scales(3)
    s[:, 1::2] *= -1.0
    want, unit = levels(s)
    got = tile_weights(s, group) / unit
    assert np.array_equal(np.rint(got), want)
    assert np.abs(got - want).max() < 0.1


@pytest.mark.parametrize("group", [4, 8])
def test_scales_whose_weights_saturate(group):
    s = bf16_scales(9) * np.float32(2.0 ** 115)
    want, _ = levels(s)
    assert np.array_equal(tile_weights(s, group), np.where(want > 0, np.float32(65504.0), np.float32(0.0)))
