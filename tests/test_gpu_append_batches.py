"""An append whose blocks go through several batches writes the bytes that appends of single batches write."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,dtype", [((3, 2, 64), torch.bfloat16), ((4, 4, 128), torch.float16)])
@pytest.mark.parametrize("tokens", [3552, 6500, 9001, 12007, 16383, 32768])   # one to five batches of 16 tokens, 8 heads
def test_bytes_do_not_depend_on_the_batches(mode, dtype, tokens):
    from jetfire_b200 import ops
    kb, vb, gs = mode
    H = 8
    g = torch.Generator(device="cuda").manual_seed(tokens)
    k, v = (torch.randn(tokens, H, 128, generator=g, device="cuda").to(dtype) for _ in range(2))
    blocks = (tokens + 15) // 16 + 1
    slots = torch.randperm(16 * blocks, generator=g, device="cuda")[:tokens].contiguous()
    slots[5], slots[-1] = -1, -1
    caches = []
    for step in (tokens, 1000):
        c = [torch.full((H, 16 * blocks, 16 * b), 0x5A, dtype=torch.uint8, device="cuda") for b in (kb, vb)]
        s = [torch.zeros(H, 16 * blocks, 128 // gs, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        for lo in range(0, tokens, step):
            hi = min(lo + step, tokens)
            ops.fused_quant_write_kv(k[lo:hi], v[lo:hi], slots[lo:hi], c[0], s[0], c[1], s[1], gs, kb, vb)
        caches.append(c + s)
    for a, b in zip(*caches):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
