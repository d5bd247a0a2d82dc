"""The reference point of the split kernel's exponentials: the query heads of a token move it together, and no other token of a
chunk moves it with them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D = 128


def _store(h, k, v, bits=4, bs=16, kg=16, dtype="float16"):
    """One context of ``k`` / ``v`` ``[tokens, h, D]`` in blocks in order, and its block table (one row)."""
    import torch
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    blocks = -(-k.shape[0] // bs)
    layout = TieredLayout(num_kv_heads=h, head_size=D, block_size=bs, mem_bits=max(bits, 4), k_group=kg, v_group=32)
    store = TieredKVCache(layout, torch.zeros(blocks + 1, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=getattr(torch, dtype))
    store.write(k, v, torch.arange(k.shape[0]), bits)
    return store, torch.arange(blocks, device="cuda", dtype=torch.int32)[None]


@pytest.mark.parametrize("bits", [8, 4, 2])
def test_a_head_moves_with_its_neighbour(bits):
    """32 tokens of score 0 and value 0, then 32 of score d and value 1.  The neighbour's scores rise by 20, so the reference of the
    first head moves to d as well: its probabilities are 1 and the average is 1 / (1 + 2^-d) up to the fp32 arithmetic (1e-5).
    With the reference left at 0 the probability 2^d would be rounded to fp16 (1e-4 of the average here)."""
    import torch
    from echokv_b200.kernels.decode import decode_attention

    d = 0.255615234375
    k = torch.zeros(64, 1, D, device="cuda", dtype=torch.float16)
    k[32:, 0, 0] = 1.0
    v = torch.zeros_like(k)
    v[32:] = 1.0
    store, table = _store(1, k, v, bits)
    gk, gv = store.gather(torch.arange(64) // 16, torch.arange(64) % 16)
    assert torch.equal(gk.cpu().float(), k.cpu().float()) and torch.equal(gv.cpu().float(), v.cpu().float())
    q = torch.zeros(1, 2, D, device="cuda", dtype=torch.float16)
    q[0, 0, 0], q[0, 1, 0] = d, 20.0
    got = decode_attention(store, q, table, torch.tensor([64], device="cuda"), float(np.log(2.0)), 4, num_splits=1)
    assert (got[0, 0] - 1 / (1 + 2.0 ** -d)).abs().max() <= 1e-5


@pytest.mark.parametrize("h,gqa,bits", [(2, 1, 4), (2, 2, 8), (2, 3, 4), (2, 4, 2), (1, 4, 4)])
def test_a_token_moves_alone(h, gqa, bits):
    """Scores that outgrow the reference often: a chunk's tokens have the bits of each token alone."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.kernels.prefill import prefill_attention

    gen = torch.Generator(device="cuda").manual_seed(gqa)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    store, table = _store(h, rand(255, h, D) * torch.linspace(0.2, 5, 255, device="cuda").half()[:, None, None], rand(255, h, D), bits)
    q, out = rand(13, h * gqa, D) * 4, torch.zeros(13, h * gqa, D, device="cuda")
    prefill_attention(store, q, out, [(0, 13, 255, 0)], [0], table, D ** -0.5)
    lens = torch.arange(243, 256, device="cuda")
    want = decode_attention(store, q, table, lens, D ** -0.5, bt_rows=torch.zeros_like(lens), max_len=255)
    assert torch.equal(out, want)
