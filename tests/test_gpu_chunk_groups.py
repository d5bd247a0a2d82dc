"""Short chunks whose consecutive tokens share a pass over the pages (``echokv_decode_chunks``): every number of query heads per KV
head that packs several tokens, chunk lengths around the groups of eight, contexts that end around tiles, blocks and splits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, TOKENS = 128, 1100
# (tokens, context): groups of 1 .. 8, 9, 15 .. 17, 33, 64 tokens; a chunk that is its whole context; ends at 16, 32, 64, 256 and 1,024
CHUNKS = [(1, 1), (2, 2), (5, 16), (7, 17), (8, 40), (9, 33), (15, 64), (16, 66), (17, 256), (33, 259), (64, 64), (64, 1024), (6, 1026),
          (8, 1031), (3, 1099), (33, 1100)]


@pytest.mark.parametrize("h,gqa,bs,kg,mem,bits,dtype", [
    (8, 4, 64, 32, 4, 4, "bfloat16"), (8, 4, 16, 16, 8, 8, "float16"), (8, 4, 16, 16, 8, 2, "bfloat16"), (4, 3, 32, 16, 8, 4, "float16"),
    (2, 2, 16, 16, 8, 8, "bfloat16"), (2, 1, 64, 64, 4, 4, "float32"), (1, 1, 32, 32, 6, 8, "float16"), (1, 4, 16, 16, 4, 4, "bfloat16"),
    (2, 8, 64, 32, 4, 4, "bfloat16")])
def test_groups_of_tokens(h, gqa, bs, kg, mem, bits, dtype):
    """Against 64-bit attention over the stored values (fp16 operands: 2^-11 per product, 2e-3 of the norm) and against one token
    at a time (the probabilities are rounded against another maximum: 2^-11)."""
    import torch
    from echokv_b200.kernels.prefill import build_rows, prefill_attention
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    dt, blocks = getattr(torch, dtype), -(-TOKENS // bs)
    layout = TieredLayout(num_kv_heads=h, head_size=D, block_size=bs, mem_bits=mem, k_group=kg, v_group=32)
    store = TieredKVCache(layout, torch.zeros(blocks + 1, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=dt)
    gen = torch.Generator(device="cuda").manual_seed(h * 100 + gqa)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).to(dt)
    order = np.random.default_rng(bits).permutation(blocks + 1)[:blocks].astype(np.int32)
    pos = np.arange(TOKENS)
    store.write(rand(TOKENS, h, D), rand(TOKENS, h, D), torch.from_numpy(order[pos // bs].astype(np.int64) * bs + pos % bs), bits)
    table = torch.from_numpy(np.tile(order, (len(CHUNKS), 1))).cuda()
    ends = np.cumsum([n for n, _ in CHUNKS])
    prefill = [(int(e - n), int(e), ctx, 0) for e, (n, ctx) in zip(ends, CHUNKS)]
    req = list(range(len(CHUNKS)))
    q = rand(int(ends[-1]), h * gqa, D)
    rows = build_rows(prefill, req, "cuda")
    got, single = (torch.full(q.shape, 7.0, device="cuda") for _ in range(2))
    prefill_attention(store, q, got, prefill, req, table, D ** -0.5, rows=rows)
    prefill_attention(store, q, single, prefill, req, table, D ** -0.5, rows=tuple(rows))
    assert (got - single).norm() <= 1e-3 * single.norm()
    k, v = store.gather(torch.from_numpy(order[pos // bs].astype(np.int64)), torch.from_numpy(pos % bs))
    kf, vf = (x.transpose(0, 1).repeat_interleave(gqa, 0).double() for x in (k, v))
    for qs, qe, ctx, _ in prefill:
        hidden = torch.arange(TOKENS, device="cuda")[None] > torch.arange(ctx - (qe - qs), ctx, device="cuda")[:, None]
        s = (q[qs:qe].transpose(0, 1).double() @ kf.transpose(1, 2) * D ** -0.5).masked_fill(hidden, -torch.inf)
        want = (torch.softmax(s, -1) @ vf).transpose(0, 1)
        assert (got[qs:qe].double() - want).norm() <= 2e-3 * want.norm(), (qs, qe, ctx)
