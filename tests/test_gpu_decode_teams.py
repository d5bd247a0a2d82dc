"""Decode attention with more than four query heads per KV head; at one KV head and pages of 4 bits the split kernel runs fewer teams an SM:
fewer work items than teams and several rounds of them, every tier, lengths around tiles, pairs and splits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, TOKENS = 128, 700


@pytest.mark.parametrize("h,gqa,mem,teams", [(1, 5, 4, 8), (1, 8, 2, 8), (1, 4, 4, 10), (1, 8, 6, 10), (1, 8, 8, 10), (2, 8, 4, 6), (4, 8, 4, 4),
                                             (8, 4, 8, 2)])
def test_team_counts(h, gqa, mem, teams):
    """Which shapes run how many teams an SM."""
    import torch
    from echokv_b200.kernels.decode import decode_parallelism
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    layout = TieredLayout(num_kv_heads=h, head_size=D, block_size=16, mem_bits=mem, k_group=16, v_group=32)
    store = TieredKVCache(layout, torch.zeros(2, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=torch.float16)
    assert decode_parallelism(store, h * gqa) == teams * torch.cuda.get_device_properties("cuda").multi_processor_count


@pytest.mark.parametrize("bits", [8, 4, 2])
@pytest.mark.parametrize("h,gqa", [(1, 5), (1, 8), (4, 7), (4, 8)])
def test_fewer_teams(h, gqa, bits):
    """Against 64-bit attention over the stored values: fp16 operands, 2^-11 per product, 2e-3 of the norm."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    bs, blocks = 16, -(-TOKENS // 16)
    layout = TieredLayout(num_kv_heads=h, head_size=D, block_size=bs, mem_bits=8 if bits == 8 else 4, k_group=16, v_group=32)
    store = TieredKVCache(layout, torch.zeros(blocks + 1, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=torch.float16)
    gen = torch.Generator(device="cuda").manual_seed(h * 10 + gqa)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    order = np.random.default_rng(bits).permutation(blocks + 1)[:blocks].astype(np.int32)
    pos = np.arange(TOKENS)
    store.write(rand(TOKENS, h, D), rand(TOKENS, h, D), torch.from_numpy(order[pos // bs].astype(np.int64) * bs + pos % bs), bits)
    k, v = store.gather(torch.from_numpy(order[pos // bs].astype(np.int64)), torch.from_numpy(pos % bs))
    kf, vf = (x.transpose(0, 1).repeat_interleave(gqa, 0).double() for x in (k, v))
    for lens in ([700], [1, 15, 16, 17, 32, 33, 700], np.resize([700, 64, 65, 31, 256, 1, 699], 300)):
        lens = torch.as_tensor(np.asarray(lens), device="cuda")
        n = lens.numel()
        q = rand(n, h * gqa, D)
        table = torch.from_numpy(np.tile(order, (n, 1))).cuda()
        got = decode_attention(store, q, table, lens, D ** -0.5, 4, num_splits=11).double()
        hidden = torch.arange(TOKENS, device="cuda")[None] >= lens[:, None]
        s = torch.einsum("nhd,htd->nht", q.double(), kf) * D ** -0.5
        want = torch.einsum("nht,htd->nhd", torch.softmax(s.masked_fill(hidden[:, None], -torch.inf), -1), vf)
        assert ((got - want).flatten(1).norm(dim=1) <= 2e-3 * want.flatten(1).norm(dim=1)).all()
