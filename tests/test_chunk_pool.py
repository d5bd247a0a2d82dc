"""Host decisions about the chunk pool of one layer, against the loops that define them."""

import numpy as np
import pytest


@pytest.mark.parametrize("form", [np.array, list, tuple, set, frozenset, iter, lambda b: dict.fromkeys(b), lambda b: np.array(b, dtype=np.int32)])
def test_block_ids_take_every_form(form):
    from echokv_b200.tiered_cache import block_ids

    for ids in ([3, 1, 7], []):
        got = block_ids(form(ids))
        assert got.dtype == np.int64 and got.ndim == 1 and sorted(got.tolist()) == sorted(ids)


def test_block_ids_of_a_tensor():
    import torch

    from echokv_b200.tiered_cache import block_ids

    assert block_ids(torch.tensor([4, 2])).tolist() == [4, 2]


@pytest.mark.parametrize("seed", range(6))
def test_release_of_blocks_of_mixed_tiers(seed):
    """Chunks return in block order, each block's first chunk first, whatever tiers the blocks hold."""
    from echokv_b200.tiered_cache import NEXTRA, ChunkPool

    rng = np.random.default_rng(seed)
    pool = ChunkPool(24, 4)
    for _ in range(4):
        pool.allot(rng.permutation(np.flatnonzero(pool.tier == 0))[:5], int(rng.choice([2, 4, 8])))
    blocks = rng.permutation(24)[:16]
    want, tier = list(pool.free), pool.tier.copy()
    for b in blocks.tolist():
        want += pool.table[b, : NEXTRA.get(int(tier[b]), 0)].tolist()
    assert len(set(tier.tolist())) > 2
    pool.release_many(blocks, 2)
    assert pool.free == want and (pool.tier[blocks] == 2).all()
    rest = np.setdiff1d(np.arange(24), blocks)
    assert np.array_equal(pool.tier[rest], tier[rest])


@pytest.mark.parametrize("seed", range(8))
def test_victims_are_those_of_the_sequential_loop(seed):
    """Every shortage from one chunk to more than there are, exact fits among them; blocks written in the same step, blocks
    that are not full, protected ones."""
    from echokv_b200.tiered_cache import NEXTRA, lru_victims

    rng = np.random.default_rng(seed)
    n = 20
    tier, full = rng.choice([0, 2, 4, 8], size=n), rng.random(n) < 0.7
    last, keep = rng.integers(0, 6, size=n), rng.permutation(n)[: int(rng.integers(0, 5))]
    for needed in range(1, 3 * n):
        want, freed = [], 0
        for b in sorted((b for b in range(n) if tier[b] >= 4 and full[b] and b not in keep), key=lambda b: (last[b], b)):
            if freed >= needed:
                break
            want.append(b)
            freed += NEXTRA[int(tier[b])]
        assert lru_victims(tier, full, last, needed, keep).tolist() == want


@pytest.mark.parametrize("keep", [[], [1], (1,), np.array([]), np.array([1.0]), np.array([1, -3, 99], dtype=np.int32)])
def test_kept_blocks_take_every_form(keep):
    """Lists, empty arrays (which are of floats) and ids outside the pool."""
    from echokv_b200.tiered_cache import lru_victims

    got = lru_victims(np.array([4, 8, 4]), np.ones(3, dtype=bool), np.arange(3), 9, keep)
    assert got.tolist() == ([0, 2] if 1 in keep else [0, 1, 2])


@pytest.mark.gpu
@pytest.mark.parametrize("form", [set, list, np.array])
def test_protected_blocks_of_every_form_stay(form):
    """Two full 8-bit blocks and no spare chunks: opening a third one demotes the older unless it is protected."""
    import torch

    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    layout = TieredLayout(num_kv_heads=2, head_size=64, block_size=32, mem_bits=4, k_group=32, v_group=32)
    for protect, demoted in ((None, 0), ([0], 1)):
        store = TieredKVCache(layout, torch.zeros(6, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                              residual_dtype=torch.bfloat16)
        for b in (0, 1):
            kv = torch.randn(2, 32, 2, 64, device="cuda").bfloat16()
            store.write(kv[0], kv[1], torch.arange(32) + 32 * b, 8)
        store.open_blocks(np.array([2]), 8, protect=None if protect is None else form(protect))
        assert store._tag_h[demoted] == 2 and store._tag_h[1 - demoted] == 8
