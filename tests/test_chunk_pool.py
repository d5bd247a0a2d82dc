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
