"""The split size of a decode step: every split count is tried, and the answer is that of trying them one after the other."""

import numpy as np
import pytest


@pytest.mark.parametrize("block_size", [16, 32, 48, 64, 128])
@pytest.mark.parametrize("num_splits", [1, 9, 64, 100])
def test_the_cheapest_split_count_wins(block_size, num_splits):
    from echokv_b200.kernels.decode import ITEM_COST_TILES, MIN_SPLIT_TOKENS, choose_blocks_per_split

    rng = np.random.default_rng(block_size + num_splits)
    for slots in (148, 296, 1480):
        for top in (40, 1000, 40000):
            lens = rng.integers(0, top, rng.integers(1, 200))
            lens[0] = top
            live = lens[lens > 0]
            nb = int(np.ceil(np.mean(-(-live // block_size))))
            tried = []
            for s in range(1, num_splits + 1):
                b = max(max(1, MIN_SPLIT_TOKENS // block_size), -(-nb // s))
                b += (b * (block_size // 16)) & 1  # an even number of tiles
                waves = -(-(live.size * -(-nb // b)) // slots)
                tried.append((waves * (b * (block_size // 16) + ITEM_COST_TILES), -b))
            assert choose_blocks_per_split(lens, block_size, num_splits, slots) == -min(tried)[1]


@pytest.mark.parametrize("block_size,blocks", [(16, 8), (32, 4), (48, 4), (64, 4), (256, 4)])
def test_split_sizes_of_the_cuda_core_kernel(block_size, blocks):
    from echokv_b200.kernels.decode import generic_blocks_per_split

    assert generic_blocks_per_split(block_size) == blocks


def test_the_split_grid_of_short_models_is_fine_only_where_its_scratch_is_small():
    """2,048 tokens in blocks of 16, 32 heads of 128: a runner of 256 sequences keeps the 136 MB of splits of 64 tokens, one of 64
    sequences has splits of 32 throughout; the CUDA-core kernel never cuts so fine."""
    from echokv_b200.kernels.decode import FINE_GRID_BYTES, split_grid

    row = 32 * (128 + 2) * 4
    assert split_grid(2048, 16, 256 * row, 296) == 32 and 32 * 256 * row < 137 << 20
    assert split_grid(2048, 16, 64 * row, 296) == 64 and 64 * 64 * row <= FINE_GRID_BYTES
    assert split_grid(2048, 16, 64 * row, 0) == 32
    assert split_grid(528, 16, 64 * row, 296) == 17 and split_grid(528, 16, 512 * row, 296) == 9
    for slots in (0, 296):  # blocks of 64 tokens and more, and long models: one answer
        assert split_grid(2048, 64, row, slots) == split_grid(2048, 64, 512 * row, slots) == 32
        assert split_grid(100000, 16, row, slots) == split_grid(100000, 16, 512 * row, slots) == 64
        assert split_grid(1, 16, row, slots) == 1
