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


def test_split_sizes_of_the_cuda_core_kernel_follow_the_batch():
    """Whole rounds of a CTA's four warps for sequences that need the whole grid; twice the tokens, and for wide query groups 16
    blocks, where the batch fills the chip many times over."""
    from echokv_b200.kernels.decode import generic_blocks_per_split as size

    assert [size(bs, np.array([500]), 64, 8, 4) for bs in (16, 32, 48, 64, 256)] == [8, 4, 4, 4, 4]
    assert size(32, np.full(16, 12000), 64, 2, 1) == 8 and size(16, np.full(3, 20000), 64, 1, 1) == 20 and size(16, np.array([20001]), 64, 1, 1) == 20
    assert size(16, np.array([500, 0, 0]), 2, 1, 1) == 16 and size(16, np.zeros(4, dtype=np.int64), 64, 8, 16) == 8
    assert size(32, np.full(256, 900), 64, 8, 4) == 8 and size(16, np.full(256, 900), 64, 8, 4) == 16
    assert size(32, np.full(128, 700), 64, 8, 16) == 16 and size(16, np.full(8, 3000), 64, 8, 16) == 16 and size(64, np.full(128, 700), 64, 8, 16) == 4
    assert size(32, np.full(32, 1500), 64, 1, 16) == 4
    for gqa in (1, 4, 8, 16):  # any length fits the grid
        for top in (1, 63, 64, 65, 4097, 100000):
            for splits in (1, 3, 64):
                assert size(16, np.array([top, 1]), splits, 8, gqa) * splits * 16 >= top
