"""Launcher of split-K paged decode attention (``csrc/decode*.cu``).

Same call surface as the reference's ``echokv_vllm/kernels/decode.py``
``decode_attention`` (:44-92).  There is no PyTorch path.
"""

from __future__ import annotations

import functools

import numpy as np
import torch

from echokv_b200 import _native as N

BLOCKS_PER_SPLIT = 16
MAX_DECODE_SPLITS = 64  # upper bound of the split grid (backend.py:67-69 of the reference caps its fixed grid alike)
EAGER_MAX_SPLITS = 32   # calls that size their own grid (the prefill row path): their scratch grows with rows x splits
# Smallest split `choose_blocks_per_split` proposes: one pair of tiles.  With several warps per head in the merge, halving the
# splits of a step that leaves the chip idle shortens it: 1 x 500 tokens x 32 layers 0.519 -> 0.444 ms, 4 x 678 in blocks of 32
# 0.561 -> 0.546; larger steps choose the sizes they chose with 64.
# Probabilities are rounded to 16 bits against a split's own maximum, so results differ by 1e-3; they are no further from 64-bit attention over
# the same pages (2-norm, six seeds, 64 / 32 tokens: 1 x 500 at 8 bits 9.1e-4 / 7.6e-4, 4 bits 8.3e-4 / 7.2e-4, 2 bits 8.5e-4 / 8.6e-4, 4 x 1,900 at
# 4 bits 1.02e-3 / 0.95e-3).
MIN_SPLIT_TOKENS = 32
# The scratch of a runner grows with its split grid, which is fixed: one for models of 2,048 tokens in blocks of 16 that allows splits
# of 32 tokens everywhere would take 273 MB at 256 sequences x 32 heads x 128, twice that of splits of 64, for batches that fill the
# chip with far fewer splits.  So only a runner whose batches are small gets it (64 sequences of the same: 68 MB with 64 splits, 18 MB
# for 528 tokens); the others still cut sequences of up to half their longest into splits of 32 tokens.
GRID_SPLIT_TOKENS, FINE_GRID_BYTES = 64, 72 << 20
# Split size of a step whose shape takes the CUDA-core kernel: a CTA's four warps take a block each, and a batch that leaves the chip
# idle wants more CTAs.  8 heads of 64 channels, blocks of 32, ms a step with 16 and with 4 blocks: 1 x 6,000 tokens 0.341 -> 0.172,
# 4 x 900 0.344 -> 0.191, 32 x 1,500 0.623 -> 0.576, 128 x 700 0.530 -> 0.523, 8 x 12,000 0.525 -> 0.527; in blocks of 16 4 blocks are too
# few (32 x 1,500: 0.773 with 16, 0.690 with 8, 0.724 with 4), in blocks of 64 2 are (0.575, 0.584 with 4, 0.755 with 2).
GENERIC_SPLIT_BLOCKS, GENERIC_SPLIT_TOKENS = 4, 128
# A batch that fills the chip many times over only pays for finer splits, in partials written and read again: from so many CTAs
# times query heads per KV head on they have twice the tokens, and in blocks of up to 32 BLOCKS_PER_SPLIT blocks where more than
# eight heads' partials are as long as the pages they come from.  us a layer at 128 / 256 / 512 tokens: 256 x 900, 8 heads of 64, 4 query
# heads each, blocks of 16 342 / 328 / 348, of 32 269 / 257 / 268; 128 x 700 of the same 139 / 142 / 150, 118 / 118 / 119; 16 query heads each of
# 128 channels, blocks of 32, 128 x 700 565 / 525 / 507, 8 x 3,000 116 / 106 / 124 and, one KV head, 32 x 1,500 44 / 50 / 74; in blocks of
# 64 32 x 1,500 - / 282 / 295, 128 x 700 - / 547 / 533.
GENERIC_MANY, GENERIC_MANY_TOKENS = 12000, 256
MMA_COLUMNS = 8         # columns of the split kernel's MMAs: query heads of a token, or of consecutive tokens of a chunk
ITEM_COST_TILES = 4     # fixed cost of a (sequence, split) work item in units of one 16-token tile's work


def decode_parallelism(store, num_q_heads: int) -> int:
    """Work items the split kernel has in work at once on the current device (0: generic kernel)."""
    return int(N.lib.echokv_decode_parallelism(store.c_layout, int(num_q_heads)))


def split_grid(max_model_len: int, block_size: int, split_bytes: int, slots: int) -> int:
    """Splits of the fixed split grid of a runner whose largest batch writes ``split_bytes`` of partials per split.

    ``slots``: ``decode_parallelism``.  Where the tensor-core kernel runs the grid allows splits of ``MIN_SPLIT_TOKENS`` for sequences
    of ``max_model_len``, as long as its scratch stays within ``FINE_GRID_BYTES``; otherwise splits of ``GRID_SPLIT_TOKENS``."""
    blocks = -(-max_model_len // block_size)
    fine, coarse = (max(1, min(-(-blocks // max(1, tokens // block_size)), MAX_DECODE_SPLITS))
                    for tokens in (MIN_SPLIT_TOKENS, GRID_SPLIT_TOKENS))
    return fine if slots and fine * split_bytes <= FINE_GRID_BYTES else coarse


def generic_blocks_per_split(block_size: int, lens=None, num_splits: int = MAX_DECODE_SPLITS, num_kv_heads: int = 1, gqa: int = 1) -> int:
    """Blocks per split for a step on the CUDA-core kernel: the smallest, or those for sequences of cache lengths ``lens``."""
    b = max(GENERIC_SPLIT_BLOCKS, GENERIC_SPLIT_TOKENS // block_size)
    if lens is None:
        return b
    blocks = -(-np.asarray(lens) // block_size)
    # The kernel itself would fit longer sequences into the grid with splits of any number of blocks, five of which keep four warps busy
    # as long as eight: 16 x 12,000, 2 heads of 64, 8 query heads each, blocks of 32 100 us a layer with 3 to 6 blocks, 74 with 8.
    longest = -(-int(blocks.max(initial=0)) // num_splits)
    b = max(b, -(-longest // GENERIC_SPLIT_BLOCKS) * GENERIC_SPLIT_BLOCKS)
    if num_kv_heads * gqa * int((-(-blocks // b)).sum()) < GENERIC_MANY:
        return b
    return max(b, BLOCKS_PER_SPLIT if gqa > MMA_COLUMNS and block_size <= 32 else GENERIC_MANY_TOKENS // block_size)


def choose_blocks_per_split(lens, block_size: int, num_splits: int, slots: int) -> int:
    """Blocks per split for one decode step of sequences with cache lengths ``lens``.

    The split kernel works on ``slots`` (sequence, split) items at a time, so the step takes
    ``ceil(items / slots)`` waves of one item's time each: a split of b blocks costs ``b * block_size / 16 +
    ITEM_COST_TILES``.  Every split count up to ``num_splits`` is tried on the mean sequence and the
    cheapest wins (ties: fewer, larger splits, which leave less to merge); splits hold an even number of tiles.  The value is a launch
    parameter shared by all sequences of the step, so for a given value results stay batch-invariant.
    """
    lens = np.asarray(lens)
    live = lens[lens > 0]
    if live.size == 0 or slots <= 0:
        return BLOCKS_PER_SPLIT
    n = int(live.size)
    nb = -(-int((-(-live // block_size)).sum()) // n)  # blocks of the mean sequence
    tiles = max(1, block_size // 16)
    # all split counts at once: one after the other they were 40 us of a step's host time
    b = np.maximum(-(-nb // _split_counts(num_splits)), max(1, MIN_SPLIT_TOKENS // block_size))
    if tiles & 1:
        b += b & 1  # the kernel works a split off in pairs of tiles: an odd count leaves one tile on the slower single path
    waves = -(-(n * -(-nb // b)) // slots)
    cost = waves * (b * tiles + ITEM_COST_TILES)
    return int(b[cost == cost.min()].max())


@functools.lru_cache(maxsize=16)
def _split_counts(num_splits: int):
    """1 .. num_splits, read-only."""
    counts = np.arange(1, max(1, num_splits) + 1)
    counts.setflags(write=False)
    return counts


class _Scratch:
    """Per-device split-partials buffer, grown on demand.

    The buffer starts zeroed: its first 256 bytes are the split kernel's work-queue state, which every
    call leaves at zero.  A CUDA graph holds the address of the buffer it was captured with, so a buffer that a capture has
    used is never freed: when a later call needs more bytes (more sequences than the captured sizes, the
    row path of a long prefill, another model in the same process) a larger buffer takes over and the old
    one is kept alive for the graphs that point at it.
    """

    def __init__(self) -> None:
        self.buf: dict[torch.device, torch.Tensor] = {}
        self.captured: set[torch.device] = set()
        self.retired: list[torch.Tensor] = []

    def get(self, device, nbytes: int) -> torch.Tensor:
        cur = self.buf.get(device)
        capturing = torch.cuda.is_current_stream_capturing()
        if cur is None or cur.numel() < nbytes:
            if capturing:
                raise RuntimeError("decode scratch must be sized before CUDA-graph capture (run one eager step first)")
            if cur is not None and device in self.captured:
                self.retired.append(cur)
                self.captured.discard(device)
            cur = self.buf[device] = torch.zeros(max(nbytes, 1 << 20), dtype=torch.uint8, device=device)
        if capturing:
            self.captured.add(device)
        return cur


_scratch = _Scratch()


def decode_attention(store, query: torch.Tensor, block_table: torch.Tensor, seq_lens: torch.Tensor,
                     softmax_scale: float, blocks_per_split: int = BLOCKS_PER_SPLIT,
                     q_rows: torch.Tensor | None = None, bt_rows: torch.Tensor | None = None,
                     out: torch.Tensor | None = None, max_len: int | None = None,
                     num_splits: int | None = None, bps_dev: torch.Tensor | None = None,
                     planned: bool = False, groups: dict | None = None) -> torch.Tensor:
    """Attention of one query token per sequence over each sequence's cache.

    Sequence ``i`` uses query row ``q_rows[i]`` and block-table row ``bt_rows[i]``
    (default: row ``i``) with cache length ``seq_lens[i]``.  Without ``out``
    returns float32 ``[S, Hq, D]``; with ``out`` writes sequence ``i`` to
    ``out[q_rows[i]]`` in ``out``'s dtype; length-0 sequences (CUDA-graph padding)
    leave their row untouched.  Each sequence is cut into at most ``num_splits``
    splits of ``max(blocks_per_split, ceil(blocks / num_splits))`` blocks -- a
    function of the sequence alone, so results are batch-invariant.  ``bps_dev`` (one int32 on the
    device, or the low half of an int64) raises ``blocks_per_split`` at run time: a captured graph
    keeps reading it, so the host can size the splits for every replayed step.  ``planned``: a write of the
    same step is ahead on the stream, and everything but the queries and the pages' rows was final before it, so the
    kernel may read that while the kernel before it still runs.  ``groups`` (from
    ``kernels.prefill.build_rows``): the sequences are tokens of chunks; per number of tokens that share a pass the device int64
    tensors ``[G, 5]`` of their runs and ``[S]`` of their split lengths (``echokv_decode_chunks``); it excludes ``bps_dev``.
    """
    L = store.layout
    given = (block_table, seq_lens, q_rows, bt_rows)
    N.require_cuda(query, block_table, seq_lens, out)
    q_shape, q_s, bt_s = query.shape, query.stride(), block_table.stride()  # each in one call: this runs once per layer and step
    if len(q_shape) != 3 or q_shape[2] != L.head_size:
        raise ValueError("query must be [T, Hq, D]")
    if q_s[2] != 1:
        query = query.contiguous()
        q_s = query.stride()
    hq = q_shape[1]
    s = seq_lens.shape[0]
    dev = query.device
    if block_table.dtype != torch.int32 or bt_s[1] != 1:
        block_table = block_table.to(torch.int32).contiguous()
        bt_s = block_table.stride()
    lens = seq_lens if seq_lens.dtype == torch.long and seq_lens.is_contiguous() else seq_lens.long().contiguous()
    if q_rows is not None and (q_rows.dtype != torch.long or not q_rows.is_contiguous()):
        q_rows = q_rows.long().contiguous()
    if bt_rows is not None and (bt_rows.dtype != torch.long or not bt_rows.is_contiguous()):
        bt_rows = bt_rows.long().contiguous()
    if out is None:
        out = torch.empty(query.shape[0], hq, L.head_size, device=dev, dtype=torch.float32)
    o_s = out.stride()
    if o_s[2] != 1:
        raise ValueError("out must have a contiguous last dim")
    if num_splits is None:
        width = block_table.shape[1]
        max_blocks = width if max_len is None else min(width, -(-max_len // L.block_size))
        num_splits = max(1, min(-(-max_blocks // blocks_per_split), EAGER_MAX_SPLITS))
    if s == 0:
        return out
    nbytes = N.lib.echokv_decode_scratch_bytes(s, hq, L.head_size, num_splits)
    scratch = _scratch.get(dev, nbytes)
    if bps_dev is not None:
        N.require_cuda(bps_dev)
        if bps_dev.dtype not in (torch.int32, torch.int64) or bps_dev.numel() < 1:
            raise TypeError("bps_dev must hold one int32 / int64 on the device")
    if groups is not None and (bps_dev is not None or not isinstance(groups, dict)):
        raise ValueError("groups must be those of build_rows, without bps_dev")
    width = 0 if groups is None else MMA_COLUMNS * L.num_kv_heads // hq
    if groups is not None and width in groups:  # two or more tokens fit
        runs, split_lens = groups[width]
        N.require_cuda(runs, split_lens)
        if split_lens.shape[0] != s:
            raise ValueError("groups must list the sequences' tokens")
        N.check(N.lib.echokv_decode_chunks(
            store.c_layout, store.c_pages, store.c_res,
            query.data_ptr(), q_s[0], q_s[1], N.dtype_code(query.dtype), N.ptr(q_rows),
            block_table.data_ptr(), bt_s[0], N.ptr(bt_rows), lens.data_ptr(),
            scratch.data_ptr(), scratch.numel(),
            out.data_ptr(), o_s[0], o_s[1], N.dtype_code(out.dtype),
            float(softmax_scale), int(num_splits), int(blocks_per_split), runs.data_ptr(), runs.shape[0], width,
            split_lens.data_ptr(), s, hq, N.stream_ptr(dev)))
        return out
    # a conversion above is itself the kernel before this one
    planned = planned and given[0] is block_table and given[1] is lens and given[2] is q_rows and given[3] is bt_rows
    launch = N.lib.echokv_decode_step if planned else N.lib.echokv_decode_ex
    N.check(launch(
        store.c_layout, store.c_pages, store.c_res,
        query.data_ptr(), q_s[0], q_s[1], N.dtype_code(query.dtype), N.ptr(q_rows),
        block_table.data_ptr(), bt_s[0], N.ptr(bt_rows), lens.data_ptr(),
        scratch.data_ptr(), scratch.numel(),
        out.data_ptr(), o_s[0], o_s[1], N.dtype_code(out.dtype),
        float(softmax_scale), int(num_splits), int(blocks_per_split), N.ptr(bps_dev), s, hq, N.stream_ptr(dev)))
    return out
