"""Chunked-prefill attention over the tiered store (launchers for ``csrc/read.cu`` / ``csrc/prefill.cu``).

Call surface of the reference's ``echokv_vllm/kernels/prefill.py``
(``prefill_attention`` :170-207, ``dequant_dense`` :90-115,
``build_dequant_work`` :77-87).  A chunk's queries attend to the request's
whole stored context (this chunk included, already written), with a
bottom-right causal mask.  There is no PyTorch path.

Two device paths:
  * row path: every query token is handed to the split-K decode kernel as a
    sequence whose length is its causal limit; with up to four query heads per KV
    head, 2 to 8 consecutive tokens of a chunk share one pass over the pages.  Every
    such pass re-reads the context, so this is for short chunks (the reference's fused path has the same
    trade-off, kernels/prefill.py:10-13).
  * dense path: dequantize every context once into ``[total_ctx, H, D]`` in the
    model dtype, then run the tensor-core attention kernel over it.
"""

from __future__ import annotations

import numpy as np
import torch

from echokv_b200 import _native as N
from echokv_b200._util import to_device
from echokv_b200.kernels.decode import decode_attention

ROW_PATH_MAX_CHUNK = 64  # longer chunks take the dense path when it is available
GROUP_WIDTHS = np.array([8, 4, 2], dtype=np.int64)  # tokens that share a pass with one, two, and three or four query heads per KV head


def build_dequant_work(prefill, req_of, block_size: int, device) -> torch.Tensor:
    """Work list ``[n, 4]`` int32: (request, block index, dense row of the block's first token, ctx);
    contexts are packed back to back in ``prefill`` order."""
    pairs = list(zip(prefill, req_of))
    ctx = np.array([p[2] for p, _ in pairs], dtype=np.int64)
    count = -(-ctx // block_size)
    rows = np.empty((int(count.sum()), 4), dtype=np.int32)
    rows[:, 0] = np.repeat(np.array([r for _, r in pairs], dtype=np.int64), count)
    rows[:, 1] = np.arange(rows.shape[0]) - np.repeat(np.cumsum(count) - count, count)
    rows[:, 2] = np.repeat(np.array([p[3] for p, _ in pairs], dtype=np.int64), count) + rows[:, 1].astype(np.int64) * block_size
    rows[:, 3] = np.repeat(ctx, count)
    return to_device(torch.from_numpy(rows), device)


def dequant_dense(store, work: torch.Tensor, total_ctx: int, block_table: torch.Tensor, dtype):
    """Dense ``[total_ctx, H, D]`` K and V (``dtype``) of the contexts in ``work``."""
    L = store.layout
    k = torch.empty(total_ctx, L.num_kv_heads, L.head_size, device=store.device, dtype=dtype)
    v = torch.empty_like(k)
    if work.numel():
        N.require_cuda(work, block_table)
        bt_s, k_s = block_table.stride(), k.stride()
        if block_table.dtype != torch.int32 or bt_s[1] != 1:
            block_table = block_table.to(torch.int32).contiguous()
            bt_s = block_table.stride()
        N.check(N.lib.echokv_dequant_dense(
            store.c_layout, store.c_pages, store.c_res, work.data_ptr(), work.shape[0],
            block_table.data_ptr(), bt_s[0], k.data_ptr(), v.data_ptr(), k_s[0], k_s[1],
            N.dtype_code(dtype), N.stream_ptr(store.device)))
    return k, v


class RowPlan(tuple):
    """What ``build_rows`` returns: a 4-tuple (query rows, block-table rows, causal limits, largest limit), with the same tokens in
    runs of consecutive ones as ``groups`` for ``decode_attention``."""

    groups: dict


def build_rows(prefill, req_of, device):
    """Row-path metadata: per query token its row, its request and its causal limit (device int64), and the largest limit."""
    chunks = np.array([(p[0], max(p[1] - p[0], 0), p[2], r) for p, r in zip(prefill, req_of)], dtype=np.int64).reshape(-1, 4)
    n, widths = int(chunks[:, 1].sum()), GROUP_WIDTHS.size
    buf, counts = np.empty((3 + 6 * widths) * n, dtype=np.int64), np.empty(widths, dtype=np.int64)
    words = [k * n for k in (0, 3, 3 + widths)]  # where the rows, the split lengths and the groups begin
    at = [buf.ctypes.data + 8 * w for w in words]
    total = N.lib.echokv_chunk_groups(chunks.ctypes.data, chunks.shape[0], n, GROUP_WIDTHS.ctypes.data, widths, *at, counts.ctypes.data)
    if total < 0:
        N.check(total)
    dev = to_device(torch.from_numpy(buf[: words[2] + 5 * total]), device)
    packed, lens, groups = dev[: words[1]].view(3, n), dev[words[1]: words[2]].view(widths, n), dev[words[2]:].view(-1, 5)
    plan = RowPlan((packed[0], packed[1], packed[2], int(buf[2 * n: 3 * n].max(initial=0))))
    plan.groups = {int(w): (g, lens[i]) for i, (w, g) in enumerate(zip(GROUP_WIDTHS, groups.split(counts.tolist())))}
    return plan


def build_dense(prefill, req_of, block_size: int, device):
    """Dense-path metadata, once per step for all layers: the dequantization work list, the total
    context rows, the chunk table ``[n, 4]`` int32 (q_start, q_end, ctx, dense_start) on the device and
    the longest chunk.  Contexts are packed back to back in ``prefill`` order; the fourth field of the
    incoming tuples is recomputed, not trusted."""
    packed, at = [], 0
    for qs, qe, ctx, _ in prefill:
        packed.append((qs, qe, ctx, at))
        at += ctx
    chunks = to_device(torch.tensor(packed, dtype=torch.int32).reshape(-1, 4), device)
    return build_dequant_work(packed, req_of, block_size, device), at, chunks, max(qe - qs for qs, qe, _, _ in packed)


def dense_attention(query: torch.Tensor, k: torch.Tensor, v: torch.Tensor, chunks: torch.Tensor, max_chunk: int,
                    out: torch.Tensor, softmax_scale: float, query_rows: int = 0) -> None:
    """Bottom-right causal attention of each chunk's queries over its dense context (``csrc/prefill.cu``).
    ``query [T, Hq, D]`` and ``k``/``v [total_ctx, H, D]`` share one 16-bit dtype; ``out [T, Hq, D]``.
    ``query_rows``: the chunks' query rows together, when known (it sizes the launch)."""
    N.require_cuda(query, k, v, chunks, out)
    q_s, k_s, o_s, q_shape, k_shape = query.stride(), k.stride(), out.stride(), query.shape, k.shape
    if query.dtype != k.dtype or k.dtype != v.dtype or k_s != v.stride():
        raise ValueError("query, K and V must share a dtype and K, V a layout")
    if q_s[2] != 1 or k_s[2] != 1 or o_s[2] != 1:
        raise ValueError("the head dimension must be contiguous")
    N.check(N.lib.echokv_prefill_ex(
        query.data_ptr(), q_s[0], q_s[1], k.data_ptr(), v.data_ptr(), k_s[0], k_s[1],
        k_shape[0], N.dtype_code(query.dtype), chunks.data_ptr(), chunks.shape[0], max_chunk, query_rows,
        out.data_ptr(), o_s[0], o_s[1], N.dtype_code(out.dtype), softmax_scale, q_shape[1],
        k_shape[1], q_shape[2], N.stream_ptr(query.device)))


def dense_supported(store, query: torch.Tensor) -> bool:
    return query.dtype in (torch.float16, torch.bfloat16) and store.layout.head_size in (64, 128)


def prefill_attention(store, query: torch.Tensor, output: torch.Tensor, prefill, req_of, block_table: torch.Tensor,
                      softmax_scale: float, tiles=None, gather=None, dense=None, rows=None) -> None:
    """Write attention for every prefill chunk into ``output [T, Hq, D]``.

    ``prefill`` holds ``(q_start, q_end, ctx, dense_start)`` per chunk and ``req_of`` the
    block-table row of each.  ``dense`` (from ``build_dense``) selects the dense path; ``rows``
    (from ``build_rows``) lets the metadata builder prepare the row path's indices once per step
    for all layers.  With neither, chunks longer than ``ROW_PATH_MAX_CHUNK`` take the dense path
    when the dtype and head size allow it.  ``tiles`` and ``gather`` belong to the reference's
    Triton and PyTorch paths and are ignored.
    """
    if not prefill:
        return
    out3 = output.view(output.shape[0], -1, query.shape[-1])
    if dense is None and rows is None and dense_supported(store, query) and \
            max(qe - qs for qs, qe, _, _ in prefill) > ROW_PATH_MAX_CHUNK:
        dense = build_dense(prefill, req_of, store.layout.block_size, query.device)
    if dense is not None and dense_supported(store, query):
        work, total, chunks, max_chunk = dense
        k, v = dequant_dense(store, work, total, block_table, query.dtype)
        dense_attention(query, k, v, chunks, max_chunk, out3, softmax_scale, sum(qe - qs for qs, qe, _, _ in prefill))
        return
    if rows is None:
        rows = build_rows(prefill, req_of, query.device)
    q_rows, reqs, lens, max_len = rows
    # Splits of the default size: a token's split then follows from its own context, and its bits from the request alone.
    decode_attention(store, query, block_table, lens, softmax_scale, q_rows=q_rows, bt_rows=reqs, out=out3,
                     max_len=max_len, groups=getattr(rows, "groups", None))
