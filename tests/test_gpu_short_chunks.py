"""Short prompt chunks (at most 64 tokens): what a call returns, accepts and allocates follows from the chunk itself, not
from the chunks it shares a step with."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, D, BS, KG = 2, 128, 64, 32


def _store(tokens: int, dtype, value_top: float | None = None, h: int = H, bits: int = 4):
    """One stored context of ``tokens`` tokens at ``bits`` (values N(0, 1), or uniform up to ``value_top``), and its block table
    (one row)."""
    import torch
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    blocks = -(-tokens // BS)
    layout = TieredLayout(num_kv_heads=h, head_size=D, block_size=BS, mem_bits=bits, k_group=KG, v_group=32)
    pages = torch.zeros(blocks + 1, layout.page_bytes, dtype=torch.uint8, device="cuda")
    store = TieredKVCache(layout, pages, residual_slots=4, residual_dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    k = torch.randn(tokens, h, D, device="cuda", generator=gen).to(dtype)
    v = torch.randn(tokens, h, D, device="cuda", generator=gen)
    if value_top is not None:
        v.uniform_(0.0, value_top, generator=gen)
    v = v.to(dtype)
    order = np.random.default_rng(tokens).permutation(blocks + 1)[:blocks].astype(np.int32)
    pos = np.arange(tokens)
    store.write(k, v, torch.from_numpy(order[pos // BS].astype(np.int64) * BS + pos % BS), bits)
    return store, torch.from_numpy(order[None]).cuda()


def _query(rows: int, gqa: int, dtype, h: int = H):
    import torch

    return torch.randn(rows, h * gqa, D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).to(dtype)


def _attend(store, query, table, chunks, out=None):
    """``chunks``: (tokens, context) per request, all over the one stored context."""
    import torch
    from echokv_b200.kernels.prefill import build_rows, prefill_attention

    ends = np.cumsum([n for n, _ in chunks])
    prefill = [(int(e - n), int(e), ctx, 0) for e, (n, ctx) in zip(ends, chunks)]
    req_of = list(range(len(chunks)))
    table = table.expand(len(chunks), -1).contiguous()
    out = torch.zeros_like(query) if out is None else out
    prefill_attention(store, query, out, prefill, req_of, table, D ** -0.5, rows=build_rows(prefill, req_of, query.device))
    return out


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_a_chunk_does_not_depend_on_its_neighbours(dtype):
    """The same bits alone, among chunks that fill the chip, and token by token through decode attention."""
    import torch
    from echokv_b200.kernels.decode import decode_attention

    dt = getattr(torch, dtype)
    store, table = _store(4000, dt)
    chunks = [(33, 1472)] + [(40 + i, 4000 - 17 * i) for i in range(16)]
    q = _query(sum(n for n, _ in chunks), 4, dt)
    together = _attend(store, q, table, chunks)
    at = 0
    for n, ctx in chunks[:3]:
        alone = _attend(store, q[at: at + n], table, [(n, ctx)])
        assert torch.equal(alone, together[at: at + n])
        lens = torch.arange(ctx - n + 1, ctx + 1, device="cuda")
        want = torch.zeros_like(alone)
        decode_attention(store, q[at: at + n], table, lens, D ** -0.5, bt_rows=torch.zeros_like(lens), out=want, max_len=ctx)
        assert torch.equal(alone, want)
        at += n


@pytest.mark.parametrize("form", ["odd output stride", "output off 16 bytes", "query off 16 bytes", "odd query stride",
                                  "head dimension strided"])
def test_any_strides_and_alignment(form):
    """Every form of query and output that a lone short chunk takes is taken by a step of many of them."""
    import torch

    store, table = _store(2000, torch.float16)
    chunks = [(48, 2000)] * 16
    q = _query(48 * 16, 4, torch.float16)
    want = _attend(store, q, table, chunks)
    rows, hq = q.shape[:2]
    query, out = q, torch.zeros_like(q)
    if form == "odd output stride":
        out = torch.zeros(rows * hq * (D + 1), device="cuda", dtype=q.dtype).view(rows, hq, D + 1)[..., :D]
    elif form == "output off 16 bytes":
        out = torch.zeros(rows * hq * D + 1, device="cuda", dtype=q.dtype)[1:].view(rows, hq, D)
    elif form == "query off 16 bytes":
        query = torch.empty(q.numel() + 1, device="cuda", dtype=q.dtype)[1:].view_as(q).copy_(q)
    elif form == "odd query stride":
        query = torch.empty(rows, hq, D + 1, device="cuda", dtype=q.dtype)[..., :D].copy_(q)
    else:
        query = q.transpose(1, 2).contiguous().transpose(1, 2)
    assert torch.equal(_attend(store, query, table, chunks, out), want)


def test_values_beyond_the_range_of_fp16():
    """bf16 values of up to 2e5 are stored as codes with statistics that fit fp16; their average is as finite as they are.
    Against 64-bit attention over the stored values: 1e-2 covers the bf16 output (2^-9) and fp16 operands (2^-11)."""
    import torch

    store, table = _store(2000, torch.bfloat16, value_top=2e5, bits=8)
    k, v = store.gather(table[0].long().repeat_interleave(BS)[:2000], torch.arange(2000) % BS)
    assert v.max().item() > 1.9e5
    chunks = [(48, 2000)] * 16
    q = _query(48 * 16, 4, torch.bfloat16)
    got = _attend(store, q, table, chunks).float()
    assert torch.isfinite(got).all()
    kf, vf = (x.transpose(0, 1).repeat_interleave(4, 0).double() for x in (k, v))
    qf = q[:48].transpose(0, 1).double()
    mask = torch.arange(2000, device="cuda")[None] <= 1952 + torch.arange(48, device="cuda")[:, None]
    want = torch.softmax((qf @ kf.transpose(1, 2) * D ** -0.5).masked_fill(~mask, -torch.inf), -1) @ vf
    assert (got[:48].double() - want.transpose(0, 1)).norm() <= 1e-2 * want.norm()


def test_temporaries_are_the_split_partials():
    """No copy of the contexts is made: beside the split partials (which the library keeps) a step allocates next to nothing."""
    import torch

    store, table = _store(8000, torch.bfloat16, h=8)
    chunks = [(33, 8000)] * 16  # 512 MiB as dense 16-bit K and V
    q = _query(33 * 16, 4, torch.bfloat16, h=8)
    out = _attend(store, q, table, chunks)  # the partials' buffer grows to its size
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    _attend(store, q, table, chunks, out)
    assert torch.cuda.max_memory_allocated() - before <= 16 << 20
