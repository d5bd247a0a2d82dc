"""Which tokens of short chunks share a pass over the pages, and that they hold no more memory than tokens taken one by one."""

import numpy as np
import pytest


def _chunks(seed: int):
    """Chunks of 0 to 64 tokens on query rows with gaps, contexts from the chunk itself on."""
    rng = np.random.default_rng(seed)
    prefill, req_of, at = [], [], 0
    for _ in range(int(rng.integers(0, 9))):
        n = int(rng.choice([0, 1, 2, 3, 7, 8, 9, 17, 33, 64]))
        at += int(rng.integers(0, 3))
        prefill.append((at, at + n, n + int(rng.choice([0, 1, 15, 16, 500, 8190])), 0))
        req_of.append(int(rng.integers(0, 9)))
        at += n
    return prefill, req_of


@pytest.mark.parametrize("seed", range(12))
def test_groups_list_every_token_once(seed, monkeypatch):
    from echokv_b200.kernels import prefill as P

    monkeypatch.setattr(P, "to_device", lambda t, device: t)
    prefill, req_of = _chunks(seed)
    plan = P.build_rows(prefill, req_of, "cpu")
    want = [(qs + i, r, ctx - (qe - qs) + 1 + i) for (qs, qe, ctx, _), r in zip(prefill, req_of) for i in range(qe - qs)]
    assert list(zip(*(t.tolist() for t in plan[:3]))) == want and plan[3] == max((ln for *_, ln in want), default=0)
    chunk_of = [c for c, (qs, qe, _, _) in enumerate(prefill) for _ in range(qe - qs)]
    assert sorted(plan.groups) == [2, 4, 8]
    for width, (groups, split_lens) in plan.groups.items():
        at = 0
        lengths = [prefill[chunk_of[g[4]]][2] for g in groups.tolist()]
        assert lengths == sorted(lengths, reverse=True)  # long contexts first
        for row, req, length, tokens, first in sorted(groups.tolist(), key=lambda g: g[4]):
            assert first == at and 1 <= tokens <= width and len(set(chunk_of[at: at + tokens])) == 1
            assert want[at: at + tokens] == [(row + i, req, length - tokens + 1 + i) for i in range(tokens)]
            assert split_lens[at: at + tokens].tolist() == [length] * tokens
            for ln in range(length - tokens + 2, length + 1):  # nothing about the kernels' tiles and splits changes inside a group
                assert ln // 16 == (ln - 1) // 16 and (ln - 1) % 512
            at += tokens
        assert at == len(want)


@pytest.mark.gpu
@pytest.mark.parametrize("h,gqa,bits", [(2, 1, 4), (2, 2, 2), (2, 3, 8), (2, 4, 4), (1, 4, 4), (2, 4, 0), (8, 1, 0)])
def test_bits_of_each_token_alone(h, gqa, bits):
    """Contexts that pass the end of a tile, of a pair of tiles, of a split (256 tokens) and of 512 blocks, from where the split size
    follows the context; loud queries, so that the reference moves; ``bits`` 0: blocks of all tiers.  However the chunk is cut,
    a token has the bits of the token alone."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.kernels.prefill import prefill_attention
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    tokens, d = 8240, 128
    layout = TieredLayout(num_kv_heads=h, head_size=d, block_size=16, mem_bits=8, k_group=16, v_group=32)
    store = TieredKVCache(layout, torch.zeros(tokens // 16, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=torch.float16)
    gen = torch.Generator(device="cuda").manual_seed(gqa)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    for at in range(0, tokens, 16 if bits == 0 else tokens):
        n = 16 if bits == 0 else tokens
        store.write(rand(n, h, d), rand(n, h, d), torch.arange(at, at + n), bits or (8, 4, 4, 2, 4, 8, 2, 2)[at // 16 % 8])
    table = torch.arange(tokens // 16, device="cuda", dtype=torch.int32).expand(6, -1).contiguous()
    chunks = [(40, 1050), (64, 8230), (7, 8195), (37, 290), (5, 5), (20, 4110)]
    ends = np.cumsum([n for n, _ in chunks]).tolist()
    q = rand(ends[-1], h * gqa, d) * 4
    lens = torch.cat([torch.arange(ctx - n + 1, ctx + 1) for n, ctx in chunks]).cuda()
    reqs = torch.arange(6, device="cuda").repeat_interleave(torch.tensor([n for n, _ in chunks], device="cuda"))
    want = decode_attention(store, q, table, lens, d ** -0.5, bt_rows=reqs, max_len=8230)
    for cut in (64, 3):
        pieces = [(i, e - n + a, min(e - n + a + cut, e), ctx - n + min(a + cut, n)) for i, (e, (n, ctx)) in enumerate(zip(ends, chunks))
                  for a in range(0, n, cut)]
        out = torch.full(q.shape, 7.0, device="cuda")
        prefill_attention(store, q, out, [(a, b, ctx, 0) for _, a, b, ctx in pieces], [i for i, *_ in pieces], table, d ** -0.5)
        assert torch.equal(out, want)


def _mixed_store(h, tokens, dtype="float16"):
    """One context whose blocks of 16 tokens are of all tiers, and its block table (one row)."""
    import torch
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    layout = TieredLayout(num_kv_heads=h, head_size=128, block_size=16, mem_bits=8, k_group=16, v_group=32)
    store = TieredKVCache(layout, torch.zeros(tokens // 16, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=getattr(torch, dtype))
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    kv = torch.randn(2, tokens, h, 128, device="cuda", generator=gen).to(getattr(torch, dtype))
    for at in range(0, tokens, 16):
        store.write(kv[0, at: at + 16], kv[1, at: at + 16], torch.arange(at, at + 16), (8, 4, 4, 2, 4, 8, 2, 2)[at // 16 % 8])
    return store, torch.arange(tokens // 16, device="cuda", dtype=torch.int32)[None]


@pytest.mark.gpu
@pytest.mark.parametrize("h,gqa", [(8, 1), (2, 4), (1, 3)])
def test_long_contexts_of_all_tiers(h, gqa):
    """Behind more than 4,096 tokens and more than 512 blocks, against 64-bit attention over the stored values (fp16 operands: 2^-11
    per product, 2e-3 of the norm)."""
    import torch
    from echokv_b200.kernels.prefill import prefill_attention

    store, table = _mixed_store(h, 8208)
    k, v = (x.transpose(0, 1).repeat_interleave(gqa, 0).double() for x in store.gather(torch.arange(8208) // 16, torch.arange(8208) % 16))
    chunks = [(20, 8205), (9, 4101), (33, 4130)]
    q = torch.randn(62, h * gqa, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(h)).half()
    out = torch.full(q.shape, 7.0, device="cuda")
    prefill = [(0, 20, 8205, 0), (20, 29, 4101, 0), (29, 62, 4130, 0)]
    prefill_attention(store, q, out, prefill, [0, 1, 2], table.expand(3, -1).contiguous(), 128 ** -0.5)
    for (n, ctx), (qs, qe, _, _) in zip(chunks, prefill):
        hidden = torch.arange(8208, device="cuda")[None] >= torch.arange(ctx - n + 1, ctx + 1, device="cuda")[:, None]
        s = (q[qs:qe].transpose(0, 1).double() @ k.transpose(1, 2) * 128 ** -0.5).masked_fill(hidden, -torch.inf)
        want = (torch.softmax(s, -1) @ v).transpose(0, 1)
        assert (out[qs:qe].double() - want).norm() <= 2e-3 * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("gqa,shared", [(1, True), (2, True), (3, True), (4, True), (5, False), (8, False)])
def test_which_shapes_share_a_pass(gqa, shared):
    """With the lengths of the tokens one by one all wrong, the result follows the groups exactly where tokens are taken together."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.kernels.prefill import build_rows

    store, table = _mixed_store(2, 320)
    q = torch.randn(20, 2 * gqa, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(gqa)).half()
    plan = build_rows([(0, 20, 310, 0)], [0], "cuda")
    rows, reqs, lens, longest = plan
    attend = lambda lens, groups: decode_attention(store, q, table, lens, 128 ** -0.5, q_rows=rows, bt_rows=reqs, max_len=longest, groups=groups)
    wrong = torch.full_like(lens, 100)
    assert torch.equal(attend(wrong, plan.groups), attend(lens if shared else wrong, None))


@pytest.mark.gpu
@pytest.mark.parametrize("gqa", [1, 2, 4])
def test_tokens_that_see_nothing(gqa):
    """A chunk longer than its context: the row of the token with a causal limit of 0 stays as it is, those behind it have the bits of
    the token alone."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.kernels.prefill import prefill_attention

    store, table = _mixed_store(2, 320)
    q = torch.randn(40, 2 * gqa, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(gqa)).half()
    out = torch.full(q.shape, 7.0, device="cuda")
    prefill_attention(store, q, out, [(0, 40, 12, 0)], [0], table, 128 ** -0.5)
    lens = torch.arange(1, 13, device="cuda")
    want = decode_attention(store, q[28:], table, lens, 128 ** -0.5, bt_rows=torch.zeros_like(lens), max_len=12)
    assert (out[27] == 7.0).all() and torch.equal(out[28:], want)


@pytest.mark.gpu
@pytest.mark.parametrize("at", [160, 256])
@pytest.mark.parametrize("h,gqa,bits", [(2, 1, 4), (2, 2, 8), (2, 4, 2), (1, 3, 4), (2, 4, 0)])
def test_infinite_values_of_later_tokens(h, gqa, bits, at):
    """A token with an infinite value, in a tile that begins where the cache of some tokens of the chunk ends (160: inside a split,
    256: at a split's begin): those tokens do not see it.  ``bits`` 0: a tile of another tier than the ones before."""
    import torch
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.kernels.prefill import prefill_attention
    from echokv_b200.tiered_cache import TieredKVCache, TieredLayout

    d = 128
    layout = TieredLayout(num_kv_heads=h, head_size=d, block_size=16, mem_bits=8, k_group=16, v_group=32)
    store = TieredKVCache(layout, torch.zeros(20, layout.page_bytes, dtype=torch.uint8, device="cuda"), residual_slots=4,
                          residual_dtype=torch.float16)
    gen = torch.Generator(device="cuda").manual_seed(gqa)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    k, v = rand(320, h, d), rand(320, h, d)
    v[at + 5] = torch.inf
    for a, b in ((0, at), (at, 320)):
        store.write(k[a:b], v[a:b], torch.arange(a, b), bits or (4 if a else 8))
    table = torch.arange(20, device="cuda", dtype=torch.int32)[None]
    n, ctx = 18, at + 9  # lengths at - 8 .. at + 9
    q, out = rand(n, h * gqa, d), torch.full((n, h * gqa, d), 7.0, device="cuda")
    prefill_attention(store, q, out, [(0, n, ctx, 0)], [0], table, d ** -0.5)
    lens = torch.arange(ctx - n + 1, ctx + 1, device="cuda")
    want = decode_attention(store, q, table, lens, d ** -0.5, bt_rows=torch.zeros_like(lens), max_len=ctx)
    seen = lens <= at
    assert torch.isfinite(want[seen]).all() and torch.equal(out[seen], want[seen]) and not torch.isfinite(want[~seen]).any()


def test_counts_that_do_not_fit_are_refused():
    from echokv_b200 import _native as N

    chunks, room = np.array([[0, 5, 9, 0], [5, -2, 9, 1]]), np.zeros(64, dtype=np.int64)
    for count, tokens in ((1, 4), (1, 6), (2, 3), (-1, 0)):
        args = [room.ctypes.data] * 4
        assert N.lib.echokv_chunk_groups(chunks.ctypes.data, count, tokens, np.array([2]).ctypes.data, 1, *args) < 0 and not room.any()


@pytest.mark.parametrize("form,gqa", [("run-time split size", 4), ("run-time split size", 8), ("a tensor", 4), ("a tensor", 8),
                                      ("another step's groups", 4)])
def test_groups_that_do_not_fit_are_refused(form, gqa, monkeypatch):
    """Whether or not the shape takes tokens together."""
    import torch
    from types import SimpleNamespace

    from echokv_b200 import _native as N
    from echokv_b200.kernels import decode, prefill

    monkeypatch.setattr(prefill, "to_device", lambda t, device: t)
    monkeypatch.setattr(N, "require_cuda", lambda *t: None)
    monkeypatch.setattr(N, "stream_ptr", lambda dev: 0)
    monkeypatch.setattr(decode._scratch, "get", lambda dev, n: torch.zeros(n, dtype=torch.uint8))
    store = SimpleNamespace(c_layout=None, c_pages=None, c_res=None, layout=SimpleNamespace(num_kv_heads=2, head_size=64, block_size=16))
    rows, reqs, lens, longest = plan = prefill.build_rows([(0, 5, 9, 0)], [0], "cpu")
    groups, bps = plan.groups, None
    if form == "run-time split size":
        bps = torch.ones(1, dtype=torch.int32)
    elif form == "another step's groups":
        groups = prefill.build_rows([(0, 3, 9, 0)], [0], "cpu").groups
    else:
        groups = groups[2][0]
    with pytest.raises(ValueError):
        decode.decode_attention(store, torch.zeros(5, 2 * gqa, 64), torch.zeros(1, 4, dtype=torch.int32), lens, 1.0, q_rows=rows,
                                bt_rows=reqs, max_len=longest, bps_dev=bps, groups=groups)


@pytest.mark.gpu
@pytest.mark.parametrize("h,gqa,n,chunks", [(8, 4, 2, 64), (8, 4, 3, 40), (2, 1, 1, 100), (1, 2, 3, 33), (2, 8, 2, 20)])
def test_partials_of_the_tokens_there_are(h, gqa, n, chunks, monkeypatch):
    """Many chunks of one to three tokens: the scratch of as many sequences, and the bits of the tokens one by one."""
    import torch
    from test_gpu_short_chunks import D, _query, _store

    from echokv_b200 import _native as N
    from echokv_b200.kernels import decode
    from echokv_b200.kernels.prefill import prefill_attention

    store, table = _store(700, torch.float16, h=h)
    table = table.expand(chunks, -1).contiguous()
    ctx = 300 + 7 * np.arange(chunks) % 400
    prefill = [(n * c, n * c + n, int(ctx[c]), 0) for c in range(chunks)]
    q, out = _query(n * chunks, gqa, torch.float16, h), torch.full((n * chunks, h * gqa, D), 7.0, device="cuda")
    asked, get = [], decode._scratch.get
    monkeypatch.setattr(decode._scratch, "get", lambda dev, nbytes: asked.append(nbytes) or get(dev, nbytes))
    prefill_attention(store, q, out, prefill, list(range(chunks)), table, D ** -0.5)
    splits = -(-(-(-int(ctx.max()) // 64)) // 16)
    assert asked == [N.lib.echokv_decode_scratch_bytes(n * chunks, h * gqa, D, splits)]
    lens = torch.from_numpy((ctx[:, None] - n + 1 + np.arange(n)).ravel()).cuda()
    reqs = torch.arange(chunks, device="cuda").repeat_interleave(n)
    want = decode.decode_attention(store, q, table, lens, D ** -0.5, bt_rows=reqs, max_len=int(ctx.max()))
    assert (out - want).norm() <= 1e-3 * want.norm()
