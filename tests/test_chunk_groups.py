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
            at += tokens
        assert at == len(want)


def test_counts_that_do_not_fit_are_refused():
    from echokv_b200 import _native as N

    chunks, room = np.array([[0, 5, 9, 0], [5, -2, 9, 1]]), np.zeros(64, dtype=np.int64)
    for count, tokens in ((1, 4), (1, 6), (2, 3), (-1, 0)):
        args = [room.ctypes.data] * 4
        assert N.lib.echokv_chunk_groups(chunks.ctypes.data, count, tokens, np.array([2]).ctypes.data, 1, *args) < 0 and not room.any()


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
