"""What the kernels of a step may read before the kernels ahead of them have completed.

The split kernel of a planned decode step reads the step's metadata (lengths, rows, block table, page headers, residual map)
ahead of its dependency wait.  Every kernel of a step lets its dependents start at once, so that is sound only because the
step's first write is launched the ordinary way, behind everything that wrote the metadata.  Such a race rarely shows in
results, so the launches themselves are checked, and the results where the metadata was written an instant before."""

import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "echokv_b200" / "csrc"


def _body(file: str, name: str) -> str:
    """Text of kernel ``name``: from its parameter list to the closing brace in column 0."""
    text = (CSRC / file).read_text()
    at = re.search(r"^(?:__global__[^;{]*?)?\b" + name + r"\(", text, re.M).start()
    return text[at: text.index("\n}\n", at)]


def test_the_first_write_of_a_step_starts_when_everything_before_it_has_completed():
    """Its launch carries no programmatic attribute; the writes of further layers may overlap the kernel before them."""
    text = (CSRC / "write.cu").read_text()
    assert text.count("launch_after(!first, write_step_kernel<T,") == 2 == text.count("write_step_kernel<T,")
    first, nxt = (text[text.index(f"int {name}("):] for name in ("echokv_write_step_first", "echokv_write_step"))
    assert "stash_dst, stash_row_bytes, true, stream);" in first[: first.index("\n}\n")]
    assert "stash_dst, stash_row_bytes, false, stream);" in nxt[: nxt.index("\n}\n")]
    assert "cfg.numAttrs = early ? 1 : 0;" in (CSRC / "common.cuh").read_text()


def test_no_load_that_may_be_moved_ahead_of_the_wait():
    """``__ldg`` promises that nobody writes the word during the kernel's lifetime, which begins ahead of the wait."""
    assert not [f.name for f in CSRC.glob("decode*.cu*") if "__ldg" in f.read_text()]


def test_which_launches_a_step_makes(monkeypatch):
    """First write, further writes, decodes with and without a write ahead of them, and with tensors the call converts."""
    import torch
    from types import SimpleNamespace

    from echokv_b200 import _native as N
    from echokv_b200.kernels import decode, write
    from echokv_b200.write_plan import WriteMeta

    made = []
    fake = {n: (lambda *a, n=n: made.append(n) or 0) for n in N.EXPORTS if n.startswith(("echokv_write_step", "echokv_decode"))}
    fake["echokv_decode_scratch_bytes"] = lambda *a: 1024
    monkeypatch.setattr(N, "lib", SimpleNamespace(**fake))
    monkeypatch.setattr(N, "require_cuda", lambda *t: None)
    monkeypatch.setattr(N, "stream_ptr", lambda dev: 0)
    monkeypatch.setattr(decode._scratch, "get", lambda dev, n: torch.zeros(n, dtype=torch.uint8))
    store = SimpleNamespace(c_layout=None, c_pages=None, c_res=None, layout=SimpleNamespace(head_size=64, block_size=16))
    kv, one = torch.zeros(3, 2, 64), torch.ones(1, dtype=torch.long)
    table, rows = torch.zeros(3, 4, dtype=torch.int32), torch.zeros(3, dtype=torch.long)
    meta = WriteMeta(tok=torch.zeros(4, 3, dtype=torch.long), fin=torch.zeros(0, 19, dtype=torch.long), fin_count=one, n_rows=3, n_fin=0)

    def attend(table=table, lens=rows, q_rows=rows):
        decode.decode_attention(store, kv, table, lens, 1.0, q_rows=q_rows, bt_rows=rows, out=kv, planned=meta.launched)

    attend()
    write.write_step(store, kv, kv, meta)
    attend()
    write.write_step(store, kv, kv, meta)
    attend()
    attend(table=table.long())
    attend(lens=rows.int())
    attend(q_rows=rows.int())
    empty = WriteMeta(tok=meta.tok, fin=meta.fin, fin_count=one, n_rows=0, n_fin=0)
    write.write_step(store, kv[:0], kv[:0], empty)
    assert not empty.launched
    assert made == ["echokv_decode_ex", "echokv_write_step_first", "echokv_decode_step", "echokv_write_step", "echokv_decode_step"] + \
        ["echokv_decode_ex"] * 3


def test_split_kernel_waits_first_unless_the_step_was_planned():
    """Nothing but shared memory is touched before the wait, which only the producer of a planned step puts off."""
    body = _body("decode_mma.cu", "decode_mma_kernel")
    ahead = body[: body.index("if (!A.planned) pdl_wait();")]
    assert not re.search(r"A\.(lens|q_rows|bt|bt_rows|bps_dev|q)\b|bps_floor|P\.pages|P\.R\b|l2_prefetch", ahead)
    assert "if (warp != H) pdl_wait();" in ahead


def test_merge_waits_first_unless_the_step_was_planned():
    """Of the step's metadata, which one function reads, the merge sees nothing ahead of its wait unless the step was planned; the splits'
    partials, its item counter and the output row are touched behind the wait."""
    body = _body("decode.cu", "decode_merge_kernel")
    ahead, behind = body.split("pdl_wait();", 1)
    plan = ahead[ahead.index("auto plan = [&]()"): ahead.index("};")]
    metadata, results = r"A\.(lens|q_rows|bps_dev)\b|bps_floor", r"A\.(ml|acc|state|out)\["
    assert re.search(metadata, plan) and not re.search(metadata, ahead.replace(plan, "")) and not re.search(metadata, behind)
    assert re.findall(r".*plan\(\);", ahead.replace(plan, "")) == ["  if (A.planned) plan();"]
    assert re.findall(r".*plan\(\);", behind) == ["  if (W == 1 && !A.planned) plan();", "  if (W > 1 && !A.planned) plan();"]
    assert not re.search(results, ahead)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n", [2, 60, 150, 400])
def test_merges_of_planned_steps(n, d):
    """Steps of 2 to 400 sequences of eight query heads over a grid of 64 splits, all the numbers of warps a head, padding rows among them:
    eager and as one replayed graph whose lengths, rows and split sizes change, the bits of a decode that plans nothing."""
    import torch
    from echokv_b200.controller import ControllerParams, LayerController
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.step import GroupRunner
    from echokv_b200.tiered_cache import TieredLayout

    h, bs, layers, held = 2, 16, 2, 4  # four sequences are stored, the step's read them over and over
    layout = TieredLayout(num_kv_heads=h, head_size=d, block_size=bs, mem_bits=8, k_group=16, v_group=32)
    per = 4096 // bs
    caches = [torch.zeros(held * per + n, layout.page_bytes, dtype=torch.uint8, device="cuda") for _ in range(layers)]
    runner = GroupRunner(layout, caches, 4 * h, d ** -0.5, [LayerController(ControllerParams(fixed_bits=b)) for b in (4, 8)],
                         residual_slots=n + held, model_dtype=torch.bfloat16, cap=512, max_model_len=4096)
    assert runner.num_splits == 64
    gen = torch.Generator(device="cuda").manual_seed(n + d)
    draw = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).bfloat16()
    for at in range(0, held * 4096, 8192):
        meta = runner.plan_step(np.arange(at, at + 8192))
        for i in range(layers):
            runner.write(i, draw(8192, h, d), draw(8192, h, d), meta)
    table = torch.arange(held * per, device="cuda", dtype=torch.int32).view(held, per)
    kv, q, out = draw(2, layers, n, h, d), draw(layers, n, 4 * h, d), torch.zeros(layers, n, 4 * h, d, device="cuda")
    own = held * 4096 + np.arange(n) * bs  # the tokens that the step itself stores, in blocks of their own
    rng = np.random.default_rng(n)

    def plan(step):
        top = (4096, 1000, 150, 20)[step % 4]
        lens = np.maximum(1, (top * rng.random(n)).astype(np.int64))
        lens[0], lens[1:: 7] = top, 0
        rows = rng.permutation(n)
        return runner.plan_step(own + step % bs, decode=(rows, rng.integers(0, held, n), lens)), lens

    def layers_of(meta, capturing):
        for i in range(layers):
            runner.write(i, kv[0, i], kv[1, i], meta, capturing=capturing)
            runner.decode(i, q[i], table, out[i], meta)

    graph, sizes, used = None, set(), set()
    for step in range(16):
        meta, lens = plan(step)
        if step == 8:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                layers_of(meta, True)
        out.fill_(7.0)
        if graph is None:
            layers_of(meta, False)
            assert meta.write.launched
        else:
            graph.replay()
        size = int(meta.bps_dev[0])
        sizes.add(size)
        used.update(-(-(-(-lens // bs)) // max(size, runner.split_floor)))
        for i in range(layers):
            want = torch.full_like(out[i], 7.0)
            decode_attention(runner.stores[i], q[i], table, meta.decode_lens, d ** -0.5, runner.split_floor, q_rows=meta.decode_rows,
                             bt_rows=meta.decode_reqs, out=want, num_splits=64, bps_dev=meta.bps_dev)
            assert torch.equal(out[i], want)
            assert bool((out[i][meta.decode_rows[torch.from_numpy(lens == 0).cuda()]] == 7.0).all())
    assert len(used) > 3 and (d == 64 or len(sizes) > 1)  # the CUDA-core kernel has one size here


@pytest.mark.gpu
def test_metadata_written_by_the_kernel_right_before():
    """Lengths, rows, tables and split sizes that a kernel just produced, or that the call itself converts, give the bits of
    settled ones."""
    import torch
    from test_gpu_short_chunks import D, _query, _store

    from echokv_b200.kernels.decode import decode_attention

    store, table = _store(1000, torch.bfloat16)
    q = _query(12, 4, torch.bfloat16)
    gen = torch.Generator(device="cuda").manual_seed(1)
    tables, zero = table.expand(12, -1).contiguous(), torch.zeros(12, dtype=torch.long, device="cuda")
    for i in range(40):
        lens = torch.randint(1, 1001, (12,), device="cuda", generator=gen)
        perm = torch.randperm(12, device="cuda", generator=gen)
        size = torch.tensor([2 + i % 7], device="cuda")
        torch.cuda.synchronize()
        want = decode_attention(store, q, tables, lens, D ** -0.5, 1, q_rows=perm, bps_dev=size)
        torch.cuda.synchronize()
        got = decode_attention(store, q, tables.long() if i % 2 else tables + 0, lens.int() if i % 3 else lens + zero, D ** -0.5,
                               1, q_rows=perm.int() if i % 5 else perm + zero, bps_dev=size + 0, planned=bool(i % 2))
        assert torch.equal(got, want)


@pytest.mark.gpu
def test_eager_steps_whose_blocks_change_tier():
    """Steps that open blocks at another tier than the one they held, back to back: the planned decode behind each layer's
    write gives the bits of a decode of the settled store."""
    import torch
    from echokv_b200.controller import ControllerParams, LayerController
    from echokv_b200.kernels.decode import decode_attention
    from echokv_b200.step import GroupRunner
    from echokv_b200.tiered_cache import TieredLayout

    h, d, bs, n, layers = 2, 128, 16, 5, 3
    layout = TieredLayout(num_kv_heads=h, head_size=d, block_size=bs, mem_bits=8, k_group=16, v_group=32)
    caches = [torch.zeros(4 * n, layout.page_bytes, dtype=torch.uint8, device="cuda") for _ in range(layers)]
    ctls = [LayerController(ControllerParams(fixed_bits=8)) for _ in range(layers)]
    runner = GroupRunner(layout, caches, 4 * h, d ** -0.5, ctls, residual_slots=2 * n, model_dtype=torch.bfloat16, cap=32, max_model_len=64)
    table_np = np.random.default_rng(0).permutation(4 * n).reshape(n, 4).astype(np.int32)
    table = torch.from_numpy(table_np).cuda()
    gen = torch.Generator(device="cuda").manual_seed(2)
    rows = np.arange(n)
    for step in range(3 * 64):  # the blocks are written over and over, each time at another tier
        pos = step % 64
        for i, ctl in enumerate(ctls):
            ctl.bits = (2, 4, 8)[(step // 16 + i) % 3]
        kv = torch.randn(2, layers, n, h, d, device="cuda", generator=gen).bfloat16()
        q = torch.randn(layers, n, 4 * h, d, device="cuda", generator=gen).bfloat16()
        out = torch.zeros(layers, n, 4 * h, d, device="cuda")
        slots = table_np[:, pos // bs].astype(np.int64) * bs + pos % bs
        meta = runner.plan_step(slots, decode=(rows, rows, np.full(n, pos + 1)))
        for i in range(layers):
            runner.write(i, kv[0, i], kv[1, i], meta)
            runner.decode(i, q[i], table, out[i], meta)
        assert meta.write.launched
        torch.cuda.synchronize()
        for i in range(layers):
            want = decode_attention(runner.stores[i], q[i], table, meta.decode_lens, d ** -0.5, runner.split_floor,
                                    num_splits=meta.num_splits, bps_dev=meta.bps_dev)
            assert torch.equal(out[i], want)
