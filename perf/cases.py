"""What a serving program has this package do, as measurable cases.

Every case drives the per-step path of one KV-cache group the way an engine does: ``GroupRunner.plan_step`` once per
step (write plan, block opening, one metadata upload), then per layer the quantize-on-write and the attention.  Four
kinds:

* ``decode``: one token per sequence.  The layers' launches are captured in a CUDA graph (engines replay decode steps
  as graphs) and every pass plans the next position and replays it; the canary is measured every eighth step.  The
  positions run through one block per sequence and start over, so blocks open, K groups complete and residual slots
  change hands at their ordinary rate, and a pass can be repeated for as long as wanted.
* ``prefill``: a chunk of prompt tokens per sequence behind ``ctx`` stored ones (0: new prompts), run eagerly.
* ``mixed``: decode tokens and one prompt chunk in the same eager step (chunked prefill).
* ``pressure``: one new prompt per pass into a pool that cannot hold every block at its tier, so that opening its
  blocks demotes the least recently written ones.

Keys are N(0, 1) with 1 % of the channels ten times larger, values and queries N(0, 1): seeded stand-ins for a model's
activations.  ``tiers`` is the cycle of per-layer bit widths, ``mem`` the page budget in bits, ``spread`` the ratio of
the shortest to the longest sequence.
"""

from __future__ import annotations

import numpy as np
import torch

from echokv_b200.controller import ControllerParams, LayerController
from echokv_b200.kernels.prefill import ROW_PATH_MAX_CHUNK, build_dense, build_rows, prefill_attention
from echokv_b200.step import GroupRunner
from echokv_b200.tiered_cache import TieredLayout

V_GROUP = 32
CANARY_EVERY, CANARY_ROWS = 8, 8
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
COST_LIMIT = 64 * 4096 * 8 * 16  # context tokens x KV heads x layers of the largest listed decode step


def _case(name, kind, h, gqa, d, bs, kg, mem, tiers, layers, seqs, ctx, chunk=0, spread=1.0, dtype="bf16") -> dict:
    case = dict(kind=kind, h=h, gqa=gqa, d=d, bs=bs, kg=kg, mem=mem, tiers=tiers, layers=layers, seqs=seqs, ctx=ctx,
                chunk=chunk, spread=spread, dtype=dtype)
    return dict(case, name=name) if name else case


def listed() -> list[dict]:
    return [
        # one user, a short conversation: launches and latency
        _case("decode_1x500", "decode", 8, 4, 128, 16, 16, 8, "8,4,2", 32, 1, 500),
        # a handful of users at the serving geometry (block 64, K groups of 32, 4-bit budget), ragged lengths
        _case("decode_8x2100_serving", "decode", 8, 4, 128, 64, 32, 4, "4", 32, 8, 2100, spread=0.2),
        # the benchmark's decode step: batch 64 at about 4,096 tokens, layers at all three tiers
        _case("decode_64x4096", "decode", 8, 4, 128, 16, 16, 8, "4,8,4,2", 16, 64, 4096, spread=0.9),
        # many short conversations at the serving geometry, fp16, layers the controller has brought down to 2 bits among them
        _case("decode_256x900_serving", "decode", 8, 4, 128, 64, 32, 4, "4,2", 8, 256, 900, spread=0.3, dtype="f16"),
        # one of eight tensor-parallel ranks of a 64 / 8-head model, long contexts
        _case("decode_16x32k_one_kv_head", "decode", 1, 8, 128, 16, 16, 4, "4", 16, 16, 32000, spread=0.6),
        # one of four ranks of the same model; 8-bit layers over a 6-bit budget: sequences of mixed tiers
        _case("decode_48x3000_mixed_tiers", "decode", 2, 8, 128, 32, 32, 6, "8", 8, 48, 3000, spread=0.5),
        # a small model with head size 64
        _case("decode_32x1500_head64", "decode", 8, 4, 64, 32, 32, 8, "8,4", 8, 32, 1500, spread=0.4, dtype="f16"),
        # chunked prefill at the end of long contexts (8 x 512 tokens behind 8,192 stored ones)
        _case("prefill_8x512_behind_8192", "prefill", 8, 4, 128, 16, 16, 8, "4,8", 8, 8, 8192, 512),
        # new prompts of uneven lengths at the serving geometry
        _case("prefill_12_prompts", "prefill", 8, 4, 128, 64, 32, 4, "4", 8, 12, 0, 2900, spread=0.03),
        # short follow-up chunks (tool outputs, draft tokens) behind short contexts
        _case("prefill_16x33_behind_1472", "prefill", 8, 4, 128, 64, 32, 4, "4", 8, 16, 1472, 33, spread=0.5),
        # one step of a busy engine: 63 decode tokens and a 512-token prompt chunk
        _case("mixed_63_and_512", "mixed", 8, 4, 128, 64, 32, 4, "4", 16, 63, 1600, 512, spread=0.3),
        # a prompt arrives while the pool is short: 8-bit blocks over a 4-bit budget, older blocks are demoted
        _case("pressure_24x1000", "pressure", 8, 4, 128, 16, 16, 4, "8", 4, 24, 0, 1000, spread=0.6),
    ]


def draw(rng) -> dict:
    """One more case of the same ranges, never dearer than the largest listed one."""
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["decode"] * 5 + ["prefill"] * 3 + ["mixed", "pressure"])
    d = rng.choice([128] * 6 + [64])
    h = rng.choice([8, 8, 8, 4, 2, 1])
    gqa = rng.choice([4, 4, 8, 7, 2, 1])
    bs, kg = rng.choice([(16, 16), (64, 32), (32, 32), (32, 16), (64, 64)])
    mem, tiers = rng.choice([(8, "8,4,2"), (4, "4"), (4, "4,2"), (8, "8"), (6, "8")])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    spread = round(rng.uniform(0.1, 1.0), 2)
    if kind == "decode":
        seqs, ctx, chunk = log(1, 256), log(100, 32000), 0
    elif kind == "prefill":
        seqs, chunk = log(1, 16), log(5, 1500)
        ctx = 0 if rng.random() < 0.4 else log(64, 8000)
    elif kind == "mixed":
        seqs, ctx, chunk = log(2, 96), log(100, 4000), log(65, 1024)
    else:
        seqs, ctx, chunk = log(4, 24), 0, log(100, 1200)
        mem, tiers = 4, "8"
    limit = COST_LIMIT // (1 if kind == "decode" else 4)
    while seqs > 1 and seqs * (ctx + chunk) * h * 4 > limit:
        seqs = max(1, seqs // 2)
    layers = max(1, min(32 if kind == "decode" else 8, limit // (seqs * (ctx + chunk + 64) * h)))
    return _case("", kind, h, gqa, d, bs, kg, mem, tiers, layers, seqs, ctx, chunk, spread, dtype)


# ---- sizes that follow from a case ------------------------------------------------------------------------------------

def _ragged(n: int, top: int, spread: float) -> np.ndarray:
    """``n`` lengths from ``spread * top`` to ``top``, spread evenly over their logarithm, odd ones among them."""
    if n == 1:
        return np.array([top])
    lo = max(1.0, spread * top)
    x = lo * (top / lo) ** (np.arange(n) / (n - 1))
    return np.random.default_rng(n * 1000 + top).permutation(np.maximum(1, np.round(x).astype(np.int64)))


def _lengths(c: dict):
    """Per sequence: tokens stored before the step (whole blocks), tokens of the step, decode phase inside the block."""
    bs, n = c["bs"], c["seqs"]
    zero = np.zeros(n, dtype=np.int64)
    if c["kind"] == "decode":
        return np.maximum(1, _ragged(n, c["ctx"], c["spread"]) // bs) * bs, zero + 1, (np.arange(n) * 7) % bs
    if c["kind"] == "mixed":  # the last sequence brings the prompt chunk
        base = np.maximum(1, _ragged(n, c["ctx"], c["spread"]) // bs) * bs
        base, step = np.append(base, base[0]), np.append(zero + 1, c["chunk"])
        return base, step, np.append((np.arange(n) * 7) % bs, 0)
    if c["kind"] == "prefill" and c["ctx"]:  # equal chunks (one token apart) behind ragged contexts
        return _ragged(n, c["ctx"], c["spread"]) // bs * bs, c["chunk"] - np.arange(n) % 2, zero
    return zero, _ragged(n, c["chunk"], c["spread"]), zero


def _tiers(c: dict) -> list[int]:
    cyc = [int(x) for x in c["tiers"].split(",")]
    return [cyc[i % len(cyc)] for i in range(c["layers"])]


def _token_bytes(c: dict, bits: int) -> float:
    """Stored bytes of one token of one layer: codes, V statistics, its share of the K statistics."""
    hd = c["h"] * c["d"]
    return hd * min(bits, c["mem"]) / 4 + 4 * hd / V_GROUP + 4 * hd / c["kg"]


def work(case: dict) -> dict:
    base, step, phase = _lengths(case)
    if case["kind"] == "pressure":  # one sequence per pass
        base, step, phase = base[:1], np.array([int(step.mean())]), phase[:1]
    hq, h, d = case["h"] * case["gqa"], case["h"], case["d"]
    ctx = (base + phase + step).astype(np.float64)
    rows = float(step.sum())
    seen = float((step * (ctx - step) + step * (step + 1) / 2).sum())  # (query token, visible key) pairs
    nbytes = 0.0
    for bits in _tiers(case):
        nbytes += (float(ctx.sum()) + rows) * _token_bytes(case, bits)  # every context read once, the step's tokens stored
        nbytes += rows * 2 * (2 * h * d + 2 * hq * d)                   # k, v, q in, the output out
    return {"bytes": nbytes, "flops": 4.0 * hq * d * seen * case["layers"]}


def tolerance(case: dict) -> dict:
    """Four times what the tensor-core kernels differ from the CUDA-core decode kernel and the other prefill kernel over
    these cases (relative 0.9e-3 - 2.7e-3, largest 0.008 - 0.043): a 16-bit output from 16-bit operands and 32-bit sums."""
    return {"rel": 0.01, "max": 0.17}


# ---- state ------------------------------------------------------------------------------------------------------------

class _State:
    pass


def _kv(st, rows: int):
    k = torch.randn(rows, st.h, st.d, device="cuda", dtype=torch.float32, generator=st.gen)
    k[..., st.loud] *= 10.0
    v = torch.randn(rows, st.h, st.d, device="cuda", dtype=torch.float32, generator=st.gen)
    return k.to(st.dtype), v.to(st.dtype)


def _slots(st, seq: np.ndarray, pos: np.ndarray) -> np.ndarray:
    return st.table_np[seq, pos // st.bs].astype(np.int64) * st.bs + pos % st.bs


def _fill(st, seq: np.ndarray, pos: np.ndarray) -> None:
    """Store the tokens (seq, pos) of every layer, a few thousand rows at a time."""
    for at in range(0, seq.size, 32768):
        meta = st.runner.plan_step(_slots(st, seq[at: at + 32768], pos[at: at + 32768]))
        for layer in range(st.layers):
            st.runner.write(layer, *_kv(st, meta.write.n_rows), meta)


def prepare(case: dict, seed: int):
    st = _State()
    st.kind, st.h, st.d, st.bs, st.layers = case["kind"], case["h"], case["d"], case["bs"], case["layers"]
    st.hq, st.scale, st.dtype = case["h"] * case["gqa"], case["d"] ** -0.5, DTYPES[case["dtype"]]
    st.gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    st.loud = torch.from_numpy(rng.permutation(st.d)[: max(1, st.d // 100)]).cuda()
    st.base, st.step, st.phase = _lengths(case)
    n = st.base.size
    layout = TieredLayout(num_kv_heads=st.h, head_size=st.d, block_size=st.bs, mem_bits=case["mem"],
                          k_group=case["kg"], v_group=V_GROUP)
    width = int((st.base + st.step + st.bs - 1).max()) // st.bs + 1
    used = (st.base + st.step + st.bs - 1) // st.bs + 1
    blocks = int(used.sum()) + 8
    page = st.bs * TieredLayout.per_token_bytes(st.h, st.d, case["mem"], case["kg"], V_GROUP)
    st.caches = [torch.zeros(blocks, page, dtype=torch.uint8, device="cuda") for _ in range(st.layers)]
    st.residual = torch.zeros(st.layers, n + 17, case["kg"], st.h, st.d, dtype=st.dtype, device="cuda")
    st.runner = GroupRunner(
        layout, st.caches, st.hq, st.scale, [LayerController(ControllerParams(fixed_bits=b)) for b in _tiers(case)],
        residual_slots=n + 16, model_dtype=st.dtype, canary_max_q=CANARY_ROWS, cap=max(64, n), max_model_len=width * st.bs,
        residuals=list(st.residual))
    perm, at = rng.permutation(blocks).astype(np.int32), 0
    st.table_np = np.zeros((n, width), dtype=np.int32)
    for s in range(n):
        st.table_np[s, : used[s]] = perm[at: at + used[s]]
        at += int(used[s])
    st.table = torch.from_numpy(st.table_np).cuda()
    have = st.base + st.phase  # tokens stored before the first pass
    seq = np.repeat(np.arange(n), have)
    _fill(st, seq, np.arange(seq.size) - np.repeat(np.cumsum(have) - have, have))
    rows = int(st.step.max() if st.kind == "pressure" else st.step.sum())
    kv = [_kv(st, rows) for _ in range(st.layers)]
    st.k, st.v = torch.stack([x[0] for x in kv]), torch.stack([x[1] for x in kv])
    st.q = torch.randn(st.layers, rows, st.hq, st.d, device="cuda", dtype=torch.float32, generator=st.gen).to(st.dtype)
    st.out = torch.zeros_like(st.q)
    st.passes, st.seen = 0, None
    st.canary = torch.zeros(st.layers, 3, device="cuda")
    st.graph = None
    if st.kind == "decode":
        meta = _plan_decode(st)
        _decode_layers(st, meta, False)  # an eager step first: a graph's scratch has to exist when it is captured
        meta = _plan_decode(st)
        torch.cuda.synchronize()
        st.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st.graph):
            _decode_layers(st, meta, True)
        st.graph.replay()
    elif st.kind == "pressure":  # every prompt once: the pool is as full as it gets
        for _ in range(n):
            run(st)
    torch.cuda.synchronize()
    return st


# ---- one step ---------------------------------------------------------------------------------------------------------

def _plan_decode(st):
    n = st.base.size
    pos = st.base + (st.phase + st.passes) % st.bs
    st.passes += 1
    rows = np.arange(n)
    return st.runner.plan_step(_slots(st, rows, pos), decode=(rows, rows, pos + 1), canary=np.resize(rows, CANARY_ROWS))


def _decode_layers(st, meta, capturing: bool) -> None:
    for layer in range(st.layers):
        st.runner.write(layer, st.k[layer], st.v[layer], meta, capturing=capturing, query=st.q[layer])
        st.runner.decode(layer, st.q[layer], st.table, st.out[layer], meta)


def _decode_pass(st) -> dict:
    if st.passes % CANARY_EVERY == 2:  # before the next plan moves the K_ref ring; read one measurement later
        if st.seen is not None:
            st.runner.observe(st.seen, float(st.base.mean()))
        st.seen = st.runner.measure_canary(min(CANARY_ROWS, st.base.size))
        if st.seen is not None:
            st.canary = st.seen
    _plan_decode(st)
    st.graph.replay()
    return {"out": st.out, "residual": st.residual, "canary": st.canary}


def _chunk_pass(st) -> dict:
    """Prompt chunks of every sequence, or (mixed) decode tokens and one chunk, or (pressure) one whole prompt."""
    n = st.base.size
    seqs = np.arange(n)
    pos0 = st.base
    if st.kind == "mixed":
        pos0 = st.base + np.where(st.step == 1, (st.phase + st.passes) % st.bs, 0)
    elif st.kind == "pressure":
        seqs = seqs[[st.passes % n]]
    st.passes += 1
    step, pos0 = st.step[seqs], pos0[seqs]
    ends = np.cumsum(step)
    row_seq = np.repeat(seqs, step)
    row_pos = np.arange(row_seq.size) - np.repeat(ends - step - pos0, step)
    single = (step == 1) if st.kind == "mixed" else np.zeros(seqs.size, dtype=bool)
    decode = None
    if single.any():
        decode = ((ends - 1)[single], seqs[single], (pos0 + 1)[single])
    meta = st.runner.plan_step(_slots(st, row_seq, row_pos), decode=decode)
    prefill = [(int(e - k), int(e), int(p + k), 0) for e, k, p, one in zip(ends, step, pos0, single) if not one]
    req_of = [int(s) for s, one in zip(seqs, single) if not one]
    dense = rows = None
    if max(qe - qs for qs, qe, _, _ in prefill) <= ROW_PATH_MAX_CHUNK:
        rows = build_rows(prefill, req_of, st.table.device)
    else:
        dense = build_dense(prefill, req_of, st.bs, st.table.device)
    t = int(ends[-1])
    for layer in range(st.layers):
        q, out = st.q[layer, :t], st.out[layer, :t]
        st.runner.write(layer, st.k[layer, :t], st.v[layer, :t], meta)
        prefill_attention(st.runner.stores[layer], q, out, prefill, req_of, st.table, st.scale, dense=dense, rows=rows)
        if decode is not None:
            st.runner.decode(layer, q, st.table, out, meta)
    return {"out": st.out[:, :t], "residual": st.residual, "pages": st.caches}


def run(state):
    return _decode_pass(state) if state.kind == "decode" else _chunk_pass(state)
