"""The write step's group passes and the split merge at the sizes where their launches change shape: stored bytes against the
numpy oracle, merged rows against the same rows merged in another shape (bits)."""

import re
from pathlib import Path

import numpy as np
import pytest

import scenarios as S
from runners import run_oracle
from test_gpu_kernel_edges import test_groups_completed_across_steps as _groups
from test_gpu_store import compare_store

pytestmark = pytest.mark.gpu
WRITE_CU = Path(__file__).resolve().parent.parent / "echokv_b200" / "csrc" / "write.cu"


@pytest.mark.parametrize("h,kg,bs,rows", [(8, 16, 16, 40), (8, 32, 64, 70), (8, 64, 64, 130), (2, 32, 32, 90), (1, 16, 32, 33)])
@pytest.mark.parametrize("graph_semantics", [False, True])
def test_group_passes_of_few_and_many_groups(h, kg, bs, rows, graph_semantics):
    """Three sequences of ``rows`` tokens a step: 6 to 9 groups, from residual rows and the step's own, each in its finest pieces."""
    _groups(h, 128, bs, kg, "bf16", rows, graph_semantics)


def _group_pass(h, d, kg, rows, n_launch, count):
    """Of a write step's group pass by its launch rule: CTAs launched for groups, pieces of work, workers."""
    chip = int(re.search(r"STEP_GROUP_CTAS = (\d+)", WRITE_CU.read_text()).group(1))
    lanes = 4 if kg == 16 else 8
    need, fine = (-(-(h * d // 8) // (128 // (lanes * f))) for f in (1, 2))
    ctas = min(n_launch * fine, max(chip - rows, chip // 2))
    if count * fine <= ctas:
        return ctas, count * fine, ctas
    return ctas, count * need, ctas if count * need <= ctas else max(ctas, min(ctas + rows, chip))


@pytest.mark.parametrize("h,d,bs,kg,seqs,tokens,joined,run", [
    (8, 128, 16, 16, 100, 1, False, 1),   # a piece per CTA, some CTAs without
    (8, 128, 32, 16, 250, 2, True, 2),    # half a group per worker; every slot given up is taken over in the step
    (8, 128, 64, 32, 170, 1, True, 3),    # runs that begin and end inside groups
    (8, 128, 128, 64, 90, 2, True, 2),
    (3, 128, 16, 16, 300, 1, True, 2),    # a group's last piece is half empty
    (2, 64, 32, 16, 500, 2, True, 1),     # a group is one piece: fewer pieces than workers
    (3, 128, 32, 16, 1000, 1, True, 4),   # runs over two and three groups
])
@pytest.mark.parametrize("graph_semantics", [False, True])
def test_groups_completed_in_lock_step(h, d, bs, kg, seqs, tokens, joined, run, graph_semantics):
    """Sequences in lock step complete their groups in one step, in more pieces of work than CTAs were launched for groups."""
    from cuda_runner import run_cuda
    from echokv_b200.write_plan import WritePlanner

    rng = np.random.default_rng(h * seqs + kg)
    per = -(-(kg + tokens) // bs)
    sp = S.StoreSpec(h=h, d=d, bs=bs, mem_bits=8, kg=kg, vg=32, num_blocks=seqs * per + 1, residual_slots=seqs, dtype="bf16", kref_window=kg)
    perm = rng.permutation(sp.num_blocks)[: seqs * per].reshape(seqs, per)
    steps = []
    for first, last, bits in ((0, kg - 1, 4), (kg - 1, kg - 1 + tokens, 8)):
        pos = np.arange(first, last)
        slots = np.concatenate([perm[:, p // bs] * bs + p % bs for p in pos] + [np.array([-1, -1])])
        k = S.round_to(rng.standard_normal((slots.size, h, d), dtype=np.float32) * 3, "bf16")
        v = S.round_to(rng.standard_normal((slots.size, h, d), dtype=np.float32), "bf16")
        steps.append((k, v, slots, bits))
    planner = WritePlanner(bs, kg, seqs)
    plan = [planner.plan(st[2]) for st in steps][1]
    rows = steps[1][2].size
    assert plan.n_fin == seqs
    if tokens > 1:
        assert np.isin(plan.tok_res[plan.tok_res >= 0], plan.fin[:, 2]).all(), "no slot is taken over in the step"
    ctas, pieces, workers = _group_pass(h, d, kg, rows, rows if graph_semantics else seqs, seqs)
    assert (workers > ctas) == joined and -(-pieces // workers) == run
    sc = S.Scenario("lock step", sp, steps)
    sc.use_kref = True
    compare_store(sc, run_cuda(sc, graph_semantics=graph_semantics), run_oracle(sc))


@pytest.mark.parametrize("d,gqa", [(64, 3), (128, 4)])
@pytest.mark.parametrize("splits", [3, 8, 40, 100])
def test_a_merge_has_one_order(d, gqa, splits):
    """2 to 400 sequences of two KV heads: eight, four, two and one warp per head, up to 67 splits in use, a dozen sequences with
    none.  A sequence's bits are those it has alone."""
    import torch
    from test_gpu_decode import _store_and_inputs

    from echokv_b200.kernels.decode import decode_attention

    sc = S.build_attention(f"merge_order{d}", 2, d, 16, 8, [1061, 470, 33, 16], [4, 8], seed=5, kg=16, dtype="f16", gqa=gqa)
    store, q, table, lens, _ = _store_and_inputs(sc)
    want = decode_attention(store, q, table, lens, sc.scale, 1, num_splits=splits)
    for n in (8, 60, 150, 400):
        of = torch.arange(n, device="cuda") % 4
        ln = lens[of].clone()
        ln[4:: max(4, n // 12)] = 0  # rows of padding
        out = torch.full((n, q.shape[1], d), 7.0, device="cuda")
        decode_attention(store, q[of].contiguous(), table, ln, sc.scale, 1, bt_rows=of, num_splits=splits, out=out)
        live = (ln > 0).cpu().numpy()
        assert torch.equal(out[torch.from_numpy(live).cuda()], want[of[torch.from_numpy(live).cuda()]])
        assert bool((out[torch.from_numpy(~live).cuda()] == 7.0).all()) and np.isfinite(out.cpu().numpy()).all()
