"""The write step's group passes and the split merge at the sizes where their launches change shape: stored bytes against the
numpy oracle, merged rows against the same rows merged in another shape (bits)."""

import pytest

from test_gpu_kernel_edges import test_groups_completed_across_steps as _groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,kg,bs,rows", [(8, 16, 16, 40), (8, 32, 64, 70), (8, 64, 64, 130), (2, 32, 32, 90), (1, 16, 32, 33)])
@pytest.mark.parametrize("graph_semantics", [False, True])
def test_group_passes_of_few_and_many_groups(h, kg, bs, rows, graph_semantics):
    """Three sequences of ``rows`` tokens a step: 8 to 18 groups, more pieces of work than CTAs in captured steps of wide rows."""
    _groups(h, 128, bs, kg, "bf16", rows, graph_semantics)


@pytest.mark.parametrize("d,gqa", [(64, 3), (128, 4)])
@pytest.mark.parametrize("splits", [3, 8, 40, 100])
def test_a_merge_has_one_order(d, gqa, splits):
    """2 to 400 sequences of two KV heads: eight, four, two and one warp per head, up to 67 splits in use, a dozen sequences with
    none.  A sequence's bits are those it has alone."""
    import numpy as np
    import scenarios as S
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
