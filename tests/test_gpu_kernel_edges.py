"""GPU kernels at the sizes where their tiles, lanes and dispatch rules have edges, against the numpy oracle (stored bytes
exactly), the general path of the same operation (bits), or plain torch in fp32.  Attention tolerances are those of the
other GPU tests: 5e-3 for float32 outputs of 16-bit operands with fp16 arithmetic, 2e-2 / 3e-2 where operands are bf16."""

import ctypes as C

import numpy as np
import pytest

import scenarios as S
from oracle import echokv_oracle as O
from runners import run_oracle
from test_gpu_store import compare_store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,kg,nq,gqa,pad", [(16, 16, 1, 1, 0), (80, 16, 3, 7, 0), (112, 16, 5, 8, 0), (64, 64, 8, 4, 1)])
def test_canary_windows_and_row_counts(w, kg, nq, gqa, pad):
    """Windows past one 64-key pass, row counts that leave warps partly or wholly idle, K_ref rows off 16-byte boundaries."""
    import torch
    from echokv_b200.canary import canary_kl_ring

    rng = np.random.default_rng(w + nq)
    q = torch.from_numpy(rng.standard_normal((2, nq, 2 * gqa, 64), dtype=np.float32)).cuda()
    ring = torch.from_numpy(rng.standard_normal((2, w, 2, 64 + pad), dtype=np.float32) * 2).cuda()[..., :64]
    got = canary_kl_ring(q, ring, 0, w, kg, 0.125).cpu().numpy()
    want = O.canary_kl(q.cpu().numpy(), ring.cpu().numpy(), (2, 4, 8), kg, 0.125)
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("d,gqa", [(64, 3), (128, 3), (128, 8), (256, 2)])
@pytest.mark.parametrize("splits", [1, 8, 9, 33, 64])
def test_merge_over_split_counts(d, gqa, splits):
    """One split, a full batch of loads, one more, more than a warp's worth; query heads that do not fill a CTA;
    16-bit output rows that a lane's channels fit and rows that they do not."""
    import torch
    from test_gpu_decode import _store_and_inputs

    from echokv_b200.kernels.decode import decode_attention

    sc = S.build_attention(f"merge{d}", 1, d, 16, 8, [1050, 33, 16], [4, 8], seed=3, kg=16, dtype="f16", gqa=gqa)
    store, q, table, lens, _ = _store_and_inputs(sc)
    want = run_oracle(sc)["attn_out"]
    got = decode_attention(store, q, table, lens, sc.scale, 1, num_splits=splits)
    assert np.abs(got.cpu().numpy() - want).max() <= 5e-3
    for pad in (8, 1):
        out = torch.zeros(q.shape[0], q.shape[1], d + pad, device="cuda", dtype=torch.float16)[..., :d]
        decode_attention(store, q, table, lens, sc.scale, 1, num_splits=splits, out=out)
        assert torch.equal(out, got.half())


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("h,gqa,kg,plan", [(8, 4, 16, [8]), (2, 8, 32, [4]), (1, 1, 64, [2, 8]), (4, 5, 32, [4, 2])])
def test_decode_of_open_groups(dtype, h, gqa, kg, plan):
    """Keys from the residual buffer in every dtype and tier order, from one token in the group to all but one; lengths so
    uneven that most first work items are empty."""
    sc = S.build_attention(f"open{dtype}{h}", h, 128, 64, 8, [1, 700, kg - 1, 64 + kg + 3, 2 * kg + 17], plan, seed=11, kg=kg, dtype=dtype, gqa=gqa)
    from cuda_runner import run_cuda

    got, want = run_cuda(sc)["attn_out"], run_oracle(sc)["attn_out"]
    assert np.abs(got - want).max() <= 5e-3


@pytest.mark.parametrize("bits", [8, 4, 2])
def test_decode_of_blocks_that_are_no_power_of_two(bits):
    """48-token blocks: a 16-token tile's rows can lie in two chunks, which the tensor-core kernel does not handle."""
    from cuda_runner import run_cuda

    sc = S.build_attention("bs48", 2, 128, 48, 8, [100, 48, 333], [bits], seed=4, kg=48, dtype="f16", gqa=4)
    got, want = run_cuda(sc)["attn_out"], run_oracle(sc)["attn_out"]
    assert np.abs(got - want).max() <= 5e-3


@pytest.mark.parametrize("pad", [0, 2])
def test_dense_attention_of_many_uneven_chunks(pad):
    """More chunks than a warp has lanes, an empty one among them, lengths around the row tiles; output rows on and off 16-byte
    boundaries.  Against torch's fp32 attention, tolerance 2e-2 (bf16)."""
    import torch
    import torch.nn.functional as F
    from echokv_b200.kernels.prefill import dense_attention

    torch.manual_seed(9)
    Hq, H, D = 8, 2, 128
    shapes = [(1 + (i * 37) % 200, (i * 53) % 90) for i in range(36)] + [(0, 40), (64, 0), (65, 128), (256, 1)]
    T, total = sum(n for n, _ in shapes), sum(n + c for n, c in shapes)
    q = torch.randn(T, Hq, D, device="cuda").bfloat16()
    k, v = torch.randn(total, H, D, device="cuda").bfloat16(), torch.randn(total, H, D, device="cuda").bfloat16()
    rows, at_q, at_k = [], 0, 0
    for n, c in shapes:
        rows.append([at_q, at_q + n, n + c, at_k])
        at_q, at_k = at_q + n, at_k + n + c
    out = torch.zeros(T, Hq, D + pad, device="cuda", dtype=torch.bfloat16)[..., :D]
    for query_rows in (T, 0):
        out.zero_()
        dense_attention(q, k, v, torch.tensor(rows, dtype=torch.int32, device="cuda"), max(n for n, _ in shapes), out, D ** -0.5, query_rows)
        for qs, qe, ctx, ks in rows:
            n = qe - qs
            if n == 0:
                continue
            kf = k[ks:ks + ctx].transpose(0, 1).repeat_interleave(Hq // H, 0).float()
            vf = v[ks:ks + ctx].transpose(0, 1).repeat_interleave(Hq // H, 0).float()
            mask = torch.arange(ctx, device="cuda")[None] <= (ctx - n + torch.arange(n, device="cuda"))[:, None]
            want = F.scaled_dot_product_attention(q[qs:qe].transpose(0, 1).float(), kf, vf, attn_mask=mask, scale=D ** -0.5)
            assert (out[qs:qe].float() - want.transpose(0, 1)).abs().max().item() <= 2e-2


@pytest.mark.parametrize("bs,kg", [(128, 64), (256, 64), (512, 64), (1024, 128)])
def test_decode_of_large_blocks(bs, kg):
    """Blocks of up to 256 tokens are what one plan of the tensor-core kernel holds; larger ones take the generic kernel."""
    from cuda_runner import run_cuda
    from echokv_b200.kernels.decode import decode_parallelism

    sc = S.build_attention(f"bs{bs}", 2, 128, bs, 8, [700, bs, 33, 2 * bs + 5], [4, 8], seed=8, kg=kg, dtype="f16", gqa=4)
    got = run_cuda(sc)
    assert (decode_parallelism(got["_store"], 8) > 0) == (bs <= 256)
    assert np.abs(got["attn_out"] - run_oracle(sc)["attn_out"]).max() <= 5e-3


@pytest.mark.parametrize("h,d,bs,kg,dtype,rows", [(1, 128, 64, 64, "bf16", 7), (3, 64, 32, 32, "f16", 5), (8, 128, 16, 16, "bf16", 16),
                                                  (5, 128, 64, 32, "bf16", 41), (2, 128, 48, 48, "f16", 20), (2, 64, 16, 16, "bf16", 600)])
@pytest.mark.parametrize("graph_semantics", [False, True])
def test_groups_completed_across_steps(h, d, bs, kg, dtype, rows, graph_semantics):
    """Groups that complete from residual rows and the step's own, at every group size that has its own kernel and one that
    has not, few groups (many CTAs each) and many (one CTA each)."""
    from cuda_runner import run_cuda

    rng = np.random.default_rng(h * d + kg)
    seqs, total = 3, max(2 * kg + 5, 2 * rows + 3)
    per = -(-total // bs)
    sp = S.StoreSpec(h=h, d=d, bs=bs, mem_bits=8, kg=kg, vg=32, num_blocks=seqs * per + 1, residual_slots=seqs * (rows // kg + 2),
                     dtype=dtype, kref_window=kg)
    perm = rng.permutation(sp.num_blocks)[: seqs * per].reshape(seqs, per)
    steps = []
    for i, at in enumerate(range(0, total, rows)):
        pos = np.arange(at, min(at + rows, total))
        slots = np.concatenate([perm[s][pos // bs] * bs + pos % bs for s in range(seqs)] + [np.array([-1, -1])])
        k = S.round_to(rng.standard_normal((slots.size, h, d), dtype=np.float32) * 3, dtype)
        v = S.round_to(rng.standard_normal((slots.size, h, d), dtype=np.float32), dtype)
        steps.append((k, v, slots, (4, 8, 2)[i % 3]))
    sc = S.Scenario(f"groups{kg}", sp, steps)
    sc.use_kref = True
    compare_store(sc, run_cuda(sc, graph_semantics=graph_semantics), run_oracle(sc))


@pytest.mark.parametrize("h,d,bs,kg", [(8, 64, 16, 16), (8, 64, 32, 32), (2, 64, 16, 16), (4, 128, 64, 64)])
def test_steps_of_more_than_512_rows(h, d, bs, kg):
    """Captured steps launch a group pass per row: above 512 rows the groups of 16 and 32 tokens of long rows take the pass with
    a thread per channel piece, those of short rows and of 64 tokens stay spread over lanes."""
    test_groups_completed_across_steps(h, d, bs, kg, "bf16", 200, True)


@pytest.mark.parametrize("h,d,bs,kg", [(2, 64, 16, 16), (1, 128, 32, 16), (8, 128, 64, 32), (8, 128, 128, 64)])
@pytest.mark.parametrize("bits", [8, 4])
def test_demotion_across_block_shapes(h, d, bs, kg, bits):
    """Blocks demoted to INT2 under pool pressure; the last shape's rows do not fit a CTA's shared memory (three launches)."""
    from cuda_runner import run_cuda

    rng = np.random.default_rng(bs + bits)
    sp = S.StoreSpec(h=h, d=d, bs=bs, mem_bits=4, kg=kg, vg=32, num_blocks=9, residual_slots=4, dtype="bf16")
    order = rng.permutation(9)
    steps = []
    for b in order[:8]:
        k = S.round_to(rng.standard_normal((bs, h, d), dtype=np.float32) * 2, "bf16")
        v = S.round_to(rng.standard_normal((bs, h, d), dtype=np.float32), "bf16")
        steps.append((k, v, b * bs + np.arange(bs), bits if b != order[3] else 8))
    sc = S.Scenario(f"demote{bs}", sp, steps)
    got = run_cuda(sc)
    assert got["demoted"] == (5 if bits == 8 else 1)
    compare_store(sc, got, run_oracle(sc))


@pytest.mark.parametrize("h,d,bs,kg,dtype", [(1, 64, 16, 16, "bf16"), (1, 128, 64, 32, "f16"), (3, 96, 48, 16, "bf16"), (2, 128, 32, 16, "f16")])
def test_dense_dequantization_of_short_rows(h, d, bs, kg, dtype):
    """Rows so short that a CTA has fewer than 256 threads once there are many of them (contexts of 5,000 tokens: 313 CTAs and
    more), and with few CTAs; against the fp32 dequantization rounded to 16 bits, same bits."""
    import torch
    from cuda_runner import run_cuda
    from echokv_b200.kernels.prefill import build_dense, dequant_dense

    for lens in ([5003, 17], [79]):
        sc = S.build_attention("short rows", h, d, bs, 8, lens, [8, 2, 4], seed=6, kg=kg, dtype=dtype, gqa=1, chunks=[1] * len(lens))
        sc.prefill, prefill, sc.query = None, sc.prefill, None
        store = run_cuda(sc)["_store"]
        table = torch.from_numpy(sc.block_table).cuda()
        work, total, _, _ = build_dense(prefill, sc.req_of, bs, "cuda")
        want = dequant_dense(store, work, total, table, torch.float32)
        for dt in (torch.float16, torch.bfloat16):
            for a, b in zip(dequant_dense(store, work, total, table, dt), want):
                assert torch.equal(a, b.to(dt))


def test_headers_of_many_pools_in_one_launch():
    """More pools than one launch takes, empty entries among them."""
    import torch
    from echokv_b200 import _native as N

    n_pools, blocks, page = 40, 6, 64
    pools = torch.zeros(n_pools, blocks, page, dtype=torch.uint8, device="cuda")
    counts = [i % 4 for i in range(n_pools)]
    ids = [torch.randperm(blocks, device="cuda")[:c] for c in counts]
    hdr = [torch.randint(1, 255, (c, 16), dtype=torch.uint8, device="cuda") for c in counts]
    want = pools.clone()
    for i in range(n_pools):
        want[i, ids[i], :16] = hdr[i]
    pages = (N.Pages * n_pools)(*[N.Pages(pools[i].data_ptr(), page, blocks, 0, 0) for i in range(n_pools)])
    ptrs = lambda ts: (C.c_void_p * n_pools)(*[t.data_ptr() for t in ts])
    N.check(N.lib.echokv_write_headers_many(pages, ptrs(ids), ptrs(hdr), (C.c_int64 * n_pools)(*counts), n_pools, N.stream_ptr(pools.device)))
    assert torch.equal(pools, want)
