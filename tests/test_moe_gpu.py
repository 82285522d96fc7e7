"""MoE kernels (router, sort, grouped GEMM, top-k reduce) against torch references on one GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    import triton_distributed_b200 as tdb

    tdb.initialize_distributed(seed=0)
    return tdb.get_runtime()


@pytest.mark.parametrize("cfg", [(37, 8, 2), (512, 128, 8), (1000, 256, 8), (5, 64, 6)])
def test_topk_router(cfg):
    from triton_distributed_b200.ops import topk_router, topk_router_reference

    T, E, k = cfg
    logits = torch.randn(T, E, device="cuda")
    ids, w = topk_router(logits, k, True)
    rids, rw = topk_router_reference(logits, k, True)
    assert torch.equal(ids.sort(-1).values, rids.sort(-1).values)
    torch.testing.assert_close(w.sum(-1), torch.ones(T, device="cuda"), rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(w.gather(1, ids.long().argsort(-1)), rw.gather(1, rids.long().argsort(-1)), rtol=1e-4, atol=1e-5)


def test_align_sort_invariants():
    from triton_distributed_b200.ops import sort_topk_ids_align_block_size

    T, E, k = 777, 32, 4
    ids = torch.randint(0, E + 1, (T, k), device="cuda", dtype=torch.int32)   # E = dropped
    s = sort_topk_ids_align_block_size(ids, E)
    flat = ids.reshape(-1)
    total, tiles = s.meta.tolist()
    assert total % 128 == 0 and tiles == total // 128
    counts = torch.bincount(flat[flat < E].long(), minlength=E)
    assert torch.equal(s.counts.long(), counts)
    sid = s.sorted_ids[:total]
    real = sid[sid >= 0].long()
    assert real.numel() == int((flat < E).sum()) and real.unique().numel() == real.numel()
    te = s.tile_expert[:tiles].long()
    for t in range(tiles):
        rows = sid[t * 128:(t + 1) * 128]
        rows = rows[rows >= 0].long()
        assert (flat[rows] == te[t]).all()
    assert (s.tile_expert[tiles:] == -1).all()
    pos = s.pos_of[:T * k].long()
    ok = flat < E
    assert torch.equal(s.sorted_ids[pos[ok]].long(), torch.nonzero(ok).squeeze(1))
    assert (pos[~ok] == -1).all()


@pytest.mark.parametrize("cfg", [(300, 16, 2, 256, 512), (2048, 32, 8, 1024, 768), (64, 8, 8, 7168, 256)])
def test_moe_mlp_single_rank(rt, cfg):
    from triton_distributed_b200 import ops

    T, E, k, H, I = cfg
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    w1 = (torch.randn(E, 2 * I, H, device="cuda") * 0.03).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, device="cuda") * 0.03).to(torch.bfloat16)
    ids, tw = ops.topk_router(torch.randn(T, E, device="cuda"), k)
    agc = ops.create_ag_group_gemm_context(T, 2 * I, H, E, k)
    rsc = ops.create_moe_rs_context(max_token_num=T, hidden_dim=H, num_experts=E, topk=k)
    # API layout: (token, slot) order
    h = ops.ag_group_gemm(x, w1, agc, ids)
    ref_h = ops.group_gemm_reference(x, w1, ids)
    torch.testing.assert_close(h.float(), ref_h.float(), rtol=3e-2, atol=3e-2)
    act = ops.silu_mul(h)
    out = ops.run_moe_reduce_rs(act, w2, ids, tw, rsc)
    ref = ops.moe_reduce_reference(act, w2, ids, tw)
    torch.testing.assert_close(out.float(), ref.float(), rtol=3e-2, atol=3e-2)
    # fused layout: stay expert-sorted between the two grouped GEMMs
    hs, srt = ops.ag_group_gemm(x, w1, agc, ids, sorted_output=True)
    out2 = ops.run_moe_reduce_rs(ops.silu_mul(hs), w2, ids, tw, rsc, sort=srt)
    torch.testing.assert_close(out2.float(), ref.float(), rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("cfg", [(512, 16, 4, 4, 1), (1024, 64, 8, 8, 3), (96, 8, 2, 2, 0)])
def test_staged_sort_and_device_tile_schedule(rt, cfg):
    """The staged sort keeps every expert's rows together, ordered by ring distance; the device-side tile schedule
    equals the host C++ reference on the same layout."""
    from triton_distributed_b200 import ops

    T, E, k, W, rank = cfg
    ids, _ = ops.topk_router(torch.randn(T, E, device="cuda"), k)
    tpr = T // W
    srt = ops.sort_topk_ids_staged(ids, E, tpr, rank, W)
    flat = ids.reshape(-1).long()
    sid = srt.sorted_ids.long()
    offs = srt.offsets.long().tolist()
    cnt = srt.counts.long().tolist()
    assert sorted(sid[sid >= 0].tolist()) == list(range(T * k))
    for e in range(E):
        rows = sid[offs[e]:offs[e] + cnt[e]]
        assert (flat[rows] == e).all() and (sid[offs[e] + cnt[e]:offs[e + 1]] == -1).all()
        stage = ((rows // k) // tpr - rank) % W
        assert (stage[1:] >= stage[:-1]).all(), "rows of an expert must be ordered by arrival stage"
    assert torch.equal(srt.sorted_ids[srt.pos_of.long()].long(), torch.arange(T * k, device="cuda"))
    order, stage = ops.tile_schedule(srt, tpr, rank, W)
    ref_order, ref_stage = ops.tile_arrival_order(srt, tpr, rank, W)
    assert torch.equal(stage.cpu(), ref_stage) and torch.equal(order.cpu(), ref_order)


@pytest.mark.parametrize("cfg", [(300, 16, 2, 256, 512), (1024, 8, 4, 7168, 256), (77, 4, 1, 64, 136)])
def test_group_gemm_with_in_kernel_gather(rt, cfg):
    from triton_distributed_b200 import ops

    T, E, k, H, N = cfg
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(E, N, H, device="cuda") * 0.03).to(torch.bfloat16)
    ids, tw = ops.topk_router(torch.randn(T, E, device="cuda"), k)
    srt = ops.sort_topk_ids_align_block_size(ids, E)
    ref = ops.group_gemm_reference(x, w, ids).float()                       # (token, slot) order
    y = ops.group_gemm_gather(x, w, srt, a_row_div=k, scatter_out=True)
    torch.testing.assert_close(y.float(), ref, rtol=3e-2, atol=3e-2)
    ys = ops.group_gemm_gather(x, w, srt, a_row_div=k, scatter_out=False, row_weight=tw)
    sid = srt.sorted_ids.long()
    ok = sid >= 0
    torch.testing.assert_close(ys[ok].float(), ref[sid[ok]] * tw.reshape(-1)[sid[ok]].unsqueeze(-1), rtol=3e-2, atol=3e-2)
    assert (ys[: int(srt.meta[0])][~ok[: int(srt.meta[0])]] == 0).all()     # padding rows of visited tiles are zeros


@pytest.mark.parametrize("n,E", [(0, 8), (1, 1), (8191, 128), (8193, 2048), (65536, 7), (65537, 128), (100, 2049)])
def test_sort_sizes(n, E):
    # both sides of the one-launch sort's limits; ids outside [0, E) are dropped, most experts of a large E are empty
    from triton_distributed_b200.ops import sort_topk_ids_align_block_size

    g = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(-1, E + 1, (n, 1), device="cuda", dtype=torch.int32, generator=g)
    s = sort_topk_ids_align_block_size(ids, E)
    flat = ids.reshape(-1).long()
    ok = (flat >= 0) & (flat < E)
    counts = torch.bincount(flat[ok], minlength=E)
    ends = ((counts + 127) // 128 * 128).cumsum(0)
    assert torch.equal(s.counts.long(), counts) and torch.equal(s.offsets[1:].long(), ends) and s.offsets[0] == 0
    assert s.meta.tolist() == [int(ends[-1]), int(ends[-1]) // 128]
    want = torch.repeat_interleave(torch.arange(E, device="cuda"), (counts + 127) // 128)
    assert torch.equal(s.tile_expert[:want.numel()].long(), want) and (s.tile_expert[want.numel():] == -1).all()
    pos = s.pos_of[:n].long()
    assert (pos[~ok] == -1).all() and torch.equal(s.sorted_ids[pos[ok]].long(), ok.nonzero().squeeze(1))
    assert ((pos[ok] >= s.offsets[flat[ok]]) & (pos[ok] < s.offsets[flat[ok]] + counts[flat[ok]])).all()
    assert int((s.sorted_ids >= 0).sum()) == int(ok.sum())


@pytest.mark.parametrize("T,E,k,H,I", [(1, 4, 2, 64, 16), (130, 5, 3, 200, 136), (700, 8, 4, 256, 248), (257, 3, 1, 72, 384)])
def test_gated_group_gemm_and_sorted_rows(rt, T, E, k, H, I):
    # SwiGLU in the epilogue, then rows that are in sorted order already; widths that end inside a tile's halves
    from triton_distributed_b200 import ops

    torch.manual_seed(T)
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    w13 = (torch.randn(E, 2 * I, H, device="cuda") * H ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, device="cuda") * I ** -0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device="cuda")[:k] for _ in range(T)]).to(torch.int32)
    rw = torch.rand(T, k, device="cuda")
    srt = ops.sort_topk_ids_align_block_size(ids, E)
    act = ops.group_gemm_gather(x, w13, srt, a_row_div=k, gated=True)
    flat = ops.group_gemm_gather(x, w13, srt, a_row_div=k, gated=True, scatter_out=True)
    y = ops.group_gemm_gather(act, w2, srt, a_row_div=0, row_weight=rw)
    torch.cuda.synchronize()
    pairs = ids.reshape(-1).long()
    g, u = torch.einsum("pk,pnk->pn", x.double().repeat_interleave(k, 0), w13.double()[pairs]).chunk(2, -1)
    ref = torch.nn.functional.silu(g) * u
    pos = srt.pos_of.long()
    # one rounding to bf16 of values of order one, and fp32 sums
    torch.testing.assert_close(act[pos].double(), ref, rtol=2 ** -8, atol=2 ** -10)
    torch.testing.assert_close(flat.double(), ref, rtol=2 ** -8, atol=2 ** -10)
    ref2 = torch.einsum("pk,pnk->pn", act[pos].double(), w2.double()[pairs]) * rw.reshape(-1, 1).double()
    torch.testing.assert_close(y[pos].double(), ref2, rtol=2 ** -8, atol=2 ** -10)
    pad = srt.sorted_ids[:int(srt.meta[0])] < 0
    assert act[:pad.numel()][pad].abs().max() == 0 if pad.any() else True


@pytest.mark.parametrize("N,gated", [(320, False), (384, False), (448, False), (264, False), (384, True), (400, True)])
def test_group_gemm_partial_column_tiles(rt, N, gated):
    # widths that leave chunks of a tile's output without a store, several tiles per CTA and few products between the stores: a staging
    # buffer must not be written again before its store has read it
    from triton_distributed_b200 import ops

    torch.manual_seed(N)
    T, E, k, K = 148 * 128 * 2 + 5, 4, 2, 64
    w = (torch.randn(E, N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    for _ in range(3):
        x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
        ids = torch.rand(T, E, device="cuda").topk(k).indices.to(torch.int32)
        srt = ops.sort_topk_ids_align_block_size(ids, E)
        y = ops.group_gemm_gather(x, w, srt, a_row_div=k, gated=gated)[srt.pos_of.long()].double()
        torch.cuda.synchronize()
        pairs, rows = ids.reshape(-1), x.repeat_interleave(k, 0)
        for e in range(E):
            at = pairs == e
            ref = rows[at].double() @ w[e].double().t()
            if gated:
                g, u = ref.chunk(2, -1)
                ref = torch.nn.functional.silu(g) * u
            # one rounding to bf16 of values of order one, and fp32 sums
            torch.testing.assert_close(y[at], ref, rtol=2 ** -8, atol=2 ** -10)


@pytest.mark.parametrize("T,E,k,H,I", [(5, 4, 2, 64, 16), (300, 6, 3, 320, 136)])
def test_sorted_rows_that_end_behind_the_last_in_use(rt, T, E, k, H, I):
    # the sorted layout has room for the worst case; x may hold the padded rows in use only
    from triton_distributed_b200 import ops

    torch.manual_seed(T)
    w2 = (torch.randn(E, H, I, device="cuda") * I ** -0.5).to(torch.bfloat16)
    ids = torch.rand(T, E, device="cuda").topk(k).indices.to(torch.int32)
    rw = torch.rand(T, k, device="cuda")
    srt = ops.sort_topk_ids_align_block_size(ids, E)
    used = int(srt.meta[0])
    assert used < srt.sorted_ids.numel()
    x = torch.randn(srt.sorted_ids.numel(), I, device="cuda", dtype=torch.bfloat16)
    ctx = ops.create_moe_ar_context(max_token_num=T, hidden_dim=H, num_experts=E, topk=k)
    whole, part = (ops.group_gemm_gather(t, w2, srt, a_row_div=0, row_weight=rw)[srt.pos_of.long()] for t in (x, x[:used].clone()))
    whole_r, part_r = (ops.run_moe_reduce_ar(t, w2, ids, rw, ctx, sort=srt) for t in (x, x[:used].clone()))
    torch.cuda.synchronize()
    assert torch.equal(whole, part) and torch.equal(whole_r, part_r)


def test_padding_rows_are_zeros_whatever_lies_in_x(rt):
    from triton_distributed_b200 import ops

    torch.manual_seed(1)
    T, E, k, I = 200, 5, 2, 96
    ids = torch.rand(T, E, device="cuda").topk(k).indices.to(torch.int32)
    srt = ops.sort_topk_ids_align_block_size(ids, E)
    pad, used = srt.sorted_ids < 0, int(srt.meta[0])
    x = torch.randn(pad.numel(), I, device="cuda", dtype=torch.bfloat16)
    x[pad] = float("nan")
    for N, gated in ((320, False), (400, True)):
        w = (torch.randn(E, N, I, device="cuda") * I ** -0.5).to(torch.bfloat16)
        y = ops.group_gemm_gather(x, w, srt, a_row_div=0, gated=gated)
        torch.cuda.synchronize()
        assert (y[:used][pad[:used]] == 0).all() and torch.isfinite(y[srt.pos_of.long()]).all()


@pytest.mark.parametrize("E", [1, 31, 128, 129, 512])
def test_router_bf16_logits(E):
    from triton_distributed_b200.ops import topk_router

    logits = torch.randn(77, E, device="cuda").to(torch.bfloat16)
    k = min(E, 6)
    a, b = topk_router(logits, k), topk_router(logits.float(), k)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    p = torch.softmax(logits.double(), -1).gather(1, a[0].long())
    torch.testing.assert_close(a[1].double(), p / p.sum(-1, keepdim=True), rtol=1e-5, atol=1e-7)
