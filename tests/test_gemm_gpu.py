"""tcgen05 GEMM against an fp32 torch reference (single GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(M, N, K, block_n=0, seed=0):
    from triton_distributed_b200.ops import gemm

    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16, generator=g)
    b = (torch.randn(N, K, device="cuda", dtype=torch.float32, generator=g) * 0.05).to(torch.bfloat16)
    out = gemm(a, b, block_n=block_n)
    ref = a.float() @ b.float().t()
    torch.cuda.synchronize()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err / scale < 2e-2, f"M={M} N={N} K={K} block_n={block_n}: max err {err} (scale {scale})"
    # element-wise: the only error a correct kernel makes is the bf16 rounding of the output (2^-9 relative); one
    # dropped or doubled 64-wide k-block moves an element by about 0.05 * 8 = 0.4, far outside this band
    torch.testing.assert_close(out.float(), ref, rtol=1e-2, atol=2e-2)


@pytest.mark.parametrize("shape", [(128, 256, 64), (128, 256, 256), (256, 512, 1024), (1024, 1024, 2048)])
def test_gemm_aligned(shape):
    _check(*shape)


@pytest.mark.parametrize("shape", [(100, 200, 72), (4091, 264, 520), (1, 5120, 3200), (257, 136, 8)])
def test_gemm_ragged(shape):
    _check(*shape)


@pytest.mark.parametrize("block_n", [128, 256])
def test_gemm_block_n(block_n):
    _check(512, 768, 512, block_n=block_n)


@pytest.mark.parametrize("shape", [(256, 256, 64), (512, 768, 512), (384, 512, 256), (1000, 520, 264),
                                   (4096, 4096, 512), (8192, 2048, 1024)])
def test_gemm_cta_pair(shape):
    # 256 x 256 tiles over two SMs (cta_group::2); 384 and 1000 rows leave the second CTA of a pair without rows
    _check(*shape, block_n=512)


def test_gemm_large_k():
    # the benchmark's K: 128 k-blocks per tile, the smem ring wraps 21 times per tile
    _check(512, 512, 8192, block_n=512)
    _check(256, 384, 8192)


@pytest.mark.parametrize("shape", [(2048, 2560, 512),    # 80 pair tiles on 74 pairs: 6 tail tiles run as 12 halves
                                   (2048, 2460, 256),    # last tile column is 156 wide: second half has 28 columns
                                   (2048, 2360, 256),    # last tile column is 56 wide: its second half is empty
                                   (2304, 2560, 320)])   # 90 tiles: 16 tail tiles as 32 halves
def test_gemm_cta_pair_split_tail(shape):
    _check(*shape, block_n=512)


def test_gemm_stall_counters():
    from triton_distributed_b200.ops import STALL_COUNTERS, gemm, new_stall_counters, summarize_stall_counters

    a = torch.randn(2048, 1024, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(2560, 1024, device="cuda") * 0.05).to(torch.bfloat16)
    st = new_stall_counters(a.device)
    out = gemm(a, b, block_n=512, stats=st)
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), a.float() @ b.float().t(), rtol=1e-2, atol=2e-2)
    summ = summarize_stall_counters(st)
    assert summ["ctas"] == 148 and summ["cta_total_cycles_max"] > 0
    assert all(0.0 <= summ[f"{n}_mean_frac"] <= 1.0 for n in STALL_COUNTERS[:-1])


def test_gemm_many_tiles_per_cta():
    # more tiles than CTAs: exercises the smem ring and both TMEM accumulator buffers across tiles
    _check(4096, 4096, 512)


def test_gemm_strided_views():
    from triton_distributed_b200.ops import gemm

    a_full = torch.randn(300, 1024, device="cuda", dtype=torch.bfloat16)
    b_full = (torch.randn(400, 1024, device="cuda") * 0.05).to(torch.bfloat16)
    a, b = a_full[:, :512], b_full[:, 512:]
    out = gemm(a, b)
    ref = a.float() @ b.float().t()
    assert (out.float() - ref).abs().max().item() / ref.abs().max().item() < 2e-2


@pytest.mark.parametrize("shape", [(1, 5120, 3200), (8, 1280, 5120), (32, 6400, 5120), (128, 5120, 3200), (200, 520, 264),
                                   (16, 18992, 5120), (3, 136, 64)])
def test_skinny_gemm_split_k(shape):
    from triton_distributed_b200.ops import skinny_gemm

    M, N, K = shape
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ref = a.float() @ b.float().t()
    for splits in (0, 1, 3):
        for _ in range(2):   # twice: the kernel must leave its scratch clean
            out = skinny_gemm(a, b, splits=splits)
        torch.cuda.synchronize()
        err = (out.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
        assert err < 2e-2, f"skinny {shape} splits={splits}: rel err {err}"


def test_skinny_gemm_stream_k_scratch_covers_the_token_pad():
    """65 tokens are padded to 128 in the column-major accumulation buffer of the stream-K form: the scratch must be
    sized by the pad (150 column tiles here, so the cluster form does not apply and every tile is split)."""
    from triton_distributed_b200.ops import gemm_ar, skinny_gemm

    M, N, K = 65, 19200, 1024
    assert gemm_ar.split_scratch_elems(M, N) == 19200 * 128
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ref = a.float() @ b.float().t()
    for splits in (0, 3):
        for _ in range(2):
            out = skinny_gemm(a, b, splits=splits)
        torch.cuda.synchronize()
        err = (out.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
        assert err < 2e-2, f"splits={splits}: rel err {err}"


@pytest.mark.parametrize("shape,cluster", [
    ((16, 2560, 5120), (1, 6)), ((16, 2560, 5120), (2, 8)), ((16, 2560, 5120), (3, 4)), ((16, 2560, 5120), (4, 3)),
    ((128, 5120, 2048), (1, 3)), ((128, 5120, 2048), (2, 5)), ((128, 5120, 2048), (3, 2)),
    ((64, 520, 264), (1, 1)), ((64, 520, 264), (2, 2)), ((33, 520, 264), (3, 1)), ((200, 1280, 1024), (1, 4)),
])
def test_skinny_gemm_cluster_forms(shape, cluster):
    """Every tile width / cluster size of the cluster form against the fp32 reference (column edge: N = 520)."""
    from triton_distributed_b200.ops import skinny_gemm

    M, N, K = shape
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ref = a.float() @ b.float().t()
    try:
        out = skinny_gemm(a, b, cluster=cluster)
    except RuntimeError as e:
        pytest.skip(f"cluster form {cluster} cannot run here: {e}")
    out = skinny_gemm(a, b, cluster=cluster)
    torch.cuda.synchronize()
    err = (out.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
    assert err < 2e-2, f"cluster form {cluster} on {shape}: rel err {err}"


@pytest.mark.parametrize("M", [1, 2, 3, 4, 8, 12, 16])
@pytest.mark.parametrize("mode", ["plain", "norm", "silu", "norm_residual"])
def test_gemv_fused(M, mode):
    # decode GEMV with fused RMSNorm / SiLU*up prologue and residual epilogue against the fp32 reference
    from triton_distributed_b200 import ops

    torch.manual_seed(M)
    for (N, K) in [(1280, 5120), (5120, 1024), (6400, 5120), (5120, 3200), (136, 64), (1003, 264)]:
        w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
        kw = {}
        if mode == "silu":
            x = torch.randn(M, 2 * K, device="cuda", dtype=torch.bfloat16)
            kw["silu_mul"] = True
        else:
            x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
        if mode.startswith("norm"):
            kw["norm_weight"] = (1.0 + 0.1 * torch.randn(K, device="cuda")).to(torch.bfloat16)
            kw["eps"] = 1e-6
        res = None
        if mode == "norm_residual":
            res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
        ref = ops.gemv_reference(x, w, residual=res, **kw).float()
        out = ops.gemv_fused(x, w, residual=res, **kw)
        torch.cuda.synchronize()
        err = (out.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
        assert err < 2e-2, f"gemv {mode} M={M} N={N} K={K}: rel err {err}"
        if res is not None:
            # in place: out aliases the residual
            buf = res.clone()
            ops.gemv_fused(x, w, out=buf, residual=buf, **kw)
            torch.cuda.synchronize()
            err = (buf.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
            assert err < 2e-2, f"gemv in-place {mode} M={M} N={N} K={K}: rel err {err}"


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (2, 1, 40), (1, 149, 264), (3, 4096, 1000), (5, 1185, 2056), (1, 20011, 520), (8, 151, 8192),
                                   (16, 4099, 6112), (1, 300, 98272)])
def test_gemv_spans(M, N, K):
    # warps' spans that begin and end inside a group, groups with fewer rows, idle warps, every depth of the weight ring
    from triton_distributed_b200 import ops

    torch.manual_seed(N)
    assert ops.gemv_supported(M, K)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    ref = x.double() @ w.double().t()
    out = ops.gemv_fused(x, w).double()
    torch.cuda.synchronize()
    # one rounding to bf16 (2^-9 of the value) and fp32 sums of K products of order one over sqrt(K)
    assert ((out - ref).abs() <= ref.abs() * 2 ** -8 + 2 ** -20 * K ** 0.5 + 1e-5).all()


@pytest.mark.parametrize("M", [1, 3, 8, 16])
def test_gemv_empty_sums(M):
    # no input features: the residual alone, or zeros, whatever the prologue; no output features: nothing to do
    from triton_distributed_b200 import ops

    x = torch.randn(M, 64, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(304, 64, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, 304, device="cuda", dtype=torch.bfloat16)
    none = torch.ones(0, device="cuda", dtype=torch.bfloat16)
    for kw, want in ((dict(), torch.zeros_like(res)), (dict(residual=res), res), (dict(norm_weight=none), torch.zeros_like(res)),
                     (dict(silu_mul=True, residual=res), res), (dict(swiglu=True), torch.zeros_like(res[:, :152]))):
        out = ops.gemv_fused(x[:, :0], w[:, :0], out=torch.full_like(want, 7.0), **kw)
        torch.cuda.synchronize()
        assert torch.equal(out, want), kw
        assert ops.gemv_fused(x, w[:0], **{k: v for k, v in kw.items() if k == "swiglu"}).shape == (M, 0)


@pytest.mark.parametrize("M,F,K", [(256, 256, 64), (257, 264, 200), (777, 520, 1024), (1024, 19 * 128, 128), (300, 5000, 72), (8, 384, 512)])
def test_gemm_swiglu(M, F, K):
    # gate and up columns that end inside a tile's halves, half-width tail tiles, rows that end inside a CTA's 128; few rows: two launches
    from triton_distributed_b200 import ops

    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    g, u = (x.double() @ w.double().t()).chunk(2, dim=-1)
    ref = torch.nn.functional.silu(g) * u
    out = ops.gemm_swiglu(x, w)
    torch.cuda.synchronize()
    # one rounding to bf16 of values of order one behind fp32 sums; three roundings where gate and up are stored
    torch.testing.assert_close(out.double(), ref, rtol=2 ** -8 if M >= 256 else 2 ** -6, atol=2 ** -10 if M >= 256 else 2 ** -8)


@pytest.mark.parametrize("form", ["pair", "gated", "single"])
@pytest.mark.parametrize("M,N", [(256 * 148 + 9, 320), (256 * 148 + 9, 528), (256 * 148 + 137, 768), (128 * 444, 392)])
def test_gemm_chunks_without_a_store(M, N, form):
    # columns and rows that leave chunks of a tile without a store, several tiles per CTA and few products between the stores: a staging
    # buffer must not be written again before its store has read it
    from triton_distributed_b200 import ops

    torch.manual_seed(N)
    K = 64
    if form == "gated":
        N *= 2
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    for _ in range(3):
        x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
        out = ops.gemm_swiglu(x, w) if form == "gated" else ops.gemm(x, w, block_n=512 if form == "pair" else 256)
        ref = x.double() @ w.double().t()
        if form == "gated":
            g, u = ref.chunk(2, dim=-1)
            ref = torch.nn.functional.silu(g) * u
        # one rounding to bf16 of values of order one behind fp32 sums
        torch.testing.assert_close(out.double(), ref, rtol=2 ** -8, atol=2 ** -10)


@pytest.mark.parametrize("M,F,K", [(9, 256, 128), (128, 264, 200), (129, 256, 64), (200, 520, 72), (255, 256, 512), (256, 128, 64), (300, 252, 64)])
def test_gemm_swiglu_two_launches(M, F, K):
    # rows and widths on this side of the pair kernel's: every GEMM below it, then the activation
    from triton_distributed_b200 import ops

    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    g, u = (x.double() @ w.double().t()).chunk(2, dim=-1)
    out = ops.gemm_swiglu(x, w)
    torch.cuda.synchronize()
    # gate, up and result are rounded to bf16
    torch.testing.assert_close(out.double(), torch.nn.functional.silu(g) * u, rtol=2 ** -6, atol=2 ** -8)


@pytest.mark.parametrize("form", ["pair", "gemv", "grouped"])
def test_swiglu_gate_range(form):
    # SiLU in the epilogues for gates from -100 to 40, down to the smallest results
    from triton_distributed_b200 import ops

    z = torch.cat([torch.linspace(-100, -80, 121), torch.linspace(-80, 40, 391)]).to("cuda", torch.bfloat16)
    M, F, K = (16, 32, 8) if form == "gemv" else (512, 256, 8) if form == "pair" else (512, 64, 8)
    out = []
    for rows in z.split(M):
        x = torch.zeros(rows.numel(), K, device="cuda", dtype=torch.bfloat16)
        x[:, 0], x[:, 1] = rows, 1
        w = torch.zeros(2 * F, K, device="cuda", dtype=torch.bfloat16)
        w[:F, 0], w[F:, 1] = 1, 1.5
        if form == "gemv":
            y = ops.gemv_fused(x, w, swiglu=True)
        elif form == "pair":
            y = ops.gemm_swiglu(x, w)
        else:
            srt = ops.sort_topk_ids_align_block_size(torch.zeros(rows.numel(), 1, device="cuda", dtype=torch.int32), 1)
            y = ops.group_gemm_gather(x, w.unsqueeze(0), srt, a_row_div=1, scatter_out=True, gated=True)
        out.append(y)
    torch.cuda.synchronize()
    y = torch.cat(out).double()
    ref = (torch.nn.functional.silu(z.double()) * 1.5).unsqueeze(1).expand_as(y)
    # one rounding to bf16; below the smallest normal number of bf16 results may be flushed
    torch.testing.assert_close(y, ref, rtol=2 ** -8, atol=1.2e-38)


@pytest.mark.parametrize("M,F,K", [(1, 4, 8), (1, 3, 264), (2, 1001, 520), (4, 12288, 256), (7, 149, 2048), (16, 300, 4096), (1, 70, 40000)])
def test_gemv_swiglu(M, F, K):
    # groups of four gate and four up rows: whole, shared by warps, partly empty
    from triton_distributed_b200 import ops

    torch.manual_seed(F)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    nw = (1.0 + 0.1 * torch.randn(K, device="cuda")).to(torch.bfloat16)
    for norm in (None, nw):
        xn = x.double()
        if norm is not None:
            xn = xn * torch.rsqrt(xn.pow(2).mean(-1, keepdim=True) + 1e-6) * norm.double()
        g, u = (xn @ w.double().t()).chunk(2, dim=-1)
        ref = torch.nn.functional.silu(g) * u
        out = ops.gemv_fused(x, w, norm_weight=norm, eps=1e-6, swiglu=True)
        torch.cuda.synchronize()
        # one rounding to bf16 of values of order one behind fp32 sums; the normed activations are rounded to bf16 before them
        torch.testing.assert_close(out.double(), ref, rtol=2 ** -8 if norm is None else 2 ** -6, atol=2 ** -10 if norm is None else 2 ** -6)
