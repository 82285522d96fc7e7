"""Attention kernels against the fp32 torch reference (single GPU)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _paged_cache(B, max_len, Hkv, D, page, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pages_per_seq = (max_len + page - 1) // page
    n_pages = B * pages_per_seq
    k = torch.randn(n_pages, page, Hkv, D, device="cuda", dtype=torch.bfloat16, generator=g)
    v = torch.randn(n_pages, page, Hkv, D, device="cuda", dtype=torch.bfloat16, generator=g)
    perm = torch.randperm(n_pages, device="cuda", generator=g).to(torch.int32)
    bt = perm.reshape(B, pages_per_seq).contiguous()
    return k, v, bt


@pytest.mark.parametrize("cfg", [(4, 8, 1, 128, 1, [1, 63, 64, 700]), (2, 32, 8, 128, 16, [4096, 1000]),
                                 (3, 16, 4, 64, 64, [129, 5, 2048]), (1, 40, 2, 128, 256, [3000])])
def test_decode_split_kv(cfg):
    from triton_distributed_b200.ops import attention_reference, gqa_fwd_batch_decode

    B, Hq, Hkv, D, page, lens = cfg
    k, v, bt = _paged_cache(B, max(lens), Hkv, D, page)
    q = torch.randn(B, Hq, D, device="cuda", dtype=torch.bfloat16)
    kv_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    ref, ref_lse = attention_reference(q, k, v, bt, cu, kv_lens, None, False, None, 0.0, True)
    for splits in (-1, 1, 3):
        out, lse = gqa_fwd_batch_decode(q, k, v, None, None, kv_lens, bt, kv_split=splits, return_lse=True)
        torch.cuda.synchronize()
        torch.testing.assert_close(out.float(), ref.float(), rtol=2e-2, atol=2e-2)
        torch.testing.assert_close(lse, ref_lse.t().contiguous(), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("D,group,page", [(64, 1, 1), (64, 16, 0), (128, 17, 24), (128, 3, 64), (256, 5, 0), (256, 2, 16)])
@pytest.mark.parametrize("splits", [-1, 1, 5, 32])
def test_decode_token_edges(D, group, page, splits):
    # a warp's 16 tokens, a block's 64, pages that end inside both, sequences without a token; one page per sequence (page 0) and many
    from triton_distributed_b200.ops import attention_reference, dense_block_table, gqa_fwd_batch_decode

    lens = [1, 15, 16, 17, 63, 64, 65, 0, 511]
    B, Hkv = len(lens), 2
    k, v, bt = _paged_cache(B, max(lens), Hkv, D, page or max(lens))
    if page == 0:
        bt = dense_block_table(B, "cuda")
    q = torch.randn(B, group * Hkv, D, device="cuda", dtype=torch.bfloat16)
    kv_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    keep = [i for i, n in enumerate(lens) if n]
    ref = attention_reference(q.float(), k.float(), v.float(), bt, cu, kv_lens, None, False)
    out = gqa_fwd_batch_decode(q, k, v, None, None, kv_lens, bt, kv_split=splits)
    torch.cuda.synchronize()
    assert out[7].abs().max() == 0
    # probabilities and output are rounded to bf16: 2^-9 each of sums of values of order one
    torch.testing.assert_close(out[keep].float(), ref[keep].float(), rtol=2 ** -7, atol=2 ** -7)


def test_decode_softcap():
    from triton_distributed_b200.ops import attention_reference, gqa_fwd_batch_decode

    B, Hq, Hkv, D = 2, 8, 2, 128
    k, v, bt = _paged_cache(B, 500, Hkv, D, 32)
    q = torch.randn(B, Hq, D, device="cuda", dtype=torch.bfloat16) * 3
    kv_lens = torch.tensor([500, 77], dtype=torch.int32, device="cuda")
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    ref = attention_reference(q, k, v, bt, cu, kv_lens, None, False, None, 20.0)
    out = gqa_fwd_batch_decode(q, k, v, None, None, kv_lens, bt, soft_cap=20.0)
    torch.testing.assert_close(out.float(), ref.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("cfg", [(2, 8, 2, 128, 16, [100, 257], [100, 257]), (1, 4, 4, 64, 64, [64], [200]),
                                 (3, 16, 2, 128, 1, [1, 70, 130], [5, 70, 300])])
def test_prefill_causal(cfg):
    from triton_distributed_b200.ops import attention_reference, flash_attn_varlen

    B, Hq, Hkv, D, page, qlens, kvlens = cfg
    k, v, bt = _paged_cache(B, max(kvlens), Hkv, D, page, seed=1)
    T = sum(qlens)
    q = torch.randn(T, Hq, D, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32, device="cuda")
    kv_lens = torch.tensor(kvlens, dtype=torch.int32, device="cuda")
    ref, ref_lse = attention_reference(q, k, v, bt, cu, kv_lens, None, True, None, 0.0, True)
    out, lse = flash_attn_varlen(q, k, v, bt, cu, kv_lens, max(qlens), causal=True, return_lse=True)
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), ref.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse, ref_lse, rtol=1e-2, atol=1e-2)
    # non-causal with explicit positions
    ref2 = attention_reference(q, k, v, bt, cu, kv_lens, None, False)
    out2 = flash_attn_varlen(q, k, v, bt, cu, kv_lens, max(qlens), causal=False)
    torch.testing.assert_close(out2.float(), ref2.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("impl", ["sm100", "mma"])
@pytest.mark.parametrize("cfg", [(2, 8, 2, 16, [300, 129], [300, 500], None),
                                 (1, 16, 8, 64, [1024], [1024], None),
                                 (2, 4, 1, 128, [128, 200], [384, 700], [256, 100])])
def test_prefill_both_kernels(cfg, impl):
    """The tcgen05 prefill kernel (KV packed into dense K / V^T, S and PV in TMEM) and the mma.sync kernel against the
    fp32 reference: ragged batches, paged caches with shuffled pages, explicit query positions (context-parallel chunks),
    causal and not."""
    from triton_distributed_b200.ops import attention_reference, flash_attn_varlen
    from triton_distributed_b200.ops.attention import check_attention_errors

    B, Hq, Hkv, page, qlens, kvlens, pos0 = cfg
    D = 128
    k, v, bt = _paged_cache(B, max(kvlens), Hkv, D, page, seed=2)
    q = torch.randn(sum(qlens), Hq, D, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32, device="cuda")
    kv_lens = torch.tensor(kvlens, dtype=torch.int32, device="cuda")
    qp = None if pos0 is None else torch.tensor(pos0, dtype=torch.int32, device="cuda")
    for causal in (True, False):
        ref, ref_lse = attention_reference(q, k, v, bt, cu, kv_lens, qp, causal, None, 0.0, True)
        out, lse = flash_attn_varlen(q, k, v, bt, cu, kv_lens, max(qlens), q_pos0=qp, causal=causal, return_lse=True, impl=impl)
        torch.cuda.synchronize()
        check_attention_errors()
        torch.testing.assert_close(out.float(), ref.float(), rtol=2e-2, atol=2e-2)
        torch.testing.assert_close(lse, ref_lse, rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("cap,sink,causal", [(0.0, False, True), (0.0, True, False), (15.0, False, True)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("qlens,kvlens,pos0", [([2048], [2048], None), ([127, 128, 129, 255, 256, 257, 1, 513], [127, 640, 129, 300, 256, 1025, 385, 513], None),
                                               ([700, 130], [900, 64], [200, 0]), ([640], [500], [-200])])
def test_prefill_two_tiles(D, qlens, kvlens, pos0, cap, sink, causal):
    # 256-row tiles of the tcgen05 kernel: rows, keys and causal edges on both sides of a tile and a block, tiles without a row or a
    # key, rows that see nothing, row maxima that outgrow their reference
    from triton_distributed_b200.ops import attention_reference, flash_attn_varlen
    from triton_distributed_b200.ops.attention import check_attention_errors

    torch.manual_seed(D)
    B, Hq, Hkv = len(qlens), 16, 2
    k, v, bt = _paged_cache(B, max(kvlens), Hkv, D, 48, seed=5)
    k *= torch.linspace(0.1, 3.0, 48, device="cuda").to(k.dtype)[None, :, None, None]
    q = torch.randn(sum(qlens), Hq, D, device="cuda", dtype=torch.bfloat16) * 2
    cu = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32, device="cuda")
    kv_lens = torch.tensor(kvlens, dtype=torch.int32, device="cuda")
    qp = None if pos0 is None else torch.tensor(pos0, dtype=torch.int32, device="cuda")
    sk = torch.randn(Hq, device="cuda") if sink else None
    ref, ref_lse = attention_reference(q.float(), k.float(), v.float(), bt, cu, kv_lens, qp, causal, None, cap, True, sk)
    out, lse = flash_attn_varlen(q, k, v, bt, cu, kv_lens, max(qlens), q_pos0=qp, causal=causal, softcap=cap, return_lse=True, impl="sm100", sink=sk)
    torch.cuda.synchronize()
    check_attention_errors()
    # probabilities and output are rounded to bf16, 2^-9 each, in sums of values of order one
    torch.testing.assert_close(out.float(), ref, rtol=2 ** -7, atol=2 ** -6)
    seen = ref_lse > float("-inf")
    assert torch.equal(lse > float("-inf"), seen)
    torch.testing.assert_close(lse[seen], ref_lse[seen], rtol=1e-4, atol=1e-4)


def _prompts_of_64(first=0, T=600, Hq=4, Hkv=2, lens=(600, 900), page=40):
    # two prompts of heads of 64, long enough for the tcgen05 kernel; q begins at element ``first`` of its storage
    B, D = len(lens), 64
    k, v, bt = _paged_cache(B, max(lens), Hkv, D, page, seed=7)
    q = torch.randn(B * T * Hq * D + 8, device="cuda").to(torch.bfloat16)[first:first + B * T * Hq * D].view(B * T, Hq, D)
    cu = torch.arange(0, (B + 1) * T, T, dtype=torch.int32, device="cuda")
    return q, k, v, bt, cu, torch.tensor(lens, dtype=torch.int32, device="cuda"), T


@pytest.mark.parametrize("first,cap", [(2, 0.0), (4, 0.0), (6, 5.0), (0, -3.0)])
def test_prefill_heads_of_64_what_tma_cannot_take(first, cap):
    from triton_distributed_b200.ops import flash_attn_varlen

    args = _prompts_of_64(first)
    out = flash_attn_varlen(*args, softcap=cap, max_kv_len=900)
    want = flash_attn_varlen(*args, softcap=cap, max_kv_len=900, impl="mma")
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    q, k, v, bt, cu, lens, T = args
    wide = torch.stack([bt, bt], 1)[:, 0]
    for impl in ("auto", "mma"):
        with pytest.raises(RuntimeError, match="block_table"):
            flash_attn_varlen(q, k, v, wide, cu, lens, T, max_kv_len=900, impl=impl)


@pytest.mark.parametrize("page", [40, 900])
def test_prefill_heads_of_64_do_not_depend_on_a_length_bound(page):
    # the block table says how many positions there may be; max_kv_len never mattered to these heads
    from triton_distributed_b200.ops import attention_reference, flash_attn_varlen

    q, k, v, bt, cu, lens, T = _prompts_of_64(page=page)
    ref = attention_reference(q.float(), k.float(), v.float(), bt, cu, lens)
    outs = [flash_attn_varlen(q, k, v, bt, cu, lens, T, max_kv_len=n) for n in (1, 64, 640, 900, 5000)]
    torch.cuda.synchronize()
    # probabilities and output are rounded to bf16, 2^-9 each, in sums of values of order one
    torch.testing.assert_close(outs[0].float(), ref.float(), rtol=2 ** -7, atol=2 ** -6)
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_prefill_heads_of_64_without_room_for_scratch(monkeypatch):
    # more scratch than the limit, or none to be had: the kernel that needs none
    from triton_distributed_b200.ops import attention, flash_attn_varlen

    args = _prompts_of_64()
    want = flash_attn_varlen(*args, max_kv_len=900, impl="mma")
    monkeypatch.setattr(attention, "SM100_SCRATCH_64", 2 * 2 * 2 * 960 * 64 * 2 - 1)
    assert torch.equal(flash_attn_varlen(*args, max_kv_len=900), want)
    monkeypatch.undo()
    tcgen05 = flash_attn_varlen(*args, max_kv_len=900)

    def full(*a, **kw):
        raise torch.cuda.OutOfMemoryError("no memory left")

    monkeypatch.setattr(attention.torch, "empty", full)
    got = flash_attn_varlen(*args, max_kv_len=900)
    monkeypatch.undo()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and not torch.equal(tcgen05, want)


def test_prefill_heads_of_64_wait_for_nothing():
    # however many calls: no error flag is read back
    from triton_distributed_b200.ops import attention, flash_attn_varlen

    args = _prompts_of_64()
    flash_attn_varlen(*args, max_kv_len=900)
    attention.check_attention_errors()
    torch.cuda.set_sync_debug_mode("error")
    try:
        for _ in range(150):
            flash_attn_varlen(*args, max_kv_len=900)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    assert not attention._PENDING_ERRORS
    # what a kernel reports is raised by the next call, once
    torch.cuda.synchronize()
    attention._STATUS_WORDS["word"][0] = 1
    with pytest.raises(RuntimeError, match="timed out"):
        flash_attn_varlen(*args, max_kv_len=900)
    flash_attn_varlen(*args, max_kv_len=900)
    attention._STATUS_WORDS["word"][0] = 2
    with pytest.raises(RuntimeError, match="aligned"):
        attention.check_attention_errors()
    attention.check_attention_errors()
