"""Gated delta rule CUDA kernel against the fp32 token recurrence."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("impl", ["chunk", "recurrent"])
@pytest.mark.parametrize("T,cu", [(257, None), (400, [0, 90, 91, 400])])
def test_gdn_kernel_matches_recurrence(T, cu, impl):
    from test_gdn_cpu import _inputs
    from triton_distributed_b200 import ops

    H, K, V = 4, 128, 128
    q, k, v, g, beta = _inputs(T, H, K, V, seed=3, dtype=torch.bfloat16, device="cuda")
    cu_t = None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda")
    n = 1 if cu is None else len(cu) - 1
    h0 = (torch.randn(n, H, K, V, device="cuda") * 0.05)
    scale = K ** -0.5
    gc, o, A, ht = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, scale, h0, True, cu_t, impl=impl)
    o_r, s_r = ops.gated_delta_rule_recurrent(q, k, v, g, beta, scale, h0, cu_t)
    torch.cuda.synchronize()
    assert A is None and gc.shape == (1, T, H)
    err_o = (o.float() - o_r).abs().max().item() / (o_r.abs().max().item() + 1e-6)
    err_s = (ht - s_r).abs().max().item() / (s_r.abs().max().item() + 1e-6)
    # the chunked form feeds bf16 copies of the state and of the WY factors to the tensor cores (as the reference does)
    assert err_o < 2e-2 and err_s < (2e-2 if impl == "chunk" else 1e-3), (impl, err_o, err_s)


@pytest.mark.parametrize("V", [64, 256])
def test_gdn_chunk_kernels_match_torch_chunked_form(V):
    """Every output of the chunk-parallel kernels (chunk-local cumulative decay, WY matrices A, outputs, final state)
    against the same algorithm in fp32 PyTorch, with ragged sequences (tail chunks of 1 and 27 tokens)."""
    from test_gdn_cpu import _inputs
    from triton_distributed_b200 import ops
    from triton_distributed_b200.ops.gdn import gated_delta_rule_chunked

    T, H, K = 64 * 3 + 1 + 91, 3, 128
    cu = torch.tensor([0, 193, 284], dtype=torch.int32, device="cuda")
    q, k, v, g, beta = _inputs(T, H, K, V, seed=5, dtype=torch.bfloat16, device="cuda")
    scale = K ** -0.5
    gc, o, A, ht = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, scale, None, True, cu, return_A=True, impl="chunk")
    gc_r, o_r, A_r, ht_r = gated_delta_rule_chunked(q, k, v, g, beta, scale, None, cu)
    torch.cuda.synchronize()
    torch.testing.assert_close(gc, gc_r, rtol=1e-4, atol=1e-4)
    assert (A - A_r).abs().max().item() < 2e-2 * max(1.0, A_r.abs().max().item())
    assert (o.float() - o_r).abs().max().item() < 2e-2 * (o_r.abs().max().item() + 1e-6)
    assert (ht - ht_r).abs().max().item() < 2e-2 * (ht_r.abs().max().item() + 1e-6)


@pytest.mark.parametrize("H,V,lens", [(2, 64, [1]), (2, 64, [64, 128]), (3, 192, [63, 65, 0, 130]), (2, 256, [0, 200, 17, 0]),
                                      (16, 128, [70]), (16, 128, [66, 129]), (16, 256, [5, 64, 100])])
def test_gdn_chunk_kernels_over_column_tiles_and_sequence_ends(H, V, lens):
    """Every width of the state walk (16 columns alone on an SM, 16 columns two to an SM, 32 columns), empty sequences, full and ragged
    last chunks.  Tolerance: operands of the products are bf16 (2^-9 relative), a result is a sum of a few of them."""
    from test_gdn_cpu import _inputs
    from triton_distributed_b200 import ops

    K, T = 128, sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    q, k, v, g, beta = _inputs(T, H, K, V, seed=11, dtype=torch.bfloat16, device="cuda")
    h0 = torch.randn(len(lens), H, K, V, device="cuda") * 0.1
    gc, o, A, ht = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, K ** -0.5, h0, True, cu, return_A=True, impl="chunk")
    o_r, s_r = ops.gated_delta_rule_recurrent(q, k, v, g, beta, K ** -0.5, h0, cu)
    cum = torch.cat([g[0, t:min(t + 64, b)].double().cumsum(0) for a, b in zip(cu.tolist(), cu.tolist()[1:]) for t in range(a, b, 64)])
    torch.testing.assert_close(gc[0].double(), cum, rtol=1e-5, atol=1e-5)
    # A of every chunk: the inverse of I + L, L = beta (k k^T) e^(gc_i - gc_j) below the diagonal, from what the kernel reads; its own
    # sums are fp32 and so are those of the inverse, 64 terms of order one at most
    for a, b in zip(cu.tolist(), cu.tolist()[1:]):
        for t in range(a, b, 64):
            n = min(t + 64, b) - t
            kk, gg, bb = k[0, t:t + n].double().transpose(0, 1), gc[0, t:t + n].double().t(), beta[0, t:t + n].double().t()
            L = ((kk @ kk.transpose(1, 2)) * bb[:, :, None] * torch.exp(gg[:, :, None] - gg[:, None, :])).tril(-1)
            want = torch.linalg.inv(torch.eye(n, device="cuda", dtype=torch.float64) + L)
            got = A[0, t:t + n].double().transpose(0, 1)
            torch.testing.assert_close(got[:, :, :n], want, rtol=1e-4, atol=1e-5)
            assert (got.triu(1) == 0).all()
    assert (o.float() - o_r).norm().item() < 2 ** -7 * o_r.norm().item()
    assert (ht - s_r).norm().item() < 2 ** -7 * s_r.norm().item()
    empty = [i for i, n in enumerate(lens) if n == 0]
    assert torch.equal(ht[empty], h0[empty])


def test_gdn_state_at_an_odd_address():
    """A contiguous initial state may begin at any element of its storage."""
    from test_gdn_cpu import _inputs
    from triton_distributed_b200 import ops

    H, K, V, lens = 2, 128, 64, [70, 5]
    cu = torch.tensor([0, 70, 75], dtype=torch.int32, device="cuda")
    q, k, v, g, beta = _inputs(75, H, K, V, seed=4, dtype=torch.bfloat16, device="cuda")
    flat = torch.randn(len(lens) * H * K * V + 3, device="cuda") * 0.1
    for first in (1, 2, 3):
        h0 = flat[first:first + len(lens) * H * K * V].view(len(lens), H, K, V)
        got = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, K ** -0.5, h0, True, cu, impl="chunk")
        want = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, K ** -0.5, h0.clone(), True, cu, impl="chunk")
        torch.cuda.synchronize()
        assert torch.equal(got[1], want[1]) and torch.equal(got[3], want[3])


def test_gdn_chunk_scratch():
    """The intermediates of a call take no more than w, u, v_new and the chunk states in the form with row-major operands did."""
    from test_gdn_cpu import _inputs
    from triton_distributed_b200 import ops

    T, H, K, V = 4096, 8, 128, 128
    q, k, v, g, beta = _inputs(T, H, K, V, seed=2, dtype=torch.bfloat16, device="cuda")
    cu = torch.tensor([0, T], dtype=torch.int32, device="cuda")
    ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, K ** -0.5, None, False, cu, impl="chunk")
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = ops.chunk_gated_delta_rule_fwd(q, k, v, g, beta, K ** -0.5, None, False, cu, impl="chunk")
    torch.cuda.synchronize()
    chunks = (T // 64 + 1) * H
    scratch = chunks * 2 * (64 * K + 2 * 64 * V + K * V)
    # results, and the allocator's 512-byte and 2 MB roundings
    assert torch.cuda.max_memory_allocated() - before <= scratch + T * H * (2 * V + 4) + (12 << 20), out[1].shape
