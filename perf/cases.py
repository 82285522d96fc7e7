"""The work this framework is used for on one GPU, as cases that can be timed and compared.

A case is a plain dict: ``kind`` says which path of the framework it takes, the rest are its sizes.  The kinds are what a serving
process spends its time on:

* ``mlp``        SwiGLU block of a dense decoder (``parallel.TP_MLP``): AG-GEMM / GEMM-RS mode for prompts, GEMM+AR mode for decode batches
* ``prefill``    causal attention of prompts over a paged KV cache, several sequences at once, some of them with cached context
* ``attention``  one decode step of attention for a batch of sequences of unequal length
* ``moe``        mixture-of-experts block of a sparse decoder (``parallel.TP_MoE``), prompts and decode batches
* ``gdn``        gated delta rule over packed sequences, the library call
* ``delta``      gated delta rule in its serving form (convolutions, unit norms, head norm and gate), packed prompts
* ``decode``     one decode step of a dense decoder from token ids to logits, captured once in a CUDA graph as the engine does
* ``fp8``        linear layer with block-scaled e4m3 operands: quantise the activations, multiply

``listed`` has one or two cases of each, ``draw`` more of the same ranges; ``exact`` restates every path in 64 bits.
"""
from __future__ import annotations

import math

import torch

import triton_distributed_b200 as tdb
from triton_distributed_b200 import ops
from triton_distributed_b200.models import DenseLLM, KV_Cache, ModelConfig
from triton_distributed_b200.parallel import TP_MLP, TP_MoE

BF = torch.bfloat16

# width and (per-rank) intermediate size of dense decoders: Qwen3-0.6B, Qwen3-8B, one of eight shards of Qwen3-32B and of Llama-3-70B
MLP_SIZES = ((1024, 3072), (4096, 12288), (5120, 3200), (8192, 3584))
# query heads, KV heads, head dim: Qwen3-8B, one of eight shards of Qwen3-32B, Qwen3-30B-A3B, and a 1b model with heads of 64
HEADS = ((32, 8, 128), (8, 1, 128), (32, 4, 128), (24, 4, 64))
# width, expert intermediate size, experts, chosen: Qwen3-30B-A3B and a 1b model
MOE_SIZES = ((2048, 768, 128, 8), (1536, 512, 32, 4))
# value heads, key heads, key and value dim of a head, taps: the 8b and 1b sizes of the several-stream decoder
DELTA_SIZES = ((32, 16, 128, 128, 4), (12, 6, 64, 128, 4))
DECODE_MODELS = ("Qwen/Qwen3-0.6B", "Qwen/Qwen3-8B", "Qwen/Qwen3-32B-tp8-shard")
DECODE_LAYERS = 4
FP8_SIZES = ((4096, 4096), (12288, 4096), (4096, 12288), (3584, 8192))


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a long prompt through the MLP of a 70B-class model: the headline AG-GEMM / GEMM-RS sizes, the largest GEMMs there are
        dict(name="mlp-prompt-8192", kind="mlp", tokens=8192, width=8192, inter=28672),
        # a portion of a prompt of odd length through an 8B model's MLP
        dict(name="mlp-prompt-777", kind="mlp", tokens=777, width=4096, inter=12288),
        # a decode batch through one of eight shards of a 32B model's MLP: weights are streamed once for a few rows
        dict(name="mlp-decode-48", kind="mlp", tokens=48, width=5120, inter=3200),
        # one 8192-token prompt, grouped-query attention of an 8B model
        dict(name="prefill-1x8192", kind="prefill", seqs=1, tokens=8192, context=0, q_heads=32, kv_heads=8, dim=128, lens_seed=0),
        # five prompts of unequal, odd lengths packed together, heads of 64, part of the context cached by an earlier step
        dict(name="prefill-5-ragged-d64", kind="prefill", seqs=5, tokens=4001, context=700, q_heads=24, kv_heads=4, dim=64, lens_seed=3),
        # a full decode batch at long context: bound by the KV cache's bytes
        dict(name="attention-64x4096", kind="attention", batch=64, context=4096, page=0, q_heads=32, kv_heads=8, dim=128, lens_seed=1),
        # a prompt through the sparse MLP of a 30B-A3B model
        dict(name="moe-prompt-4096", kind="moe", tokens=4096, width=2048, inter=768, experts=128, topk=8),
        # a small decode batch through the same block: few rows per expert
        dict(name="moe-decode-8", kind="moe", tokens=8, width=2048, inter=768, experts=128, topk=8),
        # gated delta rule over one long sequence
        dict(name="gdn-8192", kind="gdn", seqs=1, tokens=8192, heads=16, vdim=128, state=False, lens_seed=0),
        # the serving form over three packed prompts of odd lengths
        dict(name="delta-3-ragged", kind="delta", seqs=3, tokens=6001, heads=32, key_heads=16, kdim=128, vdim=128, taps=4, lens_seed=2),
        # single-stream decoding: latency of one token
        dict(name="decode-8b-batch1", kind="decode", model="Qwen/Qwen3-8B", batch=1, context=4096),
        # an fp8 linear layer on a prompt
        dict(name="fp8-4096", kind="fp8", tokens=4096, n=12288, k=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mlp", "prefill", "attention", "moe", "gdn", "delta", "decode", "fp8"))
    seed = rng.randrange(1 << 20)
    if kind == "mlp":
        width, inter = rng.choice(MLP_SIZES)
        return dict(kind=kind, tokens=_log(rng, 1, 8192), width=width, inter=inter)
    if kind == "prefill":
        hq, hkv, dim = rng.choice(HEADS)
        tokens = _log(rng, 128, 8192)
        return dict(kind=kind, seqs=rng.randint(1, min(8, tokens // 64)), tokens=tokens, context=rng.choice((0, 0, rng.randint(1, 2048))),
                    q_heads=hq, kv_heads=hkv, dim=dim, lens_seed=seed)
    if kind == "attention":
        hq, hkv, dim = rng.choice(HEADS)
        batch = _log(rng, 1, 64)
        return dict(kind=kind, batch=batch, context=_log(rng, 128, 32768 if batch <= 8 else 8192), page=rng.choice((0, 0, 16, 64)),
                    q_heads=hq, kv_heads=hkv, dim=dim, lens_seed=seed)
    if kind == "moe":
        width, inter, experts, topk = rng.choice(MOE_SIZES)
        return dict(kind=kind, tokens=_log(rng, 1, 8192), width=width, inter=inter, experts=experts, topk=topk)
    if kind == "gdn":
        tokens = _log(rng, 64, 16384)
        return dict(kind=kind, seqs=rng.randint(1, min(8, tokens // 32)), tokens=tokens, heads=rng.choice((4, 8, 16, 32)),
                    vdim=rng.choice((64, 128, 128, 256)), state=rng.random() < 0.5, lens_seed=seed)
    if kind == "delta":
        heads, key_heads, kdim, vdim, taps = rng.choice(DELTA_SIZES)
        tokens = _log(rng, 64, 8192)
        return dict(kind=kind, seqs=rng.randint(1, min(8, tokens // 32)), tokens=tokens, heads=heads, key_heads=key_heads, kdim=kdim,
                    vdim=vdim, taps=taps, lens_seed=seed)
    if kind == "decode":
        return dict(kind=kind, model=rng.choice(DECODE_MODELS), batch=_log(rng, 1, 64), context=_log(rng, 128, 8192))
    n, k = rng.choice(FP8_SIZES)
    return dict(kind=kind, tokens=_log(rng, 128, 8192), n=n, k=k)


def _lengths(total, parts, seed):
    """``parts`` unequal lengths that add up to ``total``."""
    if parts == 1:
        return [total]
    gen = torch.Generator().manual_seed(seed)
    share = 0.25 + torch.rand(parts, generator=gen, dtype=torch.float64)
    ends = [int(e) for e in (share.cumsum(0) / share.sum() * total).round().tolist()]
    return [b - a for a, b in zip([0] + ends[:-1], ends)]


def _packed(c):
    return _lengths(c["tokens"], c["seqs"], c["lens_seed"])


def _prefill_kv_lens(c):
    """Context of every sequence behind the step: the new tokens and, for every other sequence, what is cached before them."""
    return [n + (c["context"] if i % 2 == 0 else 0) for i, n in enumerate(_packed(c))]


def _decode_lens(c):
    gen = torch.Generator().manual_seed(c["lens_seed"])
    lo = (c["context"] + 1) // 2
    return [c["context"]] + torch.randint(lo, c["context"] + 1, (c["batch"] - 1,), generator=gen).tolist()


def _cu(lens, dev="cuda"):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return torch.tensor(out, dtype=torch.int32, device=dev)


def _gen(seed):
    tdb.initialize_distributed(seed=0)
    return torch.Generator(device="cuda").manual_seed(seed)


def _rnd(gen, *shape, std=1.0, dtype=BF):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(dtype)


# ------------------------------------------------------------------ inputs
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, _gen(seed), seed)


def run(state):
    with torch.no_grad():
        return state["run"](state)


def _decode_sized(c):
    return c["tokens"] <= 64


def _prepare_mlp(c, gen, seed):
    layer = TP_MLP()
    layer.init_random(c["width"], c["inter"], seed=seed)
    if _decode_sized(c):
        layer._init_gemm_ar_ctx(c["tokens"])
        layer.set_fwd("triton_dist_gemm_ar")
    else:
        layer._init_ctx(c["tokens"])
        layer.set_fwd("triton_dist")
    return dict(run=lambda s: s["layer"](s["x"]), layer=layer, x=_rnd(gen, c["tokens"], c["width"]))


def _prepare_prefill(c, gen, seed):
    lens, kv = _packed(c), _prefill_kv_lens(c)
    hq, hkv, d = c["q_heads"], c["kv_heads"], c["dim"]
    longest = max(kv)
    return dict(run=lambda s: ops.flash_attn_varlen(s["q"], s["k"], s["v"], s["table"], s["cu"], s["kv_lens"], s["max_q"], max_kv_len=s["max_kv"]),
                q=_rnd(gen, c["tokens"], hq, d), k=_rnd(gen, c["seqs"], longest, hkv, d), v=_rnd(gen, c["seqs"], longest, hkv, d),
                table=ops.dense_block_table(c["seqs"], "cuda"), cu=_cu(lens), kv_lens=torch.tensor(kv, dtype=torch.int32, device="cuda"),
                max_q=max(lens), max_kv=longest)


def _prepare_attention(c, gen, seed):
    lens, b, hq, hkv, d = _decode_lens(c), c["batch"], c["q_heads"], c["kv_heads"], c["dim"]
    page = c["page"] or c["context"]
    per = -(-c["context"] // page)
    table = torch.randperm(b * per, device="cuda", generator=gen).to(torch.int32).reshape(b, per) if c["page"] else ops.dense_block_table(b, "cuda")
    return dict(run=lambda s: ops.gqa_fwd_batch_decode(s["q"], s["k"], s["v"], None, None, s["kv_lens"], s["table"]),
                q=_rnd(gen, b, hq, d), k=_rnd(gen, b * per, page, hkv, d), v=_rnd(gen, b * per, page, hkv, d), table=table.contiguous(),
                kv_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"))


def _prepare_moe(c, gen, seed):
    layer = TP_MoE()
    layer.init_random(c["width"], c["inter"], c["experts"], c["topk"], seed=seed)
    # A trained router decides clearly: its rows are orthogonal and a token's logits lie apart by more than their rounding, so that
    # which experts are chosen does not depend on the order of a sum.
    E, W, T = c["experts"], c["width"], c["tokens"]
    rows = torch.linalg.qr(torch.randn(W, E, device="cuda", generator=gen, dtype=torch.float64))[0].t()
    layer.router_w = rows.to(BF).contiguous()
    logits = torch.rand(T, E, device="cuda", generator=gen).argsort(1).double() * (8.0 / E)
    noise = torch.randn(T, W, device="cuda", generator=gen, dtype=torch.float64)
    w = layer.router_w.double()
    back = torch.linalg.solve(w @ w.t(), logits.t() - w @ noise.t()).t()
    layer._init_ctx(T)
    layer.set_fwd("triton_dist_AR")
    return dict(run=lambda s: s["layer"](s["x"]), layer=layer, x=(noise + back @ w).to(BF))


def _prepare_gdn(c, gen, seed):
    T, H, K, V = c["tokens"], c["heads"], 128, c["vdim"]
    k = torch.nn.functional.normalize(torch.randn(1, T, H, K, device="cuda", generator=gen), dim=-1).to(BF)
    return dict(run=lambda s: ops.chunk_gated_delta_rule_fwd(s["q"], s["k"], s["v"], s["g"], s["beta"], 128 ** -0.5, s["h0"], True, s["cu"]),
                q=_rnd(gen, 1, T, H, K), k=k, v=_rnd(gen, 1, T, H, V), beta=torch.rand(1, T, H, device="cuda", generator=gen).to(BF),
                g=torch.nn.functional.logsigmoid(torch.randn(1, T, H, device="cuda", generator=gen) + 2.0),
                h0=_rnd(gen, c["seqs"], H, K, V, std=0.1, dtype=torch.float32) if c["state"] else None, cu=_cu(_packed(c)))


def _prepare_delta(c, gen, seed):
    T, H, G, dk, dv, taps, N = c["tokens"], c["heads"], c["key_heads"], c["kdim"], c["vdim"], c["taps"], c["seqs"]
    C = 2 * G * dk + H * dv
    lens = _packed(c)
    ends = _cu(lens, "cpu").tolist()
    f32 = torch.float32

    def step(s):
        out = ops.gated_delta_rule(s["z"], s["ab"], s["conv_w"], s["a_log"], s["dt_bias"], s["norm_w"], s["state"], s["conv"], s["slots"], s["pos0"],
                                   s["cu"], G, dv, dk ** -0.5, 1e-5, s["tables"])
        return out, s["state"], s["conv"]

    return dict(run=step, z=_rnd(gen, T, C + H * dv), ab=_rnd(gen, T, 2 * H, dtype=f32), conv_w=_rnd(gen, C, taps, std=taps ** -0.5, dtype=f32),
                a_log=_rnd(gen, H, std=0.5, dtype=f32), dt_bias=_rnd(gen, H, dtype=f32) - 2.0, norm_w=1.0 + _rnd(gen, dv, std=0.1, dtype=f32),
                state=torch.zeros(N, H, dk, dv, device="cuda"), conv=torch.zeros(N, taps, C, device="cuda", dtype=BF),
                slots=torch.arange(N, dtype=torch.int32, device="cuda"), pos0=torch.zeros(N, dtype=torch.int64, device="cuda"), cu=_cu(lens),
                tables=ops.gla_chunk_tables(ends, "cuda"))


def _decode_inputs(c, seed, arch):
    """Token ids and the cached keys and values [layers, batch, context, heads, dim], the same for ``prepare`` and ``exact``."""
    gen = _gen(seed + 1)
    shape = (arch.num_hidden_layers, c["batch"], c["context"], arch.num_key_value_heads, arch.head_dim)
    return torch.randint(0, arch.vocab_size, (c["batch"], 1), device="cuda", generator=gen), _rnd(gen, *shape), _rnd(gen, *shape)


def _decode_config(c, seed):
    return ModelConfig(model_name=c["model"], max_length=c["context"] + 64, num_layers_override=DECODE_LAYERS, seed=seed)


def _prepare_decode(c, gen, seed):
    mode = "triton_dist_gemm_ar"
    model = DenseLLM(_decode_config(c, seed))
    a = model.arch
    ids, k, v = _decode_inputs(c, seed, a)
    cache = KV_Cache(a.num_hidden_layers, c["batch"], c["context"] + 64, a.num_key_value_heads, a.head_dim, device="cuda")
    cache.k_cache[:, :, :c["context"]] = k
    cache.v_cache[:, :, :c["context"]] = v
    cache.kv_offset.fill_(c["context"])
    del k, v
    model.init_ctx_for(mode, c["batch"])
    model.set_fwd(mode)
    logits = torch.empty(c["batch"], a.vocab_size, device="cuda")

    def step():
        pos = cache.kv_offset[:c["batch"]].to(torch.int64).unsqueeze(1)
        logits.copy_(model.inference(ids, pos, cache))

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(side):
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        step()

    def replay(s):
        s["graph"].replay()
        return s["logits"], s["cache"].k_cache[:, :, c["context"]], s["cache"].v_cache[:, :, c["context"]]

    return dict(run=replay, graph=graph, model=model, cache=cache, ids=ids, logits=logits)


def _prepare_fp8(c, gen, seed):
    x = _rnd(gen, c["tokens"], c["k"])
    wq, ws = ops.quantize_weight_128x128(_rnd(gen, c["n"], c["k"], std=0.02))

    def step(s):
        xq, xs = ops.quantize_act_1x128(s["x"])
        return ops.gemm_fp8_blockscaled(xq, xs, s["wq"], s["ws"])

    return dict(run=step, x=x, wq=wq, ws=ws)


# ------------------------------------------------------------------ what a pass cannot do without
def work(c):
    return globals()["_work_" + c["kind"]](c)


def _work_mlp(c):
    T, W, F = c["tokens"], c["width"], c["inter"]
    return {"bytes": 2 * (3 * W * F + 2 * T * W), "flops": 6.0 * T * W * F}


def _work_prefill(c):
    pairs = sum(n * (kv - n) + n * (n + 1) / 2 for n, kv in zip(_packed(c), _prefill_kv_lens(c)))
    return {"bytes": 2 * c["dim"] * (2 * c["tokens"] * c["q_heads"] + 2 * sum(_prefill_kv_lens(c)) * c["kv_heads"]),
            "flops": 4.0 * pairs * c["dim"] * c["q_heads"]}


def _work_attention(c):
    seen = sum(_decode_lens(c))
    return {"bytes": 2 * c["dim"] * (2 * seen * c["kv_heads"] + 2 * c["batch"] * c["q_heads"]), "flops": 4.0 * seen * c["dim"] * c["q_heads"]}


def _work_moe(c):
    T, W, F, E, k = c["tokens"], c["width"], c["inter"], c["experts"], c["topk"]
    used = E * (1 - (1 - k / E) ** T)      # experts that somebody chose
    return {"bytes": 2 * (used * 3 * W * F + E * W + 2 * T * W), "flops": 6.0 * T * k * W * F + 2.0 * T * E * W}


def _work_gdn(c):
    T, H, K, V, N = c["tokens"], c["heads"], 128, c["vdim"], c["seqs"]
    return {"bytes": T * H * (2 * (2 * K + 2 * V) + 2 + 8) + 4 * N * H * K * V * (2 if c["state"] else 1), "flops": T * H * 6.0 * K * V}


def _work_delta(c):
    T, H, G, dk, dv, N = c["tokens"], c["heads"], c["key_heads"], c["kdim"], c["vdim"], c["seqs"]
    return {"bytes": T * (2 * (2 * G * dk + 3 * H * dv) + 8 * H) + 4 * N * H * dk * dv, "flops": T * H * 6.0 * dk * dv}


def _work_decode(c):
    a = _decode_config(c, 0).arch()
    W, L, B = a.hidden_size, a.num_hidden_layers, c["batch"]
    layer = W * (a.num_attention_heads * 2 + a.num_key_value_heads * 2) * a.head_dim + 3 * W * a.intermediate_size
    weights = L * layer + W * a.vocab_size
    kv = 2 * L * B * c["context"] * a.num_key_value_heads * a.head_dim
    return {"bytes": 2 * (weights + kv) + 4 * B * a.vocab_size, "flops": 2.0 * B * weights + 2.0 * kv * a.num_attention_heads / a.num_key_value_heads}


def _work_fp8(c):
    T, N, K = c["tokens"], c["n"], c["k"]
    return {"bytes": 2 * T * K + N * K + 2 * T * N, "flops": 2.0 * T * N * K}


# ------------------------------------------------------------------ how far two correct implementations may be apart
def tolerance(c):
    # Four times what the path was measured to be off its 64-bit value: activations are rounded to bf16 between kernels, so
    # results are off by a few of their 2^-9 steps; ``max`` is for single values in sums of many roundings.
    return {"mlp": {"rel": 0.014, "max": 0.1}, "prefill": {"rel": 0.008, "max": 0.1}, "attention": {"rel": 0.009, "max": 0.1},
            "moe": {"rel": 0.018, "max": 0.12}, "gdn": {"rel": 0.014, "max": 0.15}, "delta": {"rel": 0.009, "max": 0.15},
            "decode": {"rel": 0.03, "max": 0.2}, "fp8": {"rel": 0.01, "max": 0.06}}[c["kind"]]


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return globals()["_exact_" + case["kind"]](case, seed)


def _swiglu(x, gate_up, down):
    g, u = (x @ gate_up.double().t()).chunk(2, dim=-1)
    return (torch.nn.functional.silu(g) * u) @ down.double().t()


def _exact_mlp(c, seed):
    s = prepare(c, seed)
    return _swiglu(s["x"].double(), s["layer"].gate_up_proj, s["layer"].down_proj)


def _attend(q, k, v, first, scale):
    """Attention of ``q`` [n, Hq, D] at positions ``first`` .. over ``k`` / ``v`` [m, Hkv, D], a slice of queries at a time."""
    n, hq, _ = q.shape
    g = hq // k.shape[1]
    out = torch.empty(n, hq, v.shape[-1], dtype=torch.float64, device=q.device)
    for h in range(hq):
        kh, vh = k[:, h // g].double(), v[:, h // g].double()
        for i in range(0, n, 2048):
            s = q[i:i + 2048, h].double() @ kh.t() * scale
            pos = torch.arange(i, i + s.shape[0], device=q.device) + first
            s.masked_fill_(torch.arange(kh.shape[0], device=q.device) > pos[:, None], float("-inf"))
            out[i:i + 2048, h] = torch.softmax(s, dim=-1) @ vh
    return out


def _exact_prefill(c, seed):
    s = prepare(c, seed)
    out, at = [], 0
    for b, (n, kv) in enumerate(zip(_packed(c), _prefill_kv_lens(c))):
        out.append(_attend(s["q"][at:at + n], s["k"][b, :kv], s["v"][b, :kv], kv - n, c["dim"] ** -0.5))
        at += n
    return torch.cat(out)


def _exact_attention(c, seed):
    s = prepare(c, seed)
    out = []
    for b, n in enumerate(_decode_lens(c)):
        k, v = (s[x][s["table"][b].long()].reshape(-1, c["kv_heads"], c["dim"])[:n] for x in "kv")
        out.append(_attend(s["q"][b:b + 1], k, v, n - 1, c["dim"] ** -0.5))
    return torch.cat(out)


def _exact_moe(c, seed):
    s = prepare(c, seed)
    layer, x = s["layer"], s["x"].double()
    w, ids = torch.softmax(x @ layer.router_w.double().t(), dim=-1).topk(c["topk"], dim=-1)
    w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(c["experts"]):
        t, slot = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, t, w[t, slot, None] * _swiglu(x[t], layer.w13[e], layer.w2[e]))
    return out


def _delta_tokens(q, k, v, g, beta, S, scale):
    """Token by token: ``S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = scale S^T q``."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.matmul(k[t].unsqueeze(1), S).squeeze(1))
        S = S + k[t].unsqueeze(2) * u.unsqueeze(1)
        out[t] = torch.matmul(q[t].unsqueeze(1), S).squeeze(1) * scale
    return out, S


def _exact_gdn(c, seed):
    s = prepare(c, seed)
    q, k, v, g, beta = (s[x][0].double() for x in ("q", "k", "v", "g", "beta"))
    cum, outs, states, at = torch.empty_like(g), [], [], 0
    for n, length in enumerate(_packed(c)):
        i = slice(at, at + length)
        for t in range(at, at + length, 64):
            cum[t:min(t + 64, at + length)] = g[t:min(t + 64, at + length)].cumsum(0)
        S = s["h0"][n].double() if c["state"] else torch.zeros(c["heads"], 128, c["vdim"], dtype=torch.float64, device="cuda")
        o, S = _delta_tokens(q[i], k[i], v[i], g[i].exp(), beta[i], S, 128 ** -0.5)
        outs.append(o)
        states.append(S)
        at += length
    return cum.unsqueeze(0), torch.cat(outs).unsqueeze(0), None, torch.stack(states)


def _exact_delta(c, seed):
    s = prepare(c, seed)
    H, G, dk, dv, taps = c["heads"], c["key_heads"], c["kdim"], c["vdim"], c["taps"]
    F = torch.nn.functional
    C = 2 * G * dk + H * dv
    z, ab, w = s["z"].double(), s["ab"].double(), s["conv_w"].double()
    g = torch.exp(-torch.exp(s["a_log"].double()) * F.softplus(ab[:, :H] + s["dt_bias"].double()))
    beta = torch.sigmoid(ab[:, H:])
    outs, states, rings, at = [], [], [], 0
    for length in _packed(c):
        i = slice(at, at + length)
        x = F.pad(z[i, :C], (0, 0, taps - 1, 0))
        y = F.silu(sum(x[j:j + length] * w[:, j] for j in range(taps)))
        q, k, v = y.split([G * dk, G * dk, H * dv], dim=1)
        q, k = (t.reshape(length, G, dk) for t in (q, k))
        q, k = ((t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1) for t in (q, k))
        o, S = _delta_tokens(q, k, v.reshape(length, H, dv), g[i], beta[i], torch.zeros(H, dk, dv, dtype=torch.float64, device="cuda"), dk ** -0.5)
        o = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-5) * s["norm_w"].double()
        outs.append(o.reshape(length, H * dv) * F.silu(z[i, C:]))
        states.append(S)
        ring = torch.zeros(taps, C, dtype=torch.float64, device="cuda")
        for p in range(max(0, length - taps + 1), length):      # what the next token's convolution reads
            ring[p % taps] = z[at + p, :C]
        rings.append(ring)
        at += length
    return torch.cat(outs), torch.stack(states), torch.stack(rings)


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _turned(x, pos, theta):
    """Rotary embedding of ``x`` [B, heads, D] at position ``pos``, halves of the head paired."""
    half = x.shape[-1] // 2
    ang = pos * theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _exact_decode(c, seed):
    _gen(seed)
    model = DenseLLM(_decode_config(c, seed))
    a, B, n = model.arch, c["batch"], c["context"]
    ids, kc, vc = _decode_inputs(c, seed, a)
    hq, hkv, d = a.num_attention_heads, a.num_key_value_heads, a.head_dim
    x = model.embed_tokens[ids[:, 0]].double()
    new_k, new_v = [], []
    for i, l in enumerate(model.layers):
        qkv = _norm64(x, l.input_norm_w, a.rms_norm_eps) @ l.attn.wqkv.double().t()
        q, k, v = (t.reshape(B, -1, d) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
        if a.qk_norm:
            q, k = _norm64(q, l.attn.q_norm_w, a.rms_norm_eps), _norm64(k, l.attn.k_norm_w, a.rms_norm_eps)
        q, k = _turned(q, n, a.rope_theta), _turned(k, n, a.rope_theta)
        o = torch.cat([_attend(q[b:b + 1], torch.cat([kc[i, b].double(), k[b:b + 1]]), torch.cat([vc[i, b].double(), v[b:b + 1]]), n, d ** -0.5)
                       for b in range(B)])
        x = x + o.reshape(B, hq * d) @ l.attn.wo.double().t()
        x = x + _swiglu(_norm64(x, l.post_norm_w, a.rms_norm_eps), l.mlp.gate_up_proj, l.mlp.down_proj)
        new_k.append(k)
        new_v.append(v)
    return _norm64(x, model.final_norm_w, a.rms_norm_eps) @ model.lm_head.double().t(), torch.stack(new_k), torch.stack(new_v)


def _exact_fp8(c, seed):
    s = prepare(c, seed)
    T, K = s["x"].shape
    x = s["x"].double().reshape(T, K // 128, 128)
    scale = x.abs().amax(-1, keepdim=True) / 448.0
    x = (x / scale).to(torch.float8_e4m3fn).double() * scale
    w = s["wq"].double().reshape(c["n"], K // 128, 128) * s["ws"].double().repeat_interleave(128, dim=0)[:c["n"], :, None]
    return x.reshape(T, K) @ w.reshape(c["n"], K).t()
