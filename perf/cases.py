"""The work this framework is used for, as cases that can be timed and compared.

Four kinds, all through the public entry points:

* ``linear``    one W4A16 linear called as a model calls it (``WALinear.forward``; ``quant.gemm_awq_ut`` where the
                caller has only the packed tensors), weights quantised from N(0, 0.02), activations N(0, 1);
* ``step``      one token step of a decoder stack over a filled KV cache, captured in a CUDA graph as the generation
                loop does, logits out (for whatever picks the next token);
* ``prefill``   ``Decoder.forward`` over a batch of prompts: logits of the last position and the filled KV cache;
* ``quantize``  quantise-and-pack of one fp16 weight, what loading a model does once per linear.

Sizes are those of the repository's own configurations (OPT-6.7B-, LLaMA-2-7B- and BERT-large-shaped linears and
stacks, group 128 / 64) and generic ones around them.  Stacks keep the configurations' layer shapes with fewer layers:
every layer is the same work.
"""
import math
import os
import sys
from dataclasses import replace

import torch

# the packages `quant` and `w4a16` live in a folder whose name is not an identifier
_PKG = os.path.join(os.getcwd(), "sparse-quant_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import quant  # noqa: E402
from w4a16 import WALinear  # noqa: E402
from w4a16.models import Decoder, DecoderConfig  # noqa: E402


def listed():
    return [
        # the smallest call there is: one token through one square projection, an eager call at a time
        dict(name="linear 1 token", kind="linear", tokens=1, K=4096, N=4096, g=128, bias=False, relu=False, residual=False, raw=True),
        # a batch of 24 sequences through the fused q/k/v projection: more tokens than one decode tile, fewer than a prefill tile
        dict(name="linear 24 tokens", kind="linear", tokens=24, K=4096, N=12288, g=128, bias=True, relu=False, residual=False, raw=False),
        # BERT-large feed-forward up-projection, batch 4 x 128 positions: a short K, the encoder's call
        dict(name="linear 512 short K", kind="linear", tokens=512, K=1024, N=4096, g=128, bias=True, relu=False, residual=False, raw=False),
        # a prompt of odd length through a group-64 projection
        dict(name="linear 333 ragged", kind="linear", tokens=333, K=4096, N=11008, g=64, bias=False, relu=False, residual=False, raw=False),
        # prefill of 2048 tokens through the wide feed-forward projection with its ReLU
        dict(name="linear 2048 relu", kind="linear", tokens=2048, K=4096, N=16384, g=128, bias=True, relu=True, residual=False, raw=False),
        # the largest linear: 8192 tokens through the long-K projection, residual added in the epilogue
        dict(name="linear 8192 residual", kind="linear", tokens=8192, K=16384, N=4096, g=128, bias=True, relu=False, residual=True, raw=False),
        # interactive decoding: one sequence, short context, latency is everything
        dict(name="step 1 sequence", kind="step", arch="opt", layers=8, hidden=4096, heads=32, ffn=16384, vocab=50272, g=128, batch=1, context=77),
        # the OPT-6.7B workload: batch 8, 512-token prompts
        dict(name="step 8 sequences", kind="step", arch="opt", layers=8, hidden=4096, heads=32, ffn=16384, vocab=50272, g=128, batch=8, context=520),
        # the LLaMA-2-7B workload: batch 32, 1024-token prompts, group 64, rotary embedding, SwiGLU
        dict(name="step 32 sequences", kind="step", arch="llama", layers=6, hidden=4096, heads=32, ffn=11008, vocab=32000, g=64, batch=32, context=1030),
        # prefill of the OPT-6.7B workload: 8 prompts of 512 tokens
        dict(name="prefill 8x512", kind="prefill", arch="opt", layers=4, hidden=4096, heads=32, ffn=16384, vocab=50272, g=128, batch=8, seq=512),
        # a few prompts of an odd length through the LLaMA-shaped stack
        dict(name="prefill 3x333", kind="prefill", arch="llama", layers=4, hidden=4096, heads=32, ffn=11008, vocab=32000, g=64, batch=3, seq=333),
        # loading a model: quantise and pack the largest linear of the OPT-6.7B-shaped stack
        dict(name="quantize 16384x4096", kind="quantize", K=4096, N=16384, g=128),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step) * step, lo), hi))


def _stack(rng):
    """Architecture and widths of a drawn decoder stack: heads of 128, widths around the configurations' own."""
    arch = rng.choice(("opt", "llama"))
    heads = rng.choice((16, 20, 24, 32, 32, 40))
    hidden = 128 * heads
    g = rng.choice((64, 128))
    ffn = 4 * hidden if arch == "opt" else round(2.6875 * hidden / 128) * 128
    return dict(arch=arch, layers=rng.randint(2, 6), hidden=hidden, heads=heads, ffn=ffn, vocab=rng.choice((32000, 50272)), g=g)


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "step", "step", "prefill", "quantize"))
    if kind == "linear":
        g = rng.choice((64, 128))
        K, N = _log(rng, 768, 16384, g), _log(rng, 768, 22016, 32)
        tokens = _log(rng, 1, 8192)
        while tokens * K * N > 8192 * 16384 * 4096:
            tokens = tokens // 2
        return dict(kind=kind, tokens=tokens, K=K, N=N, g=g, bias=rng.random() < 0.5, relu=rng.random() < 0.25,
                    residual=rng.random() < 0.25, raw=False)
    if kind == "step":
        s = _stack(rng)
        batch = _log(rng, 1, 64)
        context = min(_log(rng, 16, 1536), 32 * 1030 // batch)
        return dict(kind=kind, **s, batch=batch, context=context)
    if kind == "prefill":
        s = _stack(rng)
        s["layers"] = min(s["layers"], 3)
        batch = _log(rng, 1, 16)
        return dict(kind=kind, **s, batch=batch, seq=min(_log(rng, 24, 1536), 3072 // batch))
    g = rng.choice((64, 128))
    return dict(kind=kind, K=_log(rng, 768, 8192, g), N=_log(rng, 768, 8192, 32), g=g)


def _randn(gen, *shape, std=1.0):
    return (torch.randn(shape, device="cuda", generator=gen) * std).half()


def _config(case):
    base = DecoderConfig.opt_6_7b() if case["arch"] == "opt" else DecoderConfig.llama2_7b()
    return replace(base, layers=case["layers"], hidden=case["hidden"], heads=case["heads"], ffn=case["ffn"],
                   vocab=case["vocab"], group_size=case["g"])


def _logits(model, tok, pos_t, stats):
    """One token step as Decoder.step_static takes it, for a caller that picks the next token itself from the logits."""
    cfg = model.cfg
    x = model.embed[tok]
    rope = None
    if cfg.kind == "opt":
        x = x + model.pos_embed.index_select(0, pos_t + 2)
    else:
        rope = (model.rope_cos, model.rope_sin)
    x = x.contiguous()
    for i, layer in enumerate(model.layers):
        x = layer.forward_static(x, pos_t, rope, stats and (stats[1] if i else None, stats[0], stats[1]))
    norm = model.final_norm
    rms = cfg.kind != "opt"
    _, h = quant.add_norm(x, None, norm.weight, None if rms else norm.bias, norm.eps, rms)
    return h[:, -1] @ model.lm_head.t()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "quantize":
        return dict(case=case, w=_randn(gen, case["N"], case["K"], std=0.02))
    if kind == "linear":
        K, N = case["K"], case["N"]
        lin = torch.nn.Linear(K, N, bias=case["bias"], device="cuda", dtype=torch.float16)
        lin.weight.data = _randn(gen, N, K, std=0.02)
        if case["bias"]:
            lin.bias.data = _randn(gen, N, std=0.02)
        q = WALinear.from_float(lin, {"n_bit": 4, "group_size": case["g"]})
        torch.cuda.synchronize()
        q.static_weights = True
        state = dict(case=case, lin=q, x=_randn(gen, 1, case["tokens"], K), extra={})
        if case["relu"]:
            state["extra"]["relu"] = True
        if case["residual"]:
            state["extra"]["residual"] = _randn(gen, 1, case["tokens"], N)
        return state
    cfg = _config(case)
    model = Decoder(cfg, seed=seed).mark_static()
    batch = case["batch"]
    if kind == "prefill":
        return dict(case=case, model=model, ids=torch.randint(0, cfg.vocab, (batch, case["seq"]), device="cuda", generator=gen))
    context = case["context"]
    model.reset(batch, context + 32)
    for layer in model.layers:
        layer.k_cache.normal_(generator=gen)
        layer.v_cache.normal_(generator=gen)
    tok = torch.randint(0, cfg.vocab, (batch, 1), device="cuda", generator=gen)
    pos_t = torch.full((1,), context, dtype=torch.long, device="cuda")
    stats = None
    if cfg.fold_norms and batch <= cfg.fold_norms_max_batch:
        stats = [quant.row_stats_buffer(cfg.hidden, "cuda") for _ in range(2)]
    side = torch.cuda.Stream()
    with torch.no_grad():
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _logits(model, tok, pos_t, stats)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = _logits(model, tok, pos_t, stats)
    return dict(case=case, model=model, graph=graph, keep=(tok, pos_t, stats), logits=logits)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        lin, x = state["lin"], state["x"]
        if case["raw"]:
            return quant.gemm_awq_ut(x, lin.weight, lin.zeros_scales, case["tokens"], case["N"], case["K"], case["g"])
        return lin(x, **state["extra"])
    if kind == "quantize":
        return quant.quantize_pack(state["w"], case["K"], case["N"], case["g"])
    model = state["model"]
    if kind == "prefill":
        model.reset(case["batch"], case["seq"] + 32)
        logits = model(state["ids"])
        return dict(logits=logits, k=[la.k_cache for la in model.layers], v=[la.v_cache for la in model.layers])
    state["graph"].replay()
    return dict(logits=state["logits"], k=[la.k_cache for la in model.layers],
                v=[la.v_cache for la in model.layers])


def _weight_bytes(K, N, g):
    return K * N // 2 + (K // g) * N * 4


def work(case):
    kind = case["kind"]
    if kind == "linear":
        M, K, N = case["tokens"], case["K"], case["N"]
        b = _weight_bytes(K, N, case["g"]) + 2 * M * (K + N * (2 if case["residual"] else 1)) + (2 * N if case["bias"] else 0)
        return dict(bytes=b, flops=2.0 * M * N * K)
    if kind == "quantize":
        K, N = case["K"], case["N"]
        return dict(bytes=4 * K * N + _weight_bytes(K, N, case["g"]), flops=0)      # fp16 in and out, packed out
    H, F, L, B, g = case["hidden"], case["ffn"], case["layers"], case["batch"], case["g"]
    shapes = [(H, 3 * H), (H, H)] + ([(H, F), (F, H)] if case["arch"] == "opt" else [(H, 2 * F), (F, H)])
    weights, macs = sum(_weight_bytes(K, N, g) for K, N in shapes), sum(K * N for K, N in shapes)
    head = case["vocab"] * H
    if kind == "step":
        ctx = case["context"] + 1
        return dict(bytes=L * (weights + 4 * B * ctx * H) + 2 * head + 2 * B * case["vocab"],
                    flops=2.0 * B * (L * (macs + 2 * ctx * H) + head))
    S = case["seq"]
    return dict(bytes=L * (weights + 4 * B * S * H) + 2 * head + 2 * B * case["vocab"] + 2 * B * S * H,
                flops=2.0 * B * (L * (S * macs + S * (S + 1) * H) + head))


def tolerance(case):
    """Four times what the path was seen to differ from itself with the same packed weights dequantised and everything
    after that in fp64 (linears) or fp32 (stacks): linears rel 3.6e-4 and max 2.1e-3 (fp16 outputs, one more fp16
    rounding of each weight or not); OPT-shaped stacks 8.5e-4 and 8.4e-3; LLaMA-shaped ones, whose first RMSNorm divides
    a small embedding up, 3.5e-3 and 5.5e-2 in a token step, 6.9e-3 and 3.3e-2 in a prefill."""
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    if kind == "linear":
        return {"rel": 1.5e-3, "max": 8e-3}
    if case["arch"] == "opt":
        return {"rel": 3.5e-3, "max": 3.5e-2}
    return {"rel": 1.4e-2, "max": 0.22} if kind == "step" else {"rel": 2.8e-2, "max": 0.13}
