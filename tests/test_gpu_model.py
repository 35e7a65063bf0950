"""Tiny OPT- and LLaMA-shaped stacks on the GPU kernels against the same stacks with every quantised
linear replaced by an fp32 matmul on the bit-exact dequantised weight."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense_forward(I, W, ZS, bias, N, g, algo=0, out=None, static_weights=False):
    import quant
    b, s, K = I.shape
    w = quant.dequant(W, ZS, N, K, g).float()
    y = I.reshape(-1, K).float() @ w.t()
    y = y.half()
    if bias is not None:
        y = y + bias.reshape(1, -1)
    return y.reshape(b, s, N)


@pytest.mark.parametrize("kind", ["opt", "llama"])
def test_decoder_logits_match_dense_reference(kind, monkeypatch):
    import w4a16.qlinear as ql
    from w4a16.models import Decoder, DecoderConfig
    if kind == "opt":
        cfg = DecoderConfig("opt", layers=3, hidden=512, heads=8, ffn=2048, vocab=1024, group_size=128, max_positions=128)
    else:
        cfg = DecoderConfig("llama", layers=3, hidden=512, heads=8, ffn=1344, vocab=1024, group_size=64, max_positions=128)
    model = Decoder(cfg, device="cuda", seed=5).mark_static()
    ids = torch.randint(0, cfg.vocab, (4, 40), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    model.reset(4, 48)
    a1 = model(ids).float()                      # prefill: 160 tokens -> tcgen05 kernel
    tok = a1.argmax(-1, keepdim=True)
    a2 = model(tok).float()                      # decode: 4 tokens -> skinny kernel
    monkeypatch.setattr(ql, "gemm_awq_bias", _dense_forward)
    model.reset(4, 48)
    b1 = model(ids).float()
    b2 = model(tok).float()
    for a, b in ((a1, b1), (a2, b2)):
        rel = ((a - b).norm() / b.norm()).item()
        assert rel <= 2e-2, rel
    toks, t_prefill, t_decode = model.generate(ids, 6)
    assert toks.shape == (4, 6) and t_prefill > 0 and t_decode > 0
    # the graph-replayed static-shape decode loop produces the same greedy tokens
    monkeypatch.undo()
    eager, _, _ = model.generate(ids, 6)
    graphed, _, _ = model.generate_graphed(ids, 6, use_graph=True)
    static, _, _ = model.generate_graphed(ids, 6, use_graph=False)
    assert torch.equal(static, graphed)
    assert (eager == graphed).float().mean().item() >= 0.75      # argmax ties may flip between attention variants


@pytest.mark.parametrize("kind", ["opt", "llama"])
def test_token_step_with_folded_normalisations(kind):
    """Five launches per layer (residual adds in the producing GEMVs, normalisations inside the consuming ones, row
    statistics in between) against seven: the hidden state going into the final normalisation agrees, and the folded
    step really launches fewer kernels."""
    import quant
    from w4a16.models import Decoder, DecoderConfig
    if kind == "opt":
        cfg = DecoderConfig("opt", layers=4, hidden=1024, heads=8, ffn=4096, vocab=512, group_size=128, max_positions=64)
    else:
        cfg = DecoderConfig("llama", layers=4, hidden=1024, heads=8, ffn=2752, vocab=512, group_size=64, max_positions=64)
    B = 3
    assert B <= cfg.fold_norms_max_batch
    model = Decoder(cfg, device="cuda", seed=9).mark_static()
    ids = torch.randint(0, cfg.vocab, (B, 12), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    arange = torch.arange(32, device="cuda")
    outs, launches = [], []
    for fold in (False, True):
        cfg.fold_norms = fold
        for layer in model.layers:
            layer.cfg.fold_norms = fold
        model.reset(B, 32)
        tok = model(ids).argmax(-1, keepdim=True)
        pos_t = torch.full((1,), 12, dtype=torch.long, device="cuda")
        n0 = quant.launch_count()
        nxt = model.step_static(tok, pos_t, arange)
        torch.cuda.synchronize()
        launches.append(quant.launch_count() - n0)
        outs.append(nxt)
    assert launches[1] <= launches[0] - 2 * (cfg.layers - 1) - 1     # two launches fewer per layer, one fewer in the first
    assert (outs[0] == outs[1]).float().mean().item() >= 0.66        # greedy tokens of random-weight models: near ties may flip


@pytest.mark.parametrize("kind", ["opt", "llama"])
@pytest.mark.parametrize("B,S", [(3, 40), (2, 150)])                 # epilogues on their own, and inside the linears
def test_prefill_kernels_match_the_torch_ops(kind, B, S):
    """DecoderLayer.forward on the library's kernels against the same layers run op by op in torch around the same
    linears: logits and the filled cache (fp16 rotary arithmetic in torch, one rounding here), then a second chunk behind it."""
    import torch.nn.functional as F
    from w4a16.models import Decoder, DecoderConfig, apply_rope
    from w4a16.tp import split_gate_up
    cfg = DecoderConfig(kind, layers=2, hidden=512, heads=8, ffn=2048 if kind == "opt" else 1344, vocab=512,
                        group_size=128 if kind == "opt" else 64, max_positions=256)
    model = Decoder(cfg, device="cuda", seed=3).mark_static()
    ids = torch.randint(0, cfg.vocab, (B, S), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))

    def plain(layer, x, pos0, rope):
        q, k, v = (t.view(B, -1, 8, 64).transpose(1, 2) for t in layer.qkv_proj(layer.ln1(x)).split(512, dim=-1))
        n = x.shape[1]
        if rope is not None:
            q, k = apply_rope(q, *rope), apply_rope(k, *rope)
        layer.k_cache[:, :, pos0:pos0 + n], layer.v_cache[:, :, pos0:pos0 + n] = k, v
        a = F.scaled_dot_product_attention(q, layer.k_cache[:, :, :pos0 + n], layer.v_cache[:, :, :pos0 + n], is_causal=n > 1 and pos0 == 0)
        x = x + layer.out_proj(a.transpose(1, 2).reshape(B, n, 512))
        h = layer.ln2(x)
        if kind == "opt":
            return x + layer.fc2(torch.relu(layer.fc1(h)))
        gate, up = split_gate_up(layer.gate_up_proj(h))
        return x + layer.fc2(F.silu(gate) * up)

    got = []
    for fused in (True, False):
        model.reset(B, S + 1)
        if not fused:
            for layer in model.layers:
                layer.forward = lambda x, pos0, rope, layer=layer: plain(layer, x, pos0, rope)
        logits = model(ids)
        nxt = model(ids[:, :1])
        got.append([logits, nxt] + [t for la in model.layers for t in (la.k_cache, la.v_cache)])
    for a, b in zip(*got):
        rel = ((a.float() - b.float()).norm() / b.float().norm()).item()
        assert rel <= 1e-2, rel                                    # fp16 stacks: one rounding in a layer travels through the rest


def _small(kind, **kw):
    from w4a16.models import Decoder, DecoderConfig
    cfg = DecoderConfig(kind, layers=2, hidden=256, heads=4, ffn=512, vocab=320, group_size=64, max_positions=512, **kw)
    return Decoder(cfg, device="cuda", seed=5).mark_static()


def _ids(model, B, S):
    return torch.randint(0, model.cfg.vocab, (B, S), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))


@pytest.mark.parametrize("kind", ["opt", "llama"])
@pytest.mark.parametrize("S", [40, 300])
def test_prompt_modules_that_are_watched_or_replaced_are_called(kind, S):
    """Decoder.forward reads its normalisations' parameters and hands epilogues to its linears; hooks on them, and modules
    of another class in their place, have to see what the layer written op by op shows them."""
    from w4a16.models import RMSNorm
    model = _small(kind)
    ids = _ids(model, 1, S)

    def logits():
        model.reset(1, S + 1)
        return model(ids).float()

    plain = logits()
    for pick in ("ln1", "ln2", "out_proj", "fc2", "fc1" if kind == "opt" else "gate_up_proj", "qkv_proj", None):
        module = model.final_norm if pick is None else getattr(model.layers[1], pick)
        seen = []
        handle = module.register_forward_hook(lambda m, args, out: seen.append((args[0].detach().clone(), out.detach().clone())))
        got = logits()
        handle.remove()
        assert len(seen) == 1 and ((got - plain).norm() / plain.norm()).item() <= 1e-2, pick
        x, y = seen[0]
        if "norm" in type(module).__name__.lower():
            assert ((module(x) - y).abs().max() <= 1e-2 * y.abs().max())
        else:
            again = module(x)                                       # the linear alone: no residual, no ReLU in what the hook saw
            assert torch.equal(again, y), pick

    class Doubled(type(model.layers[0].ln1)):
        def forward(self, x):
            return 2 * super().forward(x)

    for where, name in ((model.layers[0], "ln2"), (model, "final_norm")):
        old = getattr(where, name)
        new = Doubled(256, old.eps, "cuda") if isinstance(old, RMSNorm) else Doubled(256, device="cuda", dtype=torch.float16)
        setattr(where, name, new)
        got = logits()
        setattr(where, name, old)
        assert ((got - plain).norm() / plain.norm()).item() > 0.05, name
        if name == "final_norm":
            assert ((got - 2 * plain).norm() / plain.norm()).item() <= 2e-2


def test_prompt_layer_keeps_the_gradient_of_its_residual_stream():
    model = _small("opt")
    model.reset(1, 300)
    x = torch.randn(1, 300, 256, device="cuda").half().requires_grad_()
    y = model.layers[0](x, 0)
    assert y.requires_grad


@pytest.mark.parametrize("kind", ["opt", "llama"])
@pytest.mark.parametrize("B", [8, 24, 40])
def test_token_step_without_folded_norms(kind, B):
    """One token step (static position, attention kernel, residual of fc2 in the epilogue, SwiGLU in the epilogue or on
    alternating tiles beyond 32 sequences) against the same layers written op by op in torch around the same linears."""
    import torch.nn.functional as F
    from w4a16.models import apply_rope
    from w4a16.tp import split_gate_up
    pos, D = 9, 64
    model = _small(kind)
    model.reset(B, 16)
    g = torch.Generator(device="cuda").manual_seed(4)
    for la in model.layers:
        la.k_cache[:, :, :pos].normal_(generator=g)
        la.v_cache[:, :, :pos].normal_(generator=g)
    saved = [(la.k_cache.clone(), la.v_cache.clone()) for la in model.layers]
    x0 = torch.randn(B, 1, 256, device="cuda", generator=g).half()
    pos_t = torch.full((1,), pos, dtype=torch.long, device="cuda")
    x = x0
    with torch.no_grad():
        for la in model.layers:
            x = la.forward_static(x, pos_t, None if kind == "opt" else (model.rope_cos, model.rope_sin))
        y = x0
        for la, (k, v) in zip(model.layers, saved):
            q, kn, vn = (t.view(B, 1, 4, D).transpose(1, 2) for t in la.qkv_proj(la.ln1(y)).split(256, dim=-1))
            if kind == "llama":
                cos, sin = model.rope_cos[pos:pos + 1], model.rope_sin[pos:pos + 1]
                q, kn = apply_rope(q, cos, sin), apply_rope(kn, cos, sin)
            k[:, :, pos:pos + 1], v[:, :, pos:pos + 1] = kn, vn
            a = F.scaled_dot_product_attention(q, k[:, :, :pos + 1], v[:, :, :pos + 1]).transpose(1, 2).reshape(B, 1, 256)
            y = y + la.out_proj(a)
            h = la.ln2(y)
            if kind == "opt":
                y = y + la.fc2(torch.relu(la.fc1(h.reshape(1, B, 256)))).reshape(B, 1, 256)
            else:
                gate, up = split_gate_up(la.gate_up_proj(h))
                y = y + la.fc2(F.silu(gate) * up)
    assert ((x.float() - y.float()).norm() / y.float().norm()).item() <= 1e-2      # fp16 layers: roundings travel through the rest
    for la, (k, v) in zip(model.layers, saved):
        assert ((la.k_cache.float() - k.float()).norm() / k.float().norm()).item() <= 1e-2
        assert ((la.v_cache.float() - v.float()).norm() / v.float().norm()).item() <= 1e-2


@pytest.mark.parametrize("kind", ["opt", "llama"])
def test_token_step_hands_no_residual_to_an_fc2_that_is_watched_or_replaced(kind):
    model = _small(kind)
    B, pos_t = 8, torch.full((1,), 3, dtype=torch.long, device="cuda")
    x = torch.randn(B, 1, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).half()
    la = model.layers[0]

    def step():
        model.reset(B, 16)
        with torch.no_grad():
            return la.forward_static(x, pos_t, None if kind == "opt" else (model.rope_cos, model.rope_sin)).float()

    plain, seen = step(), []
    handle = la.fc2.register_forward_hook(lambda m, args, out: seen.append((args[0].clone(), out.clone())))
    assert ((step() - plain).norm() / plain.norm()).item() <= 1e-3
    handle.remove()
    assert torch.equal(la.fc2(seen[0][0]), seen[0][1])

    class Nothing(torch.nn.Module):
        def forward(self, f):
            return torch.zeros(f.shape[:-1] + (256,), dtype=f.dtype, device=f.device)

    la.fc2 = Nothing()
    assert not torch.equal(step(), plain)
