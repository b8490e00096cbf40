"""Performance cases: what programs that use this framework spend their time on, on one GPU, through the entry points such programs call.

* ``train``: forward and backward of a decoder (``DeepSeekTransformer.forward_loss``), all weight gradients;
* ``moe``: forward and backward of one routed feed-forward (``MoEFFNLayer``).  It is measured by itself because a whole model re-routes
  tokens whenever an earlier layer rounds differently, and outputs could then not be compared;
* ``moe_step``: the same layer in a decode step, replayed from a CUDA graph as the serving engine does;
* ``decode``: one decode step of a decoder through ``GenerationEngine.graph_decoder``, bf16 or 4-bit weights;
* ``prefill`` / ``step``: a prompt (``GenerationEngine.prefill``) and one decode step of the layer-listed designs.

Sizes are those of the presets (``dense_1b``, ``b1_moe``, ``mixtral_8x7b``, ``hybrid_fp8``) and of the design benchmark, with fewer layers
where layers only repeat each other.  Weights are random with the initialisation of the presets, token ids uniform.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

VOCAB = 32000


def listed():
    return [
        # pre-training step of the 1.1 B dense preset: 8 sequences of 2,048 tokens, 64-wide heads
        dict(name="train_dense", kind="train", width=2048, heads=32, kv_heads=4, ff=5632, layers=4, batch=8, seq=2048),
        # one long sequence through a wider model with 128-wide heads (the attention of the Mixtral-shaped preset)
        dict(name="train_wide", kind="train", width=4096, heads=32, kv_heads=8, ff=11008, layers=1, batch=1, seq=4096),
        # fine-tuning a small model on a short batch whose length is no multiple of any tile
        dict(name="train_ragged", kind="train", width=1024, heads=16, kv_heads=4, ff=2816, layers=4, batch=3, seq=1000),
        # routed layer of the headline training configuration at its micro-batch
        dict(name="moe_8_experts", kind="moe", width=2048, ff=5632, experts=8, top_k=2, tokens=16384),
        # fine-grained experts of the hybrid preset, token count no multiple of a tile
        dict(name="moe_16_experts", kind="moe", width=2048, ff=1408, experts=16, top_k=2, tokens=3000),
        # serving batch of 64 on the Mixtral shape: every expert weight is read for a handful of rows
        dict(name="moe_step", kind="moe_step", width=4096, ff=14336, experts=8, top_k=2, tokens=64),
        # interactive generation, one sequence: latency of the weights' stream and of the launches
        dict(name="decode_1", kind="decode", width=2048, heads=32, kv_heads=4, ff=5632, layers=8, batch=1, context=512, bits=16),
        # serving batch of the decode benchmark on the same model
        dict(name="decode_64", kind="decode", width=2048, heads=32, kv_heads=4, ff=5632, layers=8, batch=64, context=1024, bits=16),
        # a few sequences on 4-bit weights
        dict(name="decode_int4", kind="decode", width=2048, heads=32, kv_heads=4, ff=5632, layers=8, batch=4, context=300, bits=4),
        # prompts of the design benchmark: sliding-window latent attention and the gated delta rule
        dict(name="prefill_vimodra", kind="prefill", design="vimodra", width=2048, heads=16, ff=8192, batch=8, seq=2048),
        # prompts of odd length: lightning attention, capped attention, channel-wise delta rule
        dict(name="prefill_nemipel", kind="prefill", design="nemipel", width=2048, heads=16, ff=5504, batch=3, seq=1501),
        # one decode step of a serving batch with recurrent states
        dict(name="step_nemipel", kind="step", design="nemipel", width=2048, heads=16, ff=5504, batch=64, context=256),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["train", "train", "moe", "moe_step", "decode", "decode", "prefill", "prefill", "step"])
    if kind == "train":
        d, heads = rng.choice([(64, 8), (64, 12), (64, 16), (64, 32), (128, 8), (128, 16)])
        width = d * heads
        seq = rng.choice([256, 512, 1024, 2048, log(100, 2048)])
        tokens = log(seq, 12000)
        return dict(kind=kind, width=width, heads=heads, kv_heads=heads // rng.choice([1, 2, 4]), ff=128 * rng.randint(width // 64, width * 11 // 512),
                    layers=rng.randint(1, 4), batch=max(1, tokens // seq), seq=seq)
    if kind == "moe":
        E, ff = rng.choice([(8, 5632), (8, 2816), (16, 1408)])
        return dict(kind=kind, width=rng.choice([1024, 2048]), ff=ff, experts=E, top_k=rng.choice([1, 2]), tokens=log(300, 14000))
    if kind == "moe_step":
        return dict(kind=kind, width=rng.choice([2048, 4096]), ff=rng.choice([5632, 14336]), experts=8, top_k=2, tokens=log(1, 128))
    if kind == "decode":
        width, heads, ff = rng.choice([(1024, 16, 2816), (2048, 32, 5632), (2048, 16, 5504)])
        bits = rng.choice([16, 16, 4])
        return dict(kind=kind, width=width, heads=heads, kv_heads=heads // rng.choice([2, 4, 8]), ff=ff, layers=rng.randint(2, 8), batch=log(1, 64), context=log(30, 1500),
                    bits=bits)
    design = rng.choice(["vimodra", "nemipel"])
    width, heads = rng.choice([(1024, 8), (2048, 16)])
    ff = 4 * width if design == "vimodra" else width * 43 // 16
    if kind == "prefill":
        seq = rng.choice([512, 1024, 2048, log(60, 2000)])
        return dict(kind=kind, design=design, width=width, heads=heads, ff=ff, batch=max(1, log(seq, 12000) // seq), seq=seq)
    return dict(kind=kind, design=design, width=width, heads=heads, ff=ff, batch=log(1, 64), context=log(30, 1500))


# ------------------------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _normal(g, *shape, std=1.0, mean=0.0):
    return (torch.randn(*shape, generator=g, device=g.device) * std + mean).to(torch.bfloat16)


def _ids(g, batch, n):
    return torch.randint(0, VOCAB, (batch, n), generator=g, device=g.device)


def _dense_weights(c, g):
    """In the order and with the shapes of ``DeepSeekTransformer.named_parameters``, N(0, 0.02) matrices and norms of one."""
    D, d = c["width"], c["width"] // c["heads"]
    w = {"embed_tokens.weight": _normal(g, VOCAB, D, std=0.02), "lm_head_weight": _normal(g, VOCAB, D, std=0.02), "norm.weight": _normal(g, D, std=0.0, mean=1.0)}
    for i in range(c["layers"]):
        p = f"layers.{i}."
        w[p + "input_norm.weight"] = _normal(g, D, std=0.1, mean=1.0)
        w[p + "post_attn_norm.weight"] = _normal(g, D, std=0.1, mean=1.0)
        w[p + "self_attn.qkv_proj"] = _normal(g, (c["heads"] + 2 * c["kv_heads"]) * d, D, std=0.02)
        w[p + "self_attn.o_proj"] = _normal(g, D, D, std=0.02)
        w[p + "ffn.gate_up_proj"] = _normal(g, 2 * c["ff"], D, std=0.02)
        w[p + "ffn.down_proj"] = _normal(g, D, c["ff"], std=0.02)
    return w


def _dense_model(c, weights, seq):
    from adaptivetrainingsystem_b200.config import ModelConfig
    from adaptivetrainingsystem_b200.models import DeepSeekTransformer
    cfg = ModelConfig(vocab_size=VOCAB, hidden_size=c["width"], num_layers=c["layers"], num_heads=c["heads"], num_kv_heads=c["kv_heads"], intermediate_size=c["ff"],
                      seq_length=seq, tie_word_embeddings=False)
    with torch.device("meta"):
        model = DeepSeekTransformer(cfg)
    for name, p in list(model.named_parameters()):
        owner = model
        for part in name.split(".")[:-1]:
            owner = getattr(owner, part)
        setattr(owner, name.split(".")[-1], torch.nn.Parameter(weights[name]))
    model.rope = type(model.rope)(cfg.head_dim, seq, cfg.rope_theta).to(_device())
    return model


def _moe_inputs(c, seed):
    g = _generator(seed)
    D, I, E, T = c["width"], c["ff"], c["experts"], c["tokens"]
    return dict(x=_normal(g, T, D), dy=_normal(g, T, D, std=0.01), gate=_normal(g, E, D, std=0.02), w1=_normal(g, E, 2 * I, D, std=0.02), w2=_normal(g, E, D, I, std=0.02))


def _moe_layer(c, t):
    from adaptivetrainingsystem_b200.config import ModelConfig
    from adaptivetrainingsystem_b200.models.transformer import MoEFFNLayer
    cfg = ModelConfig(vocab_size=VOCAB, hidden_size=c["width"], num_layers=1, num_heads=16, num_kv_heads=4, intermediate_size=c["ff"], use_moe=True,
                      num_experts=c["experts"], moe_top_k=c["top_k"], capacity_factor=1.25, load_balancing_weight=0.01)
    with torch.device("meta"):
        layer = MoEFFNLayer(cfg, 0)
    layer = layer.to_empty(device=_device())
    layer.gate.weight = torch.nn.Parameter(t["gate"])
    for name, w in (("experts_w1", t["w1"]), ("experts_w2", t["w2"])):
        setattr(layer, name, torch.nn.Parameter(w))
        getattr(layer, name)._ats_expert = True
    for b in layer.buffers():
        b.zero_()
    return layer


def _design(c):
    """config.json of a four-layer model with the proportions of the design benchmark."""
    H, dim = c["heads"], 128
    vimodra = c["design"] == "vimodra"
    mlp = {"kind": "dense", "ff": c["ff"]}

    def layer(kind, **mixer):
        return {"type": kind, "mlp": mlp, "mixer": mixer}
    rec = layer("delta" if vimodra else "channel_delta", heads=H, kv_heads=H // 2, dim=dim, vdim=dim, conv=4)
    if vimodra:
        att = layer("latent_attention", heads=H, dim=dim, rot_dim=64, vdim=dim, kv_rank=512, q_rank=768, mask={"size": 1024}, rot={"base": 10000.0, "dims": 64},
                    scale=192 ** -0.5)
        return {"vocab": VOCAB, "width": c["width"], "norm": {"eps": 1e-5}, "layers": [att, att, att, rec]}

    def att(**kw):
        return layer("attention", heads=H, kv_heads=H // 4, dim=dim, vdim=dim, rot={"base": 10000.0, "dims": 64}, scale=128 ** -0.5, softcap=25.0, **kw)
    light = layer("lightning", heads=H, dim=dim, vdim=dim, decay=[1.0 - 2.0 ** (-1 - 8.0 * i / H) for i in range(H)])
    return {"vocab": VOCAB, "width": c["width"], "norm": {"eps": 1e-6}, "postln_alpha": 2.0, "logit_softcap": 20.0, "layers": [light, att(), rec, att(kv_from=1)]}


def _design_weights(c, g):
    cfg = _design(c)
    D, w = c["width"], {}

    def mat(name, n, k, s=1.0):
        w[name] = _normal(g, n, k, std=s / math.sqrt(k))

    def vec(name, n, mean, std):
        w[name] = _normal(g, n, mean=mean, std=std)

    def dyt(name):
        vec(name, D, 1.0, 0.1), vec(name + ".b", D, 0.0, 0.1)
        w[name + ".alpha"] = torch.tensor(0.5, device=g.device)
    vimodra = c["design"] == "vimodra"
    w["embed"] = _normal(g, VOCAB, D)
    mat("head", VOCAB, D)
    if vimodra:
        dyt("final.norm")
    else:
        vec("final.norm", D, 1.0, 0.1)
    for i, L in enumerate(cfg["layers"]):
        p, q, m = f"l{i}.", f"l{i}.mix.", L["mixer"]
        H, d, vd = m["heads"], m["dim"], m["vdim"]
        if vimodra:
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                dyt(p + n)
            vec(p + "ls1", D, 1.0, 0.1), vec(p + "ls2", D, 1.0, 0.1)
            mat(p + "mlp.up", c["ff"], D), vec(p + "mlp.up.b", c["ff"], 0.0, 0.1)
            mat(p + "mlp.down", D, c["ff"]), vec(p + "mlp.down.b", D, 0.0, 0.1)
        else:
            vec(p + "norm1", D, 1.0, 0.1), vec(p + "norm2", D, 1.0, 0.1)
            mat(p + "mlp.gate", c["ff"], D), mat(p + "mlp.up", c["ff"], D), mat(p + "mlp.down", D, c["ff"])
        if L["type"] == "latent_attention":
            mat(q + "dq", m["q_rank"], D), vec(q + "dq.norm", m["q_rank"], 1.0, 0.1), mat(q + "uq", H * (d + m["rot_dim"]), m["q_rank"])
            mat(q + "dkv", m["kv_rank"] + m["rot_dim"], D), vec(q + "dkv.norm", m["kv_rank"], 1.0, 0.1)
            mat(q + "uk", H * d, m["kv_rank"]), mat(q + "uv", H * vd, m["kv_rank"]), mat(q + "g", H * vd, D), mat(q + "o", D, H * vd)
        elif L["type"] == "lightning":
            mat(q + "q", H * d, D), mat(q + "k", H * d, D), mat(q + "v", H * vd, D), mat(q + "g", H * vd, D), mat(q + "o", D, H * vd), vec(q + "norm", H * vd, 1.0, 0.1)
        elif L["type"] == "attention":
            G = m["kv_heads"]
            mat(q + "q", H * d, D), vec(q + "q.norm", H * d, 1.0, 0.1), mat(q + "g", H, D), mat(q + "o", D, H * vd)
            if "kv_from" not in m:
                mat(q + "k", G * d, D), vec(q + "k.norm", G * d, 1.0, 0.1), mat(q + "v", G * vd, D)
        else:
            KH = m["kv_heads"]
            for n, rows in (("q", KH * d), ("k", KH * d), ("v", H * vd)):
                mat(q + n, rows, D)
                w[q + n + ".conv"] = _normal(g, rows, m["conv"], std=0.5)
            mat(q + "b", H, D), vec(q + "A_log", H, 0.0, 0.5), vec(q + "norm", vd, 1.0, 0.1), mat(q + "o", D, H * vd)
            if vimodra:
                mat(q + "a", H, D), vec(q + "dt_bias", H, -2.0, 0.5), mat(q + "g", H * vd, D)
            else:
                mat(q + "a1", d, D), mat(q + "a2", H * d, d), vec(q + "dt_bias", H * d, -2.0, 0.5), mat(q + "g1", vd, D), mat(q + "g2", H * vd, vd)
    return w


def _design_model(c, w):
    from adaptivetrainingsystem_b200.config import NemipelConfig, VimodraConfig
    from adaptivetrainingsystem_b200.models import Nemipel, Vimodra
    conf, cls = (VimodraConfig, Vimodra) if c["design"] == "vimodra" else (NemipelConfig, Nemipel)
    return cls.from_tensors(conf.from_dict(_design(c)), w.__getitem__, list(w), torch.bfloat16, _device())


# ------------------------------------------------------------------------------------------------------------------------------------
# the passes
# ------------------------------------------------------------------------------------------------------------------------------------
NEW_TOKENS = 256   # a generation continues this far behind its prompt, then the row starts again behind the same prompt


def prepare(case, seed):
    from adaptivetrainingsystem_b200.inference.engine import GenerationEngine
    from adaptivetrainingsystem_b200.ops import int4
    c, g = case, _generator(seed)
    kind = c["kind"]
    if c.get("bits") != 4:
        int4.set_enabled(False)
        int4.clear()
    if kind == "train":
        model = _dense_model(c, _dense_weights(c, g), c["seq"]).train()
        ids = _ids(g, c["batch"], c["seq"] + 1)
        return dict(kind=kind, model=model, ids=ids[:, :-1].contiguous(), labels=ids[:, 1:].contiguous())
    if kind in ("moe", "moe_step"):
        t = _moe_inputs(c, seed)
        layer = _moe_layer(c, t)
        if kind == "moe":
            return dict(kind=kind, layer=layer.train(), x=t["x"].requires_grad_(True), dy=t["dy"])
        layer.eval().requires_grad_(False)
        x, side = t["x"], torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side), torch.no_grad():
            layer(x, x)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph), torch.no_grad():
            out = layer(x, x)[0]
        return dict(kind=kind, layer=layer, x=x, graph=graph, out=out)
    if kind == "decode":
        total = c["context"] + NEW_TOKENS
        model = _dense_model(c, _dense_weights(c, g), total).eval().requires_grad_(False)
        ids = _ids(g, c["batch"], c["context"] + 1)
        if c["bits"] == 4:
            from types import SimpleNamespace
            from adaptivetrainingsystem_b200.training.precision import QuantizationManager
            QuantizationManager(SimpleNamespace(quantization_method="int4", quantization_bits=4)).quantize_model(model)
    else:
        model = _design_model(c, _design_weights(c, g))
        if kind == "prefill":
            ids = _ids(g, c["batch"], c["seq"])
            return dict(kind=kind, engine=GenerationEngine(model), ids=ids, cache=model.make_cache(c["batch"], c["seq"] + NEW_TOKENS))
        total = c["context"] + NEW_TOKENS
        ids = _ids(g, c["batch"], c["context"] + 1)
    engine = GenerationEngine(model, max_len=total)
    cache = model.make_cache(c["batch"], total)
    engine.prefill(ids[:, :-1].contiguous(), cache)
    return dict(kind=kind, engine=engine, cache=cache, decoder=engine.graph_decoder(cache), tokens=ids[:, -1].contiguous(), context=c["context"])


def _states(cache):
    seen, out = set(), []
    for st in cache.states:
        for k in sorted(st):
            if st[k].data_ptr() not in seen:
                seen.add(st[k].data_ptr())
                out.append(st[k])
    return out


def run(state):
    s, kind = state, state["kind"]
    if kind == "train":
        model = s["model"]
        model.zero_grad(set_to_none=True)
        loss = model.forward_loss(s["ids"], s["labels"])["loss"]
        loss.backward()
        return {"loss": loss.detach(), "grads": {n: p.grad for n, p in model.named_parameters()}}
    if kind == "moe":
        layer, x = s["layer"], s["x"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        out, aux = layer(x)
        torch.autograd.backward([out, aux], [s["dy"], None])
        return {"out": out.detach(), "aux": aux.detach(), "dx": x.grad, "dgate": layer.gate.weight.grad, "dw1": layer.experts_w1.grad, "dw2": layer.experts_w2.grad}
    if kind == "moe_step":
        s["graph"].replay()
        return s["out"]
    cache = s["cache"]
    if kind == "prefill":
        cache.reset()
        return {"logits": s["engine"].prefill(s["ids"], cache), "states": _states(cache)}
    if cache.length + 1 > cache.max_len:   # the generation is at its end: the next one starts behind the same prompt
        cache.length = s["context"]
        cache.device_lengths.fill_(s["context"])
        cache.device_positions.fill_(s["context"])
    logits = s["decoder"].step(s["tokens"])
    return logits if kind == "decode" else {"logits": logits, "states": [st["S"] for st in cache.states if "S" in st]}


# ------------------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    D = c["width"]
    if kind in ("moe", "moe_step"):
        E, I, T, k = c["experts"], c["ff"], c["tokens"], c["top_k"]
        weights, per_row = 3 * E * I * D + E * D, 2 * 3 * I * D
        if kind == "moe":
            return {"bytes": 2 * (2 * weights + 5 * T * D), "flops": 3 * T * k * per_row}
        return {"bytes": 2 * (weights * (1 - (1 - 1 / E) ** (T * k)) + 3 * T * D), "flops": T * k * per_row}
    if kind in ("train", "decode"):
        d, ff, n = D // c["heads"], c["ff"], c["layers"]
        proj = D * (c["heads"] + 2 * c["kv_heads"]) * d + D * D
        layer, head = proj + 3 * ff * D, VOCAB * D
        if kind == "train":
            T = c["batch"] * c["seq"]
            attention = 2 * c["batch"] * c["heads"] * d * c["seq"] ** 2   # causal scores and values
            return {"bytes": 2 * 2 * (n * layer + 2 * head) + 16 * T, "flops": 6 * T * (n * layer + head) + n * attention * 3.5}
        B, ctx = c["batch"], c["context"] + NEW_TOKENS // 2
        kv = n * B * 2 * ctx * c["kv_heads"] * d * 2
        return {"bytes": n * layer * (c["bits"] / 8 + (0.03125 if c["bits"] == 4 else 0)) + 2 * head + kv + 2 * B * VOCAB,
                "flops": 2 * B * (n * layer + head) + n * B * 4 * c["heads"] * d * ctx}
    B, H, d = c["batch"], c["heads"], 128
    vimodra = c["design"] == "vimodra"
    L = c["seq"] if kind == "prefill" else 1
    seen = c["seq"] / 2 if kind == "prefill" else c["context"] + NEW_TOKENS / 2
    weights, flops, state = 0.0, 0.0, 0.0
    for layer in _design(c)["layers"]:
        m, t = layer["mixer"], layer["type"]
        w = (2 if vimodra else 3) * D * c["ff"] + D * H * d
        if t == "latent_attention":
            own = D * (768 + 576 + H * d) + 768 * H * 192 + 512 * H * 256
            n = min(seen, 1024)
            flops += 2 * B * L * H * n * (192 + 128 if kind == "prefill" else 576 + 512)
            state += B * 2 * 576 * (min(1024, c["seq"]) if kind == "prefill" else min(1024, seen))
        elif t == "attention":
            own = D * (H * d + H + (0 if "kv_from" in m else 2 * (H // 4) * d))
            flops += 4 * B * L * H * d * seen
            state += B * 2 * 2 * (H // 4) * d * ((c["seq"] if "kv_from" not in m else 0) if kind == "prefill" else seen)
        else:
            own = D * H * d * 4 if t == "lightning" else D * d * (2 * (H // 2) + (2 if vimodra else 1) * H + (0 if vimodra else 2)) + (0 if vimodra else 2 * H * d * d)
            flops += B * L * H * d * d * (4 if t == "lightning" else 6)
            state += B * H * d * d * 4 * (1 if kind == "prefill" else 2)
        weights += w + own
    head = VOCAB * D
    return {"bytes": 2 * (weights + head) + state + 2 * B * L * D + 4 * B * VOCAB, "flops": 2 * B * L * weights + 2 * B * head + flops}


# Activations between products are bf16.  A pass is this far from its 64-bit values: train 0.004 (one layer) to 0.012 (four), moe 0.0045,
# moe_step 0.0035, decode 0.007 (two layers) to 0.013 (eight), prefill and step 0.005; two correct passes are further apart by a square root of two.
def tolerance(case):
    return {"train": {"rel": 0.02, "max": 0.6}, "moe": {"rel": 0.012, "max": 0.3}, "moe_step": {"rel": 0.012, "max": 0.3}, "decode": {"rel": 0.025, "max": 0.6},
            "prefill": {"rel": 0.02, "max": 0.8}, "step": {"rel": 0.02, "max": 0.8}}[case["kind"]]


# ------------------------------------------------------------------------------------------------------------------------------------
# the same passes in 64 bits
# ------------------------------------------------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(n, dims, base):
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=_device()) / dims)
    a = torch.arange(n, dtype=torch.float64, device=_device())[:, None] * f
    return torch.cos(a)[:, None], torch.sin(a)[:, None]     # [n, 1, dims / 2]


def _rotate_half(x, base=10000.0):
    """x [.., n, heads, dims]: dimension i turns with i + dims / 2."""
    c, s = _angles(x.shape[-3], x.shape[-1], base)
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _rotate_pairs(x, dims, base):
    """The first ``dims`` dimensions of x [.., n, heads, dim]: 2i turns with 2i + 1."""
    c, s = _angles(x.shape[-3], dims, base)
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)


def _attend(q, k, v, scale, cap=0.0, window=0):
    """q [B, n, H, d], k, v [B, n, G, .], causal -> [B, n, H, .]; one sequence and key head at a time."""
    B, n, H, _ = q.shape
    G = k.shape[2]
    at = torch.arange(n, device=q.device)
    gap = at[:, None] - at[None, :]
    hidden = (gap < 0) if not window else (gap < 0) | (gap >= window)

    def head(qh, kh, vh):      # [n, r, d], [n, d], [n, .]
        s = torch.einsum("nrd,md->rnm", qh, kh) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        return torch.einsum("rnm,mv->nrv", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), vh)
    r = H // G
    out = [torch.stack([checkpoint(head, q[b, :, g * r:(g + 1) * r], k[b, :, g], v[b, :, g], use_reentrant=False) for g in range(G)], 1) for b in range(B)]
    return torch.stack(out).flatten(2, 3)


def _dense_block(x, w, p, c):
    B, n, D = x.shape
    H, G, d = c["heads"], c["kv_heads"], D // c["heads"]
    qkv = (_rms(x, 1e-6) * w[p + "input_norm.weight"]) @ w[p + "self_attn.qkv_proj"].T
    q, k, v = qkv.view(B, n, H + 2 * G, d).split([H, G, G], 2)
    a = _attend(_rotate_half(q), _rotate_half(k), v, d ** -0.5)
    x = x + a.reshape(B, n, D) @ w[p + "self_attn.o_proj"].T
    g, u = ((_rms(x, 1e-6) * w[p + "post_attn_norm.weight"]) @ w[p + "ffn.gate_up_proj"].T).chunk(2, -1)
    return x + (F.silu(g) * u) @ w[p + "ffn.down_proj"].T


def _dense_exact(c, w, ids):
    """-> normalised hidden states."""
    x = w["embed_tokens.weight"][ids] * math.sqrt(c["width"])
    for i in range(c["layers"]):
        x = checkpoint(_dense_block, x, w, f"layers.{i}.", c, use_reentrant=False)
    return _rms(x, 1e-6) * w["norm.weight"]


def _four_bits(w):
    """Groups of 128 inputs, 16 levels over the group's range around zero, bf16 scales, round to nearest."""
    t = w.float().view(w.shape[0], -1, 128)
    lo, hi = t.amin(-1, keepdim=True).clamp(max=0), t.amax(-1, keepdim=True).clamp(min=0)
    scale = ((hi - lo) / 15).clamp(min=1e-8).bfloat16().float()
    zero = torch.round(-lo / scale).clamp(0, 15)
    return (((torch.round(t / scale) + zero).clamp(0, 15) - zero).double() * scale.double()).view(w.shape)


def _moe_exact(c, t):
    t = {k: v.double().requires_grad_(c["kind"] == "moe" and k != "dy") for k, v in t.items()}
    T, E, k = c["tokens"], c["experts"], c["top_k"]
    x = t["x"]
    p = torch.softmax(x @ t["gate"].T, -1)
    weight, chosen = p.topk(k, -1)
    weight = weight / weight.sum(-1, keepdim=True)
    hit = F.one_hot(chosen.reshape(-1), E)
    rank = ((hit.cumsum(0) - hit) * hit).sum(-1).view(T, k)      # how many earlier slots the expert has had
    room = -(-math.ceil(1.25 * k * T / E) // 128) * 128 if c["kind"] == "moe" else T
    out = torch.zeros_like(x)
    for e in range(E):
        tok, slot = ((chosen == e) & (rank < room)).nonzero(as_tuple=True)
        g, u = (x[tok] @ t["w1"][e].T).chunk(2, -1)
        out = out.index_add(0, tok, ((F.silu(g) * u) @ t["w2"][e].T) * weight[tok, slot][:, None])
    if c["kind"] == "moe_step":
        return (out + x).detach()
    aux = 0.01 * E * (hit.double().mean(0) * p.mean(0)).sum()
    torch.autograd.backward([out, aux], [t["dy"], torch.ones_like(aux)])
    return {"out": out.detach(), "aux": aux.detach(), "dx": x.grad, "dgate": t["gate"].grad, "dw1": t["w1"].grad, "dw2": t["w2"].grad}


def _conv(x, w):
    """x [B, n, channels], w [channels, taps]: causal, the last tap weighs the current token; silu."""
    taps = w.shape[1]
    full = F.pad(x, (0, 0, taps - 1, 0))
    return F.silu(sum(full[:, j:j + x.shape[1]] * w[:, j] for j in range(taps)))


def _recur(q, k, v, decay, beta=None):
    """q, k [B, n, H, d], v [B, n, H, vd], decay [B, n, H, d or 1]; with ``beta`` the delta rule, else plain linear attention -> outputs, state."""
    B, n, H, d = q.shape
    S = torch.zeros(B, H, d, v.shape[-1], dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(n):
        S = S * decay[:, t, :, :, None]
        u = v[:, t] if beta is None else beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
    return out, S


def _delta_exact(w, p, m, h, eps, channel):
    B, n, _ = h.shape
    H, KH, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_conv(h @ w[p + s].T, w[p + s + ".conv"]).view(B, n, -1, x) for s, x in (("q", d), ("k", d), ("v", vd)))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = ((x * f).repeat_interleave(H // KH, 2) for x, f in ((q, d ** -0.5), (k, 1.0)))
    a = (h @ w[p + "a1"].T) @ w[p + "a2"].T if channel else h @ w[p + "a"].T
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * F.softplus(a + w[p + "dt_bias"]).view(B, n, H, -1))
    o, S = _recur(q, k, v, decay, torch.sigmoid(h @ w[p + "b"].T))
    gate = torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T) if channel else F.silu(h @ w[p + "g"].T)
    return ((_rms(o, eps) * w[p + "norm"]).flatten(2) * gate) @ w[p + "o"].T, S


def _vimodra_exact(c, w, ids):
    cfg = _design(c)
    eps, states = cfg["norm"]["eps"], []

    def norm(x, name):
        return torch.tanh(x * w[name + ".alpha"]) * w[name] + w[name + ".b"]
    x = w["embed"][ids]
    B, n, _ = x.shape
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        h, q_ = norm(x, p + "norm1"), p + "mix."
        if L["type"] == "delta":
            y, S = _delta_exact(w, q_, m, h, eps, False)
            states += [S, None]
        else:
            H, d, rd, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            q = ((_rms(h @ w[q_ + "dq"].T, eps) * w[q_ + "dq.norm"]) @ w[q_ + "uq"].T).view(B, n, H, d + rd)
            ckv = h @ w[q_ + "dkv"].T
            lat = _rms(ckv[..., :rank], eps) * w[q_ + "dkv.norm"]
            kr = _rotate_half(ckv[:, :, None, rank:]).expand(B, n, H, rd)
            k = torch.cat([(lat @ w[q_ + "uk"].T).view(B, n, H, d), kr], -1)
            q = torch.cat([q[..., :d], _rotate_half(q[..., d:])], -1)
            o = _attend(q, k, (lat @ w[q_ + "uv"].T).view(B, n, H, -1), m["scale"], window=m["mask"]["size"]).flatten(2)
            y = (o * torch.sigmoid(h @ w[q_ + "g"].T)) @ w[q_ + "o"].T
            states.append(None)
        x = x + norm(y, p + "norm1b") * w[p + "ls1"]
        up = norm(x, p + "norm2") @ w[p + "mlp.up"].T + w[p + "mlp.up.b"]
        x = x + norm(F.gelu(up, approximate="tanh") @ w[p + "mlp.down"].T + w[p + "mlp.down.b"], p + "norm2b") * w[p + "ls2"]
    return norm(x[:, -1], "final.norm") @ w["head"].T, states


def _nemipel_exact(c, w, ids):
    cfg = _design(c)
    eps, alpha, states = cfg["norm"]["eps"], cfg["postln_alpha"], []
    x = w["embed"][ids]
    B, n, _ = x.shape
    kv = None
    for i, L in enumerate(cfg["layers"]):
        p, q_, m = f"l{i}.", f"l{i}.mix.", L["mixer"]
        H, d, vd = m["heads"], m["dim"], m["vdim"]
        if L["type"] == "lightning":
            q, k, v = (F.silu(x @ w[q_ + s].T).view(B, n, H, -1) for s in "qkv")
            decay = torch.tensor(m["decay"], dtype=x.dtype, device=x.device).view(1, 1, H, 1).expand(B, n, H, 1)
            o, S = _recur(q, k, v, decay)
            y = (_rms(o.flatten(2), eps) * w[q_ + "norm"] * torch.sigmoid(x @ w[q_ + "g"].T)) @ w[q_ + "o"].T
            states.append(S)
        elif L["type"] == "channel_delta":
            y, S = _delta_exact(w, q_, m, x, eps, True)
            states += [S, None]
        else:
            rot = m["rot"]
            if "kv_from" not in m:
                k = (_rms(x @ w[q_ + "k"].T, eps) * w[q_ + "k.norm"]).view(B, n, -1, d)
                kv = _rotate_pairs(k, rot["dims"], rot["base"]), (x @ w[q_ + "v"].T).view(B, n, -1, vd)
                states += [None, None]
            q = _rotate_pairs((_rms(x @ w[q_ + "q"].T, eps) * w[q_ + "q.norm"]).view(B, n, H, d), rot["dims"], rot["base"])
            o = _attend(q, *kv, m["scale"], cap=m["softcap"])
            y = (o * torch.sigmoid(x @ w[q_ + "g"].T)[..., None]).flatten(2) @ w[q_ + "o"].T
        x = _rms(alpha * x + y, eps) * w[p + "norm1"]
        f = (F.silu(x @ w[p + "mlp.gate"].T) * (x @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = _rms(alpha * x + f, eps) * w[p + "norm2"]
    cap = cfg["logit_softcap"]
    return cap * torch.tanh((_rms(x[:, -1], eps) * w["final.norm"]) @ w["head"].T / cap), states


def exact(case, seed):
    c, kind, g = case, case["kind"], _generator(seed)
    if kind in ("moe", "moe_step"):
        return _moe_exact(c, _moe_inputs(c, seed))
    if kind == "train":
        w = {n: t.double().requires_grad_(True) for n, t in _dense_weights(c, g).items()}
        ids = _ids(g, c["batch"], c["seq"] + 1)
        h = _dense_exact(c, w, ids[:, :-1]).flatten(0, 1)
        labels, T = ids[:, 1:].flatten(), h.shape[0]

        def part(hc, lc, head):
            return F.cross_entropy(hc @ head.T, lc, reduction="sum")
        loss = sum(checkpoint(part, h[i:i + 4096], labels[i:i + 4096], w["lm_head_weight"], use_reentrant=False) for i in range(0, T, 4096)) / T
        loss.backward()
        return {"loss": loss.detach(), "grads": {n: t.grad for n, t in w.items()}}
    with torch.no_grad():
        if kind == "decode":
            w = {n: (_four_bits(t) if c["bits"] == 4 and t.dim() == 2 and n.startswith("layers") else t.double()) for n, t in _dense_weights(c, g).items()}
            ids = _ids(g, c["batch"], c["context"] + 1)
            return torch.cat([_dense_exact(c, w, part)[:, -1] @ w["lm_head_weight"].T for part in ids.split(8)])
        w = {n: t.double() for n, t in _design_weights(c, g).items()}
        ids = _ids(g, c["batch"], c["seq"] if kind == "prefill" else c["context"] + 1)
        model = _vimodra_exact if c["design"] == "vimodra" else _nemipel_exact
        parts = [model(c, w, part) for part in ids.split(16)]
        states = [None if s[0] is None else torch.cat(s) for s in zip(*(p[1] for p in parts))]
        if kind == "step":
            states = [s for s in states if s is not None]
        return {"logits": torch.cat([p[0] for p in parts]), "states": states}
