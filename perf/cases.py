"""The work that programs have this framework do, as cases that can be timed and checked.

Four kinds of work, all through the entry points that the providers use:

  decode        one token for each running sequence: `ModelRunner.decode` over the paged cache, logits returned
  prefill       prompts, or portions of prompts on top of cached context: `ModelRunner.prefill`, logits returned
  image_step    one evaluation of the rectified-flow transformer: `FluxDiTGpu.forward_graphed`
  image_decode  latents to pixels: `VaeDecoderGpu.decode`

Text decoders are the Llama-3-8B configuration of `bench.py` (dense, bf16 or packed Q4_K / Q8_0 projections) and the
64-expert Qwen2-MoE configuration of `benchmarks/bench_zobunex.py`; images take the FLUX.1 configuration and its
autoencoder. All weights are random, N(0, 0.02) for projections, and in text decoders smaller by the
root of the depth for those that add to the stream.

Each kind has `exact`: the same function of the same inputs in 64 bits with plain torch."""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from inference_b200.engine.llm_engine import EngineConfig, LlmEngine
from inference_b200.models import ModelConfig
from inference_b200.models.dit_flux import FluxConfig, FluxDiTGpu, make_ids, random_flux_weights, rope_table
from inference_b200.models.registry import gpu_model
from inference_b200.models.vae import VaeConfig, VaeDecoderGpu, random_vae_weights
from inference_b200.ops.quant import quantize_on_device

STD = 0.02
DENSE = {"architectures": ["LlamaForCausalLM"], "hidden_size": 4096, "intermediate_size": 14336, "num_hidden_layers": 32,
         "num_attention_heads": 32, "num_key_value_heads": 8, "vocab_size": 128256, "rms_norm_eps": 1e-5,
         "rope_theta": 500000.0, "tie_word_embeddings": False, "max_position_embeddings": 8192}
MOE = {"model_type": "qwen2_moe", "hidden_size": 2048, "intermediate_size": 1024, "num_hidden_layers": 12,
       "num_attention_heads": 16, "num_key_value_heads": 4, "head_dim": 128, "vocab_size": 32768, "num_experts": 64,
       "num_experts_per_tok": 8, "moe_intermediate_size": 1024, "shared_expert_intermediate_size": 0,
       "tie_word_embeddings": True, "rope_theta": 500000.0, "rms_norm_eps": 1e-5}
TEXT = {"dense": DENSE, "moe": MOE}
# bytes of one packed weight (a super-block of 256 in 144 bytes, a block of 32 in 34)
PACKED = {"bf16": 2.0, "Q4_K": 144 / 256, "Q8_0": 34 / 32}


def _text(name, kind, batch, new, context, model="dense", weights="bf16"):
    return {"name": name, "kind": kind, "model": model, "weights": weights, "batch": batch, "new": new, "context": context}


def listed():
    return [
        # one user waits for each token: the latency of a chat
        _text("decode_1", "decode", 1, 1, 731),
        # a few users with long documents in the cache: weights and cache both count
        _text("decode_8_long", "decode", 8, 1, 7900),
        # a full server, the batch of the headline benchmark
        _text("decode_64", "decode", 64, 1, 1100),
        # a small server on packed weights, quantised when they were loaded
        _text("decode_4_q4k", "decode", 4, 1, 900, weights="Q4_K"),
        # a few users of a sparse model
        _text("decode_8_moe", "decode", 8, 1, 1000, model="moe"),
        # a short question: time to the first token where launches count
        _text("prefill_short", "prefill", 1, 45, 0),
        # prompts that arrived together, one wave of the scheduler's token budget
        _text("prefill_8", "prefill", 8, 1100, 0),
        # a new turn on top of a cached conversation, or one portion of a long prompt
        _text("prefill_on_context", "prefill", 1, 700, 5900),
        # prompts of the sparse model
        _text("prefill_4_moe", "prefill", 4, 1100, 0, model="moe"),
        # a small odd picture without guidance embedding (the few-step model)
        {"name": "image_step_small", "kind": "image_step", "height": 624, "width": 400, "text": 256, "guidance": False},
        # the picture of the headline benchmark
        {"name": "image_step_1024", "kind": "image_step", "height": 1024, "width": 1024, "text": 512, "guidance": True},
        # a portrait to pixels
        {"name": "image_decode_portrait", "kind": "image_decode", "height": 1216, "width": 832, "batch": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "image_step", "image_decode"])
    if kind == "decode":
        model, weights = rng.choice([("dense", "bf16"), ("dense", "bf16"), ("dense", "Q4_K"), ("dense", "Q8_0"), ("moe", "bf16")])
        batch = _log(rng, 1, 64)
        c = _text("", kind, batch, 1, _log(rng, 20, min(8000, 72000 // batch)), model, weights)
    elif kind == "prefill":
        model, weights = rng.choice([("dense", "bf16"), ("dense", "bf16"), ("dense", rng.choice(["Q4_K", "Q8_0"])), ("moe", "bf16")])
        batch = rng.choice([1, 1, 2, 3, 8])
        # packed weights are expanded for prompts: documents and not short questions
        new = _log(rng, 18, 6000 // batch) if weights == "bf16" else _log(rng, 700, 6000) // batch
        context = rng.choice([0, 0, _log(rng, 30, 6000 // batch)])
        c = _text("", kind, batch, new, context, model, weights)
    elif kind == "image_step":
        c = {"kind": kind, "height": 16 * rng.randint(16, 62), "width": 16 * rng.randint(16, 62), "text": rng.choice([256, 512]),
             "guidance": rng.random() < 0.5}
    else:
        # heights of whole 32 pixels: the decoder's attention takes a multiple of 8 latent pixels
        h, w = rng.choice([(1024, 1024), (512, 512), (32 * rng.randint(10, 32), 16 * rng.randint(20, 64))])
        c = {"kind": kind, "height": h, "width": w, "batch": 1}
    c.pop("name", None)
    return c


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000 * seed + salt)


# ---- text ------------------------------------------------------------------------------------------------------------
def _lengths(case):
    """(new tokens, cached tokens) of each sequence: the first has the full length, the others are up to a third shorter."""
    got = []
    for i in range(case["batch"]):
        cut = ((i * 37) % 64) / 192
        new = case["new"] if case["kind"] == "decode" else max(1, case["new"] - int(case["new"] * cut))
        got.append((new, max(0, case["context"] - int(case["context"] * cut))))
    return got


def _text_weights(case, seed):
    """Full checkpoint tensors by their usual names, bf16 on the GPU."""
    m, g = TEXT[case["model"]], _generator(seed, 1)
    H, D = m["hidden_size"], 128
    packed = case["weights"] != "bf16"

    def rnd(*shape, std=STD):
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)

    # The stream starts at the size of its embedding, and each sublayer adds a little, as in a trained decoder: projections back into
    # the stream are smaller by the square root of their number.
    back = STD / (2 * m["num_hidden_layers"]) ** 0.5

    def norm(n):        # packed weights are made from the checkpoint's own: unit norms leave them as they are
        one = torch.ones(n, dtype=torch.bfloat16, device="cuda")
        return one if packed else one + rnd(n) * 5

    w = {"model.embed_tokens.weight": rnd(m["vocab_size"], H, std=1.0), "model.norm.weight": norm(H)}
    if not m["tie_word_embeddings"]:
        w["lm_head.weight"] = rnd(m["vocab_size"], H)
    for i in range(m["num_hidden_layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = norm(H), norm(H)
        for n, heads in (("q", m["num_attention_heads"]), ("k", m["num_key_value_heads"]), ("v", m["num_key_value_heads"])):
            w[f"{p}self_attn.{n}_proj.weight"] = rnd(heads * D, H)
            if case["model"] == "moe":
                w[f"{p}self_attn.{n}_proj.bias"] = rnd(heads * D)
        w[p + "self_attn.o_proj.weight"] = rnd(H, m["num_attention_heads"] * D, std=back)
        if case["model"] == "dense":
            mlps, ff = [p + "mlp."], m["intermediate_size"]
        else:
            w[p + "mlp.gate.weight"] = rnd(m["num_experts"], H)
            mlps, ff = [f"{p}mlp.experts.{e}." for e in range(m["num_experts"])], m["moe_intermediate_size"]
        for q in mlps:
            w[q + "gate_proj.weight"], w[q + "up_proj.weight"], w[q + "down_proj.weight"] = rnd(ff, H), rnd(ff, H), rnd(H, ff, std=back)
    return w


def _tokens(case, seed):
    g = torch.Generator().manual_seed(seed * 7 + 3)
    return [torch.randint(0, TEXT[case["model"]]["vocab_size"], (n,), generator=g).tolist() for n, _ in _lengths(case)]


def _cached(case, seed, layer):
    """Keys (rotated) and values of the cached tokens of one layer, all sequences one behind the other: [2, tokens, heads, 128].
    Their size is that of a projection of normed activations."""
    m = TEXT[case["model"]]
    n = sum(c for _, c in _lengths(case))
    x = torch.empty((2, n, m["num_key_value_heads"], 128), dtype=torch.bfloat16, device="cuda")
    return x.normal_(0.0, STD * m["hidden_size"] ** 0.5, generator=_generator(seed, 100 + layer))


def _prepare_text(case, seed):
    cfg = ModelConfig.from_json(TEXT[case["model"]])
    model = gpu_model(cfg, device=torch.device("cuda", torch.cuda.current_device())).load_state_dict(_text_weights(case, seed))
    if case["weights"] != "bf16":
        model.quantize_(case["weights"])
    lengths = _lengths(case)
    longest = max(n + c for n, c in lengths)
    eng = LlmEngine(model, EngineConfig(max_batch=case["batch"], max_seq_len=(longest + 31) // 16 * 16))
    seqs = [eng.new_sequence() for _ in lengths]
    if case["context"]:
        slots = torch.tensor([x for s, (_, c) in zip(seqs, lengths) for x in s.reserve(c)], device="cuda")
        block, place = slots // eng.pool.block_size, slots % eng.pool.block_size
        for layer in range(cfg.num_layers):
            kv = _cached(case, seed, layer)
            for j in range(2):
                eng.pool.data[layer, j][block, :, place] = kv[j]
    state = {"case": case, "engine": eng, "seqs": seqs, "cached": [c for _, c in lengths], "tokens": _tokens(case, seed)}
    if case["kind"] == "decode":        # a server's step graph is there from its first tokens on
        _run_text(state)
    return state


def _run_text(state):
    runner = state["engine"].runner
    for s, n in zip(state["seqs"], state["cached"]):        # back to the cached context: every pass appends the same tokens
        s.truncate(n)
    if state["case"]["kind"] == "decode":
        return runner.decode(state["seqs"], [t[0] for t in state["tokens"]], want_logits=True)
    return runner.prefill(state["seqs"], state["tokens"], want_logits=True)


def _run_prefill(state):
    logits = _run_text(state)
    pool = state["engine"].pool.data
    return {"logits": logits, "cache": pool}


def _work_text(case):
    m, lengths = TEXT[case["model"]], _lengths(case)
    H, L, D, V = m["hidden_size"], m["num_hidden_layers"], 128, m["vocab_size"]
    hq, hkv = m["num_attention_heads"], m["num_key_value_heads"]
    T, B = sum(n for n, _ in lengths), case["batch"]
    attn = (2 * hq + 2 * hkv) * D * H
    if case["model"] == "dense":
        read = used = attn + 3 * H * m["intermediate_size"]
    else:
        E, k, one = m["num_experts"], m["num_experts_per_tok"], 3 * H * m["moe_intermediate_size"]
        read = attn + E * H + one * E * (1 - (1 - k / E) ** T)      # experts that some token takes
        used = attn + E * H + one * k
    row = 2 * hkv * D * 2
    bytes_ = L * (read * PACKED[case["weights"]] + row * (sum(c for _, c in lengths) + T)) + V * H * 2 + T * H * 2 + B * V * 4
    pairs = sum(n * c + n * (n + 1) // 2 for n, c in lengths)
    return {"bytes": bytes_, "flops": 2.0 * L * used * T + 2.0 * V * H * B + 4.0 * L * hq * D * pairs}


def _rms64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _packed64(w, fmt):
    """What a matrix is after quantise-on-load: the packed blocks read back by their published layout."""
    if fmt == "bf16":
        return w.double()
    n, k = w.shape
    raw = quantize_on_device(w, fmt).packed.reshape(n, -1)
    half = lambda t: t.contiguous().view(torch.float16).double()  # noqa: E731
    if fmt == "Q8_0":
        b = raw.reshape(n, k // 32, 34)
        return (half(b[..., :2]) * b[..., 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    b = raw.reshape(n, k // 256, 144)
    s = b[..., 4:16].int()
    scale = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | (s[..., 0:4] >> 6 << 4)], -1).double()
    least = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | (s[..., 4:8] >> 6 << 4)], -1).double()
    q = b[..., 16:].reshape(n, k // 256, 4, 32)
    q = torch.stack([q & 15, q >> 4], -2).reshape(n, k // 256, 8, 32).double()
    d, dmin = half(b[..., 0:2])[..., None], half(b[..., 2:4])[..., None]
    return (d * scale[..., None] * q - dmin * least[..., None]).reshape(n, k)


def _exact_text(case, seed):
    m, w, lengths = TEXT[case["model"]], _text_weights(case, seed), _lengths(case)
    D, hq, hkv, eps = 128, m["num_attention_heads"], m["num_key_value_heads"], m["rms_norm_eps"]
    ids = torch.tensor([t for row in _tokens(case, seed) for t in row], device="cuda")
    pos = torch.cat([torch.arange(c, c + n, device="cuda") for n, c in lengths]).double()
    inv = m["rope_theta"] ** (-torch.arange(0, D, 2, device="cuda").double() / D)
    cos, sin = (pos[:, None] * inv).cos()[:, None], (pos[:, None] * inv).sin()[:, None]
    T, fmt = ids.numel(), case["weights"]

    def rotate(x):
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def lin(x, name):
        y = x @ _packed64(w[name + ".weight"], fmt).T
        return y + w[name + ".bias"].double() if name + ".bias" in w else y

    def gated(x, p, f):
        return (F.silu(x @ f(w[p + "gate_proj.weight"]).T) * (x @ f(w[p + "up_proj.weight"]).T)) @ f(w[p + "down_proj.weight"]).T

    x = w["model.embed_tokens.weight"][ids].double()
    for layer in range(m["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        h = _rms64(x, w[p + "input_layernorm.weight"], eps)
        q = rotate(lin(h, p + "self_attn.q_proj").view(T, hq, D))
        k = rotate(lin(h, p + "self_attn.k_proj").view(T, hkv, D))
        v = lin(h, p + "self_attn.v_proj").view(T, hkv, D)
        kv = _cached(case, seed, layer)
        out, at, back = torch.empty_like(q), 0, 0
        for n, c in lengths:
            seen = torch.arange(c + n, device="cuda")[None, :] <= torch.arange(c, c + n, device="cuda")[:, None]
            for g in range(hkv):
                keys = torch.cat([kv[0, back:back + c, g].double(), k[at:at + n, g]])
                values = torch.cat([kv[1, back:back + c, g].double(), v[at:at + n, g]])
                heads = slice(g * (hq // hkv), (g + 1) * (hq // hkv))
                s = torch.einsum("nhd,kd->hnk", q[at:at + n, heads], keys) * D ** -0.5
                out[at:at + n, heads] = (s.masked_fill_(~seen, -math.inf).softmax(-1) @ values).transpose(0, 1)
            at, back = at + n, back + c
        x = x + lin(out.reshape(T, hq * D), p + "self_attn.o_proj")
        h = _rms64(x, w[p + "post_attention_layernorm.weight"], eps)
        if case["model"] == "dense":
            x = x + gated(h, p + "mlp.", lambda t: _packed64(t, fmt))
        else:
            share, which = (h @ w[p + "mlp.gate.weight"].double().T).softmax(-1).topk(m["num_experts_per_tok"], -1)
            y = torch.zeros_like(x)
            for e in range(m["num_experts"]):
                row, place = (which == e).nonzero(as_tuple=True)
                if row.numel():
                    y.index_add_(0, row, gated(h[row], f"{p}mlp.experts.{e}.", torch.Tensor.double) * share[row, place][:, None])
            x = x + y
    last = torch.tensor([n for n, _ in lengths], device="cuda").cumsum(0) - 1
    head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
    h = _rms64(x[last], w["model.norm.weight"], eps)
    return torch.cat([h @ head[i:i + 16384].double().T for i in range(0, head.shape[0], 16384)], -1)


# ---- images ----------------------------------------------------------------------------------------------------------
def _image_inputs(case, seed, cfg):
    h, w, g = case["height"] // 16, case["width"] // 16, _generator(seed, 2)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda").bfloat16()

    txt_ids, img_ids = make_ids(h, w, case["text"], device="cuda")
    return {"img": rnd(1, h * w, cfg.in_channels), "img_ids": img_ids, "txt": rnd(1, case["text"], cfg.context_in_dim), "txt_ids": txt_ids,
            "timesteps": torch.rand(1, generator=g, device="cuda"), "y": rnd(1, cfg.vec_in_dim),
            "guidance": torch.full((1,), 3.5, device="cuda") if case["guidance"] else None}


def _prepare_step(case, seed):
    cfg = FluxConfig(guidance_embed=case["guidance"])
    dit = FluxDiTGpu(cfg, device=torch.device("cuda", torch.cuda.current_device()))
    dit.load_state_dict(random_flux_weights(cfg, seed, STD, torch.bfloat16, "cuda"))
    x = _image_inputs(case, seed, cfg)
    x["rope"] = rope_table(torch.cat([x["txt_ids"], x["img_ids"]]), cfg.axes_dim, cfg.theta)
    dit.forward_graphed(**x)        # all steps of a picture but the first find the graph
    return {"case": case, "dit": dit, "inputs": x}


def _work_step(case):
    cfg = FluxConfig()
    H, M, si, st = cfg.hidden_size, cfg.mlp_hidden, case["height"] * case["width"] // 256, case["text"]
    S = si + st
    block = 4 * H * H + 2 * H * M
    mods = (12 * cfg.depth + 3 * cfg.depth_single + 2) * H * H
    ends = (cfg.in_channels * 2 + 0) * H
    embeds = (2 if case["guidance"] else 1) * (256 + H) * H + (cfg.vec_in_dim + H) * H
    weights = 2 * cfg.depth * block + cfg.depth_single * block + mods + ends + cfg.context_in_dim * H + embeds
    flops = 2.0 * ((cfg.depth + cfg.depth_single) * block * S + mods + embeds + cfg.in_channels * 2 * H * si + cfg.context_in_dim * H * st)
    return {"bytes": 2.0 * (weights + 2 * si * cfg.in_channels + st * cfg.context_in_dim),
            "flops": flops + 4.0 * (cfg.depth + cfg.depth_single) * H * S * S}


def _exact_step(case, seed):
    cfg = FluxConfig(guidance_embed=case["guidance"])
    w, x = random_flux_weights(cfg, seed, STD, torch.bfloat16, "cuda"), _image_inputs(case, seed, cfg)
    H, NH, D = cfg.hidden_size, cfg.num_heads, cfg.hidden_size // cfg.num_heads
    ids = torch.cat([x["txt_ids"], x["img_ids"]]).double()
    ang = torch.cat([ids[:, i, None] * cfg.theta ** (-torch.arange(0, d, 2, device="cuda").double() / d)
                     for i, d in enumerate(cfg.axes_dim)], -1)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    St = case["text"]

    def lin(t, name):
        return t @ w[name + ".weight"].double().T + w[name + ".bias"].double()

    def embed(t, name):
        return lin(F.silu(lin(t, name + ".in_layer")), name + ".out_layer")

    def wave(t):        # the sinusoids are 32-bit by definition of the model
        f = torch.exp(-math.log(10000.0) * torch.arange(128, dtype=torch.float32, device="cuda") / 128)
        a = (1000.0 * t.float())[:, None] * f[None]
        return torch.cat([a.cos(), a.sin()], -1).double()

    def ln(t, scale, shift):
        return F.layer_norm(t, (H,), eps=1e-6) * (1 + scale) + shift

    def heads(t, p):
        q, k, v = t.view(-1, 3, NH, D).unbind(1)
        return _rms64(q, w[p + ".query_norm.scale"], 1e-6), _rms64(k, w[p + ".key_norm.scale"], 1e-6), v

    def attend(q, k, v):
        out = torch.empty_like(q)
        for r in (q, k):
            a, b = r[..., 0::2].clone(), r[..., 1::2].clone()
            r[..., 0::2], r[..., 1::2] = a * cos - b * sin, b * cos + a * sin
        for i in range(NH):
            out[:, i] = (q[:, i] @ k[:, i].T * D ** -0.5).softmax(-1) @ v[:, i]
        return out.reshape(-1, H)

    vec = embed(wave(x["timesteps"]), "time_in") + embed(x["y"].double(), "vector_in")
    if case["guidance"]:
        vec = vec + embed(wave(x["guidance"]), "guidance_in")
    sv = F.silu(vec)
    s = {"img": lin(x["img"][0].double(), "img_in"), "txt": lin(x["txt"][0].double(), "txt_in")}
    for i in range(cfg.depth):
        p = f"double_blocks.{i}."
        mod = {n: lin(sv, p + n + "_mod.lin").chunk(6, -1) for n in s}
        qkv = {n: heads(lin(ln(s[n], mod[n][1], mod[n][0]), p + n + "_attn.qkv"), p + n + "_attn.norm") for n in s}
        a = attend(*(torch.cat([t, u]) for t, u in zip(qkv["txt"], qkv["img"])))
        for n, part in (("txt", a[:St]), ("img", a[St:])):
            y = s[n] + mod[n][2] * lin(part, p + n + "_attn.proj")
            h = F.gelu(lin(ln(y, mod[n][4], mod[n][3]), p + n + "_mlp.0"), approximate="tanh")
            s[n] = y + mod[n][5] * lin(h, p + n + "_mlp.2")
    t = torch.cat([s["txt"], s["img"]])
    for i in range(cfg.depth_single):
        p = f"single_blocks.{i}."
        shift, scale, gate = lin(sv, p + "modulation.lin").chunk(3, -1)
        y = lin(ln(t, scale, shift), p + "linear1")
        q, k, v = heads(y[:, :3 * H], p + "norm")
        t = t + gate * lin(torch.cat([attend(q, k, v), F.gelu(y[:, 3 * H:], approximate="tanh")], -1), p + "linear2")
    shift, scale = lin(sv, "final_layer.adaLN_modulation.1").chunk(2, -1)
    return lin(ln(t[St:], scale, shift), "final_layer.linear")[None]


def _latents(case, seed):
    return torch.randn(case["batch"], VaeConfig().z_channels, case["height"] // 8, case["width"] // 8, generator=_generator(seed, 3),
                       device="cuda")


def _prepare_decode(case, seed):
    vae = VaeDecoderGpu(VaeConfig(), device=torch.device("cuda", torch.cuda.current_device()))
    vae.load_state_dict(random_vae_weights(VaeConfig(), seed, device="cuda"))
    return {"case": case, "vae": vae, "latents": _latents(case, seed)}


def _work_decode(case):
    """Convolutions level by level; the largest level's activations need not touch memory."""
    cfg = VaeConfig()
    px = case["batch"] * case["height"] // 8 * case["width"] // 8
    c = cfg.ch * cfg.ch_mult[-1]
    macs, params = px * 9 * cfg.z_channels * c, 9 * cfg.z_channels * c
    mid = 4 * 9 * c * c + 4 * c * c
    macs += px * mid + 2 * px * (px // case["batch"]) * c
    params += mid
    for level in reversed(range(len(cfg.ch_mult))):
        out = cfg.ch * cfg.ch_mult[level]
        for _ in range(cfg.num_res_blocks + 1):
            one = 9 * c * out + 9 * out * out + (c * out if c != out else 0)
            macs, params, c = macs + px * one, params + one, out
        if level:
            px *= 4
            macs, params = macs + px * 9 * c * c, params + 9 * c * c
    macs += px * 9 * c * cfg.out_ch
    return {"bytes": 2.0 * params + 4.0 * case["batch"] * cfg.z_channels * case["height"] * case["width"] / 64 + 2.0 * px * 8, "flops": 2.0 * macs}


def _exact_decode(case, seed):
    cfg = VaeConfig()
    w = {k: t.bfloat16().double() for k, t in random_vae_weights(cfg, seed, device="cuda").items()}

    def conv(t, name):
        k = w[name + ".weight"]
        if k.shape[-1] == 1:
            return torch.einsum("oc,bchw->bohw", k[:, :, 0, 0], t) + w[name + ".bias"][:, None, None]
        B, C, rows, cols = t.shape      # one product per tap: 64-bit convolutions of the library are slow
        t, y = F.pad(t, (1, 1, 1, 1)), w[name + ".bias"][:, None, None].expand(k.shape[0], rows, cols).repeat(B, 1, 1, 1)
        for i in range(3):
            for j in range(3):
                y.view(B, -1, rows * cols).baddbmm_(k[:, :, i, j].expand(B, -1, -1), t[:, :, i:i + rows, j:j + cols].reshape(B, C, -1))
        return y

    def gn(t, name):
        return F.group_norm(t, 32, w[name + ".weight"], w[name + ".bias"], 1e-6)

    def res(t, name):
        h = conv(F.silu(gn(t, name + ".norm1")), name + ".conv1")
        h = conv(F.silu(gn(h, name + ".norm2")), name + ".conv2")
        return (conv(t, name + ".nin_shortcut") if name + ".nin_shortcut.weight" in w else t) + h

    h = conv(_latents(case, seed).double() / cfg.scale_factor + cfg.shift_factor, "decoder.conv_in")
    h = res(h, "decoder.mid.block_1")
    n = gn(h, "decoder.mid.attn_1.norm")
    q, k, v = (conv(n, f"decoder.mid.attn_1.{x}").flatten(2).transpose(1, 2) for x in "qkv")
    a = ((q @ k.transpose(1, 2)) * q.shape[-1] ** -0.5).softmax(-1) @ v
    h = res(h + conv(a.transpose(1, 2).reshape(h.shape), "decoder.mid.attn_1.proj_out"), "decoder.mid.block_2")
    for level in reversed(range(len(cfg.ch_mult))):
        for i in range(cfg.num_res_blocks + 1):
            h = res(h, f"decoder.up.{level}.block.{i}")
        if level:
            h = conv(F.interpolate(h, scale_factor=2, mode="nearest"), f"decoder.up.{level}.upsample.conv")
    h = conv(F.silu(gn(h, "decoder.norm_out")), "decoder.conv_out").permute(0, 2, 3, 1)
    return F.pad(h, (0, 8 - h.shape[-1]))       # pixels come eight channels wide


# ---- the functions that measure and check a case call -----------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] in ("decode", "prefill"):
        return _prepare_text(case, seed)
    return _prepare_step(case, seed) if case["kind"] == "image_step" else _prepare_decode(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "decode":
        return _run_text(state)
    if kind == "prefill":
        return _run_prefill(state)
    if kind == "image_step":
        return state["dit"].forward_graphed(**state["inputs"])
    return state["vae"].decode(state["latents"])


def work(case):
    return {"decode": _work_text, "prefill": _work_text, "image_step": _work_step, "image_decode": _work_decode}[case["kind"]](case)


def tolerance(case):
    """Rounding to bf16 between dozens of layers. Measured against `exact`: 0.01 to 0.025 for every kind (2-norm), and the largest
    single difference up to 0.25 of the root mean square; two correct implementations are up to 1.4 times that apart."""
    return {"rel": 0.03, "max": 0.6}


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "decode":
        return _exact_text(case, seed)
    if case["kind"] == "prefill":       # the cache's layout is the framework's own
        return {"logits": _exact_text(case, seed), "cache": None}
    return _exact_step(case, seed) if case["kind"] == "image_step" else _exact_decode(case, seed)
