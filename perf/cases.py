"""The work that programs built on this framework have it do, as measurable cases.

A case is a dict of plain values.  `part` names the path:

  vision     LlavaLlamaModel.encode_images: SigLIP tower (two of its equal layers) + projector, `tiles` images of 448 x 448
  prefill    Qwen2ForCausalLM.prefill_hidden_graphed of one prompt + the logits of its last token, at NVILA-8B / -Lite-3B widths
  decode     the greedy loop of one request: first token from the prompt's last hidden state, then one graph replay per token
  serve      TokenEngine.step of a whole token-id model (four layers): prompts admitted together, then decoded step by step
  experts    a routed feed-forward block of the token-id models: router, grouping, two grouped projections, residual sum
  attention  an attention block over the paged k | v pool: rotation / norm / append, then attention; `form` names the variant
  scan       a recurrent mixer over per-sequence states; `form` names the recurrence
  head       final norm + output head, fp32 logits

Blocks of decoded tokens are held as a captured CUDA graph, as GraphDecoder and TokenEngine hold theirs; everything else is
called eagerly.  exact() restates each path in float64 with plain torch.
"""
from __future__ import annotations

import gc
import math

import torch
import torch.nn.functional as F

DEV = "cuda"
BF = torch.bfloat16
PAGE = 64
EPS = 1e-5


# ---- the cases ---------------------------------------------------------------------------------------
def listed():
    lm = dict(heads=16, kv_heads=4)
    return [
        # one image: what every single-picture question pays before its prompt
        dict(name="image_tower", part="vision", tiles=1),
        # one picture cut into tiles (12 + thumbnail), or a short video
        dict(name="tiled_image_tower", part="vision", tiles=13),
        # the prompt of the headline request: 256 image tokens + 23 text tokens
        dict(name="image_prompt", part="prefill", size="8b", tokens=279, layers=2),
        # a 64-frame video prompt
        dict(name="video_prompt", part="prefill", size="8b", tokens=16470, layers=1),
        # token generation of the headline request
        dict(name="image_decode", part="decode", size="8b", context=279, tokens=9, layers=2),
        # continuous batching: prompts of several users, then some decoded tokens for each
        dict(name="serve_engine", part="serve", width=1024, seqs=4, rows=200, steps=6),
        # a 2048-token prompt portion (the scheduler's step budget) through the routed experts
        dict(name="experts_prompt", part="experts", rows=2048, width=2048, experts=32, top=4, ff=704),
        # eight decoded tokens through the same block
        dict(name="experts_decode", part="experts", rows=8, width=2048, experts=32, top=4, ff=704),
        # causal attention of a 2048-token prompt: capped scores, output gate
        dict(name="attention_prompt", part="attention", form="capped", seqs=1, rows=2048, context=0, **lm),
        # eight decoded tokens, each over 1024 cached ones
        dict(name="attention_decode", part="attention", form="capped", seqs=8, rows=1, context=1024, **lm),
        # scalar-decay state-space recurrence over a 2048-token prompt
        dict(name="scan_prompt", part="scan", form="ssd", seqs=1, rows=2048, width=2048, context=0),
        # logits of eight decoded tokens
        dict(name="head_decode", part="head", rows=8, width=2048, vocab=32768),
    ]


FORMS = ("capped", "talk", "window", "chunk", "diff")
SCANS = ("ssd", "decay", "gla", "delta", "hgrn2")


def draw(rng):
    def log_int(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    part = rng.choice(["vision", "prefill", "decode", "serve", "experts", "experts", "attention", "attention", "attention",
                       "scan", "scan", "head"])
    if part == "vision":
        return dict(part=part, tiles=log_int(1, 13))
    if part == "prefill":
        return dict(part=part, size=rng.choice(["8b", "3b"]), tokens=log_int(17, 8000), layers=rng.choice([1, 2]))
    if part == "decode":
        return dict(part=part, size=rng.choice(["8b", "3b"]), context=log_int(40, 8000), tokens=rng.choice([5, 9]), layers=2)
    if part == "serve":
        return dict(part=part, width=1024, seqs=rng.choice([1, 2, 3, 5]), rows=log_int(17, 190), steps=rng.choice([3, 6]))
    if part == "head":
        return dict(part=part, rows=log_int(1, 96), width=rng.choice([1024, 2048, 4096]), vocab=log_int(8000, 65536))
    width = rng.choice([1024, 2048, 2048, 4096])
    if part == "experts":
        experts, top, ff = {1024: (16, 2, 512), 2048: (32, 4, 704), 4096: (64, 6, 1408)}[width]
        rows = rng.choice([rng.randint(1, 16), log_int(17, 2048 * 2048 // width if width > 2048 else 2048)])
        return dict(part=part, rows=rows, width=width, experts=experts, top=top, ff=ff)
    decode = rng.random() < 0.4
    if part == "attention":
        heads = width // 128
        kv = rng.choice([heads, heads // 4, heads // 4])
        if decode:
            return dict(part=part, form=rng.choice(FORMS), seqs=log_int(1, 24), rows=1, context=log_int(30, 4000), heads=heads,
                        kv_heads=kv)
        rows = log_int(9, 2048 if heads <= 16 else 1024)
        seqs = rng.randint(1, max(1, min(8, (2048 if heads <= 16 else 1024) // rows)))
        return dict(part=part, form=rng.choice(FORMS), seqs=seqs, rows=rows, context=rng.choice([0, 0, log_int(64, 1024)]),
                    heads=heads, kv_heads=kv)
    if decode:
        return dict(part=part, form=rng.choice(SCANS), seqs=log_int(1, 24), rows=1, width=width, context=log_int(30, 4000))
    rows = log_int(9, 2048)
    return dict(part=part, form=rng.choice(SCANS), seqs=rng.randint(1, max(1, min(8, 2048 // rows))), rows=rows, width=width,
                context=rng.choice([0, 0, 500]))


# ---- shared helpers ------------------------------------------------------------------------------------
class State:
    """What a case holds between passes: .step is one pass, a function of the state."""


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, mean=0.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device=DEV) * std + mean).to(dtype)


def _rand(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=g, device=DEV) * (hi - lo) + lo


def _captured(fn):
    """fn() as a graph replay: a program captures the launches of a decoded step once and replays them."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        fn()
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()

    def replay(_):
        graph.replay()
        return out
    return replay


def _rms(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _sigmoid(x):
    return torch.sigmoid(x)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(u, pos, dims, base, halves):
    """u [T, heads, d] float64, pos [T]"""
    half = dims // 2
    inv = base ** (-2.0 * torch.arange(half, device=u.device, dtype=torch.float64) / dims)
    ang = pos.double()[:, None, None] * inv
    c, s = torch.cos(ang), torch.sin(ang)
    out = u.clone()
    a, b = (u[..., :half], u[..., half:dims]) if halves else (u[..., 0:dims:2], u[..., 1:dims:2])
    if halves:
        out[..., :half], out[..., half:dims] = a * c - b * s, b * c + a * s
    else:
        out[..., 0:dims:2], out[..., 1:dims:2] = a * c - b * s, b * c + a * s
    return out


# ---- vision ----------------------------------------------------------------------------------------------
def _vision_inputs(c, seed):
    from vila_b200.model import LlavaConfig, LlavaLlamaModel
    from vila_b200.model.configuration import Qwen2Config, SiglipVisionConfig
    cfg = LlavaConfig(vision_tower_cfg=SiglipVisionConfig(num_hidden_layers=3), llm_cfg=Qwen2Config(num_hidden_layers=0, vocab_size=64))
    s = State()
    s.model = LlavaLlamaModel(cfg, device=DEV).init_random(seed, device_rng=True)
    s.pixels = _randn(_gen(seed + 1), c["tiles"], 3, 448, 448)
    return s


def _vision_prepare(c, seed):
    s = _vision_inputs(c, seed)
    s.step = lambda s: s.model.encode_images(s.pixels)
    s.step(s)   # the model keeps a graph per input shape
    return s


def _vision_exact(c, seed):
    s = _vision_inputs(c, seed)
    m = s.model
    d = lambda p: p.detach().double()
    vm, cfg = m.vision_tower.vision_tower.vision_model, m.vision_tower.config
    B, C, H = c["tiles"], cfg.hidden_size, cfg.num_attention_heads
    outs = []
    for px in s.pixels.double():
        x = F.conv2d(px[None], d(vm.embeddings.patch_embedding.weight), d(vm.embeddings.patch_embedding.bias), stride=cfg.patch_size)
        x = x.flatten(2)[0].T + d(vm.embeddings.position_embedding.weight)
        for L in list(vm.encoder.layers)[:cfg.num_hidden_layers - 1]:
            h = F.layer_norm(x, (C,), d(L.layer_norm1.weight), d(L.layer_norm1.bias), cfg.layer_norm_eps)
            q, k, v = (F.linear(h, d(p.weight), d(p.bias)).view(-1, H, C // H).transpose(0, 1)
                       for p in (L.self_attn.q_proj, L.self_attn.k_proj, L.self_attn.v_proj))
            a = torch.softmax(q @ k.transpose(1, 2) * (C // H) ** -0.5, -1) @ v
            x = x + F.linear(a.transpose(0, 1).reshape(-1, C), d(L.self_attn.out_proj.weight), d(L.self_attn.out_proj.bias))
            h = F.layer_norm(x, (C,), d(L.layer_norm2.weight), d(L.layer_norm2.bias), cfg.layer_norm_eps)
            h = F.gelu(F.linear(h, d(L.mlp.fc1.weight), d(L.mlp.fc1.bias)), approximate="tanh")
            x = x + F.linear(h, d(L.mlp.fc2.weight), d(L.mlp.fc2.bias))
        n = int(x.shape[0] ** 0.5)
        # 2 x 2 neighbouring patches side by side: (row, column) offsets in row-major order
        x = x.view(n // 2, 2, n // 2, 2, C).permute(0, 2, 1, 3, 4).reshape(-1, 4 * C)
        ln, l1, l2 = (p for _, p in m.mm_projector._program)
        x = F.layer_norm(x, (4 * C,), d(ln.weight), d(ln.bias), 1e-5)
        outs.append(F.linear(F.gelu(F.linear(x, d(l1.weight), d(l1.bias))), d(l2.weight), d(l2.bias)))
    return torch.stack(outs)


def _vision_work(c):
    C, I, T, W = 1152, 4304, 1024 * c["tiles"], 3584
    weights = 588 * C + 2 * (4 * C * C + 2 * C * I) + 4 * C * W + W * W
    return dict(bytes=2 * weights + 2 * c["tiles"] * (3 * 448 * 448 + 256 * W),
                flops=2.0 * T * (588 * C + 2 * (4 * C * C + 2 * C * I + 2 * 1024 * C)) + 2.0 * T / 4 * (4 * C * W + W * W))


# ---- Qwen2 -----------------------------------------------------------------------------------------------
SIZES = {"8b": dict(hidden_size=3584, intermediate_size=18944, num_attention_heads=28, num_key_value_heads=4),
         "3b": dict(hidden_size=2048, intermediate_size=11008, num_attention_heads=16, num_key_value_heads=2)}
VOCAB = 16384


def _qwen2(c, seed):
    """Random weights; the output head is the embedding shifted by one row, so that a trained model's confident choices are
    met: after token i comes token i + 1, by a wide margin."""
    from vila_b200.model.configuration import Qwen2Config
    from vila_b200.model.qwen2 import Qwen2ForCausalLM
    m = Qwen2ForCausalLM(Qwen2Config(num_hidden_layers=c["layers"], vocab_size=VOCAB, **SIZES[c["size"]]), device=DEV)
    g = _gen(seed)
    with torch.no_grad():
        for name, p in m.named_parameters():
            if "embed_tokens" in name or "lm_head" in name:
                continue
            p.copy_(_randn(g, *p.shape, std=0.02, mean=1.0 if "norm" in name else 0.0))
        m.model.embed_tokens.weight.copy_(_randn(g, VOCAB, m.config.hidden_size))
        m.lm_head.weight.copy_(m.model.embed_tokens.weight.roll(1, 0) * 0.02)
    s = State()
    s.model = m
    s.ids = torch.randint(0, VOCAB - 64, (c.get("tokens") if "context" not in c else c["context"],), generator=g, device=DEV)
    s.embeds = m.model.embed_tokens.weight[s.ids].contiguous()
    return s


def _qwen2_layers(m, x, upto=None):
    """x [S, hidden] float64 -> (hidden before the last norm, per layer (k rotated, v))"""
    cfg = m.config
    Hq, Hkv, D, S = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, x.shape[0]
    d = lambda p: p.detach().double()
    pos, kv = torch.arange(S, device=DEV), []
    for L in m.model.layers:
        h = _rms(x, cfg.rms_norm_eps) * d(L.input_layernorm.weight)
        q, k, v = (F.linear(h, d(p.weight), d(p.bias)).view(S, -1, D) for p in (L.self_attn.q_proj, L.self_attn.k_proj, L.self_attn.v_proj))
        q, k = (_rotate(u, pos, D, cfg.rope_theta, True) for u in (q, k))
        kv.append((k, v))
        a = torch.empty_like(q)
        for i in range(Hq):
            g = i // (Hq // Hkv)
            for r in range(0, S, 4096):
                e = min(S, r + 4096)
                sc = q[r:e, i] @ k[:e, g].T * D ** -0.5
                sc.masked_fill_(pos[None, :e] > pos[r:e, None], float("-inf"))
                a[r:e, i] = torch.softmax(sc, -1) @ v[:e, g]
        x = x + a.view(S, -1) @ d(L.self_attn.o_proj.weight).T
        h = _rms(x, cfg.rms_norm_eps) * d(L.post_attention_layernorm.weight)
        x = x + (_silu(h @ d(L.mlp.gate_proj.weight).T) * (h @ d(L.mlp.up_proj.weight).T)) @ d(L.mlp.down_proj.weight).T
    return x, kv


def _prefill_prepare(c, seed):
    s = _qwen2(c, seed)
    s.cache = s.model.new_cache(c["tokens"])

    def step(s):
        with torch.inference_mode():
            s.cache.length = 0
            hid = s.model.prefill_hidden_graphed(s.embeds, s.cache)
            return [hid, s.model.logits_from_hidden(hid[-1:])]
    s.step = step
    s.step(s)   # the model keeps a graph per short prompt length
    return s


def _prefill_exact(c, seed):
    s = _qwen2(c, seed)
    x, _ = _qwen2_layers(s.model, s.embeds.double())
    w = s.model
    return [x, (_rms(x[-1:], w.config.rms_norm_eps) * w.model.norm.weight.double()) @ w.lm_head.weight.double().T]


def _qwen2_sizes(c):
    z = SIZES[c["size"]]
    W, I, q, kv = z["hidden_size"], z["intermediate_size"], z["num_attention_heads"] * 128, z["num_key_value_heads"] * 128
    return W, q, kv, c["layers"] * (W * (2 * q + 2 * kv) + 3 * W * I)


def _prefill_work(c):
    W, q, kv, weights = _qwen2_sizes(c)
    S = c["tokens"]
    return dict(bytes=2 * (weights + VOCAB * W) + S * (4 * W + 4 * kv * c["layers"]),
                flops=2.0 * S * weights + c["layers"] * 2.0 * S * (S + 1) * q + 2.0 * VOCAB * W)


def _decode_prepare(c, seed):
    s = _qwen2(c, seed)
    S, n = c["context"], c["tokens"]
    with torch.inference_mode():
        s.dec = s.model.decoder(n)
        s.cache = s.dec.cache_for(S + n)
        s.last = s.model.prefill_hidden(s.embeds, s.cache)[-1].clone()

    def step(s):
        with torch.inference_mode():
            s.cache.length = S
            s.dec.start(s.last, s.cache)
            s.dec.run(n)
            return [s.dec.hist[:n], s.cache.pool.flatten(2, 3)[:, :, S:S + n - 1]]
    s.step = step
    s.step(s)   # the decoder keeps the graph of a token
    return s


def _decode_exact(c, seed):
    s = _qwen2(c, seed)
    S, n = c["context"], c["tokens"]
    new = (s.ids[-1] + 1 + torch.arange(n - 1, device=DEV)) % VOCAB
    _, kv = _qwen2_layers(s.model, torch.cat([s.embeds, s.model.model.embed_tokens.weight[new]]).double())
    return [None, torch.stack([torch.stack([k[S:], v[S:]]) for k, v in kv])]


def _decode_work(c):
    W, q, kv, weights = _qwen2_sizes(c)
    steps, mean = c["tokens"] - 1, c["context"] + c["tokens"] / 2
    return dict(bytes=2.0 * c["tokens"] * VOCAB * W + 2.0 * steps * (weights + c["layers"] * 2 * mean * kv),
                flops=2.0 * steps * (weights + c["layers"] * 2 * mean * q) + 2.0 * c["tokens"] * VOCAB * W)


# ---- a whole token-id model in the engine ------------------------------------------------------------------
def _serve_model(c, seed):
    from vila_b200.model import BivizenConfig, BivizenForCausalLM
    W = c["width"]
    H = W // 128
    ff = {"ff": 4 * W * 2 // 3 // 64 * 64, "kind": "dense", "limit": 7.0}
    att = {"dim": 128, "heads": H, "kv_heads": H // 4, "rot": {"base": 500000.0, "dims": 128}, "scale": 128 ** -0.5, "softcap": 30.0,
           "v_mix": True, "vdim": 128}
    gla = {"dim": 128, "heads": H, "tau": 8.0, "vdim": 128}
    delta = {"conv": 4, "dim": 128, "heads": H, "kv_heads": H // 2, "vdim": 128}
    layers = [{"type": t, "mixer": dict(m), "mlp": dict(ff)} for t, m in (("attention", att), ("gla", gla), ("delta", delta), ("attention", att))]
    cfg = {"architecture": "Bivizen", "layers": layers, "norm": {"eps": EPS}, "vocab": 32768, "width": W}
    s = State()
    s.config = cfg
    s.model = BivizenForCausalLM(BivizenConfig.from_dict(cfg), DEV, BF).init_random(seed, on_device=True)
    g = torch.Generator().manual_seed(seed)
    s.tokens = torch.randint(0, 32768, (c["seqs"], c["rows"] + c["steps"]), generator=g)
    return s


def _serve_prepare(c, seed):
    from vila_b200.serving import TokenEngine
    s = _serve_model(c, seed)
    n, S = c["seqs"], c["rows"]
    s.engine = TokenEngine(s.model, max_tokens=n * (S + c["steps"] + PAGE), slots=n)
    prompts = [(i, s.tokens[i, :S].tolist(), [S - 1]) for i in range(n)]
    steps = [[(i, [int(s.tokens[i, S + k])], [0]) for i in range(n)] for k in range(c["steps"])]

    def step(s):
        for i in range(n):
            s.engine.release(i)
        return torch.stack([s.engine.step(prompts)] + [s.engine.step(e) for e in steps])
    s.step = step
    s.step(s)   # the engine captures its decode graph while it serves
    return s


def _serve_exact(c, seed):
    s = _serve_model(c, seed)
    w = {k: v.to(DEV).double() for k, v in s.model.weights.items()}
    B, T = s.tokens.shape
    x, v_first, pos = w["embed"][s.tokens.to(DEV)], None, torch.arange(T, device=DEV)
    conv = lambda u, k: F.conv1d(F.pad(u.transpose(1, 2), (k.shape[1] - 1, 0)), k[:, None], groups=u.shape[2]).transpose(1, 2)
    for i, spec in enumerate(s.config["layers"]):
        m, p, q_ = spec["mixer"], f"l{i}.", f"l{i}.mix."
        H, D = m["heads"], 128
        h = _rms(x, EPS) * w[p + "norm1"]
        lin = lambda n: h @ w[q_ + n].T
        if spec["type"] == "attention":
            q, k, v = (lin(n) + w[q_ + n + ".b"] for n in "qkv")
            q, k, v = q.view(B, T, H, D), k.view(B, T, -1, D), v.view(B, T, -1, D)
            if v_first is None:
                v_first = v
            else:
                v = (1 - w[q_ + "vmix"]) * v + w[q_ + "vmix"] * v_first
            q, k = (torch.stack([_rotate(u[b], pos, D, 500000.0, True) for b in range(B)]) for u in (q, k))
            k, v = (u.repeat_interleave(H // u.shape[2], 2) for u in (k, v))
            sc = 30.0 * torch.tanh(torch.einsum("bihd,bjhd->bhij", q, k) * D ** -0.5 / 30.0)
            sc = sc.masked_fill(pos[None, :] > pos[:, None], float("-inf"))
            o = torch.einsum("bhij,bjhd->bihd", torch.softmax(sc, -1), v) * _sigmoid(lin("g"))[..., None]
        else:
            if spec["type"] == "delta":
                q, k, v = (_silu(conv(lin(n), w[q_ + n + ".conv"])) for n in "qkv")
                q, k = (u.view(B, T, H // 2, D).repeat_interleave(2, 2) for u in (q, k))
                q, k = (u / torch.sqrt(u.pow(2).sum(-1, keepdim=True) + 1e-6) for u in (q, k))
                v, beta = v.view(B, T, H, D), _sigmoid(lin("b"))
                keep = torch.exp(-torch.exp(w[q_ + "A_log"]) * F.softplus(lin("a") + w[q_ + "dt_bias"]))[..., None].expand(B, T, H, D)
            else:
                q, k, v = (lin(n).view(B, T, H, D) for n in "qkv")
                keep = _sigmoid(lin("a1") @ w[q_ + "a2"].T + w[q_ + "a2.b"]).pow(1 / 8.0).view(B, T, H, D)
                beta = None
            S, o = torch.zeros(B, H, D, D, device=DEV, dtype=torch.float64), torch.empty(B, T, H, D, device=DEV, dtype=torch.float64)
            for t in range(T):
                S = keep[:, t, ..., None] * S
                u = v[:, t] if beta is None else beta[:, t, :, None] * (v[:, t] - torch.einsum("bhde,bhd->bhe", S, k[:, t]))
                S = S + k[:, t, ..., None] * u[:, :, None]
                o[:, t] = torch.einsum("bhde,bhd->bhe", S, q[:, t]) * D ** -0.5
            nw = w[q_ + "norm"]
            o = _rms(o, EPS) * nw * _silu(lin("g")).view(B, T, H, D)
        y = o.reshape(B, T, -1) @ w[q_ + "o"].T * w[p + "ls1"]
        g = torch.clamp_max(h @ w[p + "mlp.gate"].T, 7.0)
        u = torch.clamp(h @ w[p + "mlp.up"].T, -7.0, 7.0)
        x = x + y + (g * _sigmoid(1.702 * g) * (u + 1)) @ w[p + "mlp.down"].T * w[p + "ls2"]
    z = _rms(x[:, c["rows"] - 1:], EPS) * w["final.norm"] @ w["head"].T
    return z.transpose(0, 1)


def _serve_work(c):
    W, V = c["width"], 32768
    ff = 4 * W * 2 // 3 // 64 * 64
    per = 4 * 3 * ff * W + 2 * int(2.5 * W) * W + 2 * 5 * W * W
    passes, rows = c["steps"] + 1, c["seqs"] * (c["rows"] + c["steps"])
    return dict(bytes=2.0 * passes * (per + V * W) + 4.0 * passes * c["seqs"] * V,
                flops=2.0 * rows * per + 2.0 * passes * c["seqs"] * V * W + 4.0 * c["seqs"] * c["rows"] ** 2 * W)


# ---- routed experts ------------------------------------------------------------------------------------------
LIMIT = 7.0


def _experts_inputs(c, seed):
    g, s = _gen(seed), State()
    R, W, E, f = c["rows"], c["width"], c["experts"], c["ff"]
    s.h = _randn(g, R, W)
    s.x = torch.randn(R, W, generator=g, device=DEV)
    s.router = torch.randn(E, W, generator=g, device=DEV) * W ** -0.5
    s.correction = torch.randn(E, generator=g, device=DEV) * 0.02
    s.up = torch.empty(E, 2 * f, W, device=DEV, dtype=BF)     # rows gate_0, up_0, gate_1, ...
    s.down = torch.empty(E, W, f, device=DEV, dtype=BF)
    for e in range(E):
        s.up[e] = _randn(g, 2 * f, W, std=W ** -0.5)
        s.down[e] = _randn(g, W, f, std=f ** -0.5)
    return s


def _experts_prepare(c, seed):
    from vila_b200 import ops
    s = _experts_inputs(c, seed)
    top, E = c["top"], c["experts"]

    def step(s):
        idx, wt = ops.moe_route_sigmoid(s.h, s.router, s.correction, top, 4, 2)
        seg, srt = ops.moe_group(idx, E)
        act = ops.glinear(s.h, s.up, groups=E, seg=seg, a_rows=srt, a_row_div=top, glu_clamp=(1.702, LIMIT))
        part = ops.glinear(act, s.down, groups=E, seg=seg, o_rows=srt, row_scale=wt.view(-1), out_dtype=torch.float32,
                           out_rows_total=c["rows"] * top)
        ops.residual_add_rows(s.x, part=part, n_partials=top)
        return [idx, part, s.x]
    s.step = _captured(lambda: step(s)) if c["rows"] <= 16 else step
    if c["rows"] <= 16:
        s.x.copy_(_experts_inputs(c, seed).x)   # what the capture's trial run added
    return s


def _experts_exact(c, seed):
    s = _experts_inputs(c, seed)
    R, E, top = c["rows"], c["experts"], c["top"]
    h = s.h.double()
    score = _sigmoid(h @ s.router.double().T)
    choice = score + s.correction.double()
    best = choice.view(R, 4, E // 4).topk(2, -1).values.sum(-1).topk(2, -1).indices
    barred = torch.ones(R, 4, dtype=torch.bool, device=DEV).scatter_(1, best, False)
    idx = choice.masked_fill(barred.repeat_interleave(E // 4, 1), float("-inf")).topk(top, -1).indices
    wt, part = score.gather(1, idx), torch.zeros(R, top, c["width"], device=DEV, dtype=torch.float64)
    for e in range(E):
        r, j = (idx == e).nonzero(as_tuple=True)
        z = h[r] @ s.up[e].double().T
        gt, u = torch.clamp_max(z[:, 0::2], LIMIT), torch.clamp(z[:, 1::2], -LIMIT, LIMIT)
        part[r, j] = (gt * _sigmoid(1.702 * gt) * (u + 1)) @ s.down[e].double().T * wt[r, j][:, None]
    return [None, part.view(R * top, -1), s.x.double() + part.sum(1)]


def _experts_work(c):
    R, W, E, f, top = (c[k] for k in ("rows", "width", "experts", "ff", "top"))
    hit = E * (1 - (1 - top / E) ** R)
    return dict(bytes=2.0 * hit * 3 * f * W + 4.0 * E * W + R * W * (2 + 8) + R * top * W * 4.0, flops=2.0 * R * top * 3 * f * W + 2.0 * R * E * W)


# ---- attention over the paged pool -----------------------------------------------------------------------------
ATT = {  # rotated columns, base, pairing; what each form adds
    "capped": dict(dim=128, rot=128, base=500000.0, halves=True),
    "talk": dict(dim=128, rot=64, base=10000.0, halves=False),
    "window": dict(dim=128, rot=128, base=10000.0, halves=True, window=1024, keep=64),
    "chunk": dict(dim=128, rot=0, base=1.0, halves=False, chunk=512),
    "diff": dict(dim=64, rot=64, base=10000.0, halves=True, window=1024),
}
VDIM = 128
DIFF = (0.45, 0.6, 1e-5)


def _attention_inputs(c, seed):
    g, s, z = _gen(seed), State(), ATT[c["form"]]
    B, n, ctx, H, G = (c[k] for k in ("seqs", "rows", "context", "heads", "kv_heads"))
    maps = 2 if c["form"] == "diff" else 1
    D, T, pages = z["dim"], B * n, (ctx + n + PAGE - 1) // PAGE
    s.width = (H + G) * maps * D + (0 if c["form"] == "chunk" else G * VDIM)
    s.qkv = _randn(g, T, s.width + 8)[:, :s.width]
    s.gate = _randn(g, T, H)
    s.pool = _randn(g, B * pages * PAGE, G * (maps * D + VDIM))
    s.tables = torch.randperm(B * pages, generator=g, device=DEV).to(torch.int32).view(B, pages)
    s.pos = (ctx + torch.arange(n, device=DEV, dtype=torch.int32)).repeat(B)
    s.slot = torch.arange(B, device=DEV).repeat_interleave(n)
    s.rows = (s.tables[s.slot, (s.pos // PAGE).long()] * PAGE + s.pos % PAGE).to(torch.int32)
    tile = 1 if n == 1 else 16
    s.tiles = torch.tensor([(b * n + o, min(tile, n - o), ctx + o, b) for b in range(B) for o in range(0, n, tile)], dtype=torch.int32, device=DEV)
    s.inv = (z["base"] ** (-2.0 * torch.arange(z["rot"] // 2, device=DEV, dtype=torch.float64) / z["rot"])) if z["rot"] else None
    s.talk = torch.eye(H, device=DEV) * 0.8 + torch.randn(H, H, generator=g, device=DEV) * 0.4 * H ** -0.5
    s.sink = torch.randn(H, generator=g, device=DEV)
    s.temp = _rand(g, H, lo=0.7, hi=1.3)
    s.qn, s.kn = (1 + 0.1 * torch.randn(D, generator=g, device=DEV) for _ in range(2))
    s.bias = torch.randn(512, H, generator=g, device=DEV) * 0.5
    return s


def _attention_prepare(c, seed):
    from vila_b200 import ops
    s, z, form = _attention_inputs(c, seed), ATT[c["form"]], c["form"]
    head = dict(heads=c["heads"], kv_heads=c["kv_heads"], dim=z["dim"], vdim=VDIM)
    add = dict(unit_norm=form in ("talk", "chunk"), eps=EPS, halves=z["halves"])
    kw = dict(scale=z["dim"] ** -0.5)
    if form == "capped":
        kw.update(softcap=30.0, gate=s.gate)
    elif form == "talk":
        kw.update(talk=s.talk, sink=s.sink)
    elif form == "window":
        kw.update(talk=s.talk, talk_after=True, head_scale=s.temp, window=z["window"], keep_first=z["keep"])
    elif form == "chunk":
        add.update(q_norm_w=s.qn, k_norm_w=s.kn, v_from_k=True)
        kw.update(sink=s.sink, dist_bias=s.bias, chunk=z["chunk"], gate=s.gate)
    else:
        add.update(maps=2)
        kw.update(window=z["window"], diff=DIFF, gate=s.gate)
    decode = c["rows"] == 1
    see = z.get("window", 0) + z.get("keep", 0)
    splits = min(16, max(1, s.pool.shape[0] // 256))   # as HybridCache deals the keys of decoded tokens
    if see:
        splits = min(splits, (see + 63) // 64)

    def step(s):
        q = ops.rope_append(s.qkv, s.pos, s.rows, s.pool, inv_freq=s.inv, **head, **add)
        o = ops.paged_attention(q, s.pool, s.tables, s.tiles, page=PAGE, max_rows=1 if decode else 16, nsplit=splits if decode else 1,
                                out_dtype=BF, **head, **kw)
        return [o, s.pool]
    s.step = _captured(lambda: step(s)) if decode else step
    return s


def _attention_exact(c, seed):
    s, z, form = _attention_inputs(c, seed), ATT[c["form"]], c["form"]
    B, n, ctx, H, G, D = c["seqs"], c["rows"], c["context"], c["heads"], c["kv_heads"], z["dim"]
    maps = 2 if form == "diff" else 1
    T, rep = B * n, H // G
    x = s.qkv.double()
    q, k = x[:, :H * maps * D].reshape(T, H * maps, D), x[:, H * maps * D:(H + G) * maps * D].reshape(T, G * maps, D)
    v = k if form == "chunk" else x[:, (H + G) * maps * D:].reshape(T, G, VDIM)
    if z["rot"]:
        q, k = (_rotate(u, s.pos, z["rot"], z["base"], z["halves"]) for u in (q, k))
    if form in ("talk", "chunk"):
        q, k = _rms(q, EPS), _rms(k, EPS)
    if form == "chunk":
        q, k = q * s.qn.double(), k * s.kn.double()
    pool = s.pool.double()
    pool[s.rows.long()] = torch.cat([k.reshape(T, -1), v.reshape(T, -1)], 1)
    out = torch.empty(T, H, VDIM, device=DEV, dtype=torch.float64)
    j = torch.arange(ctx + n, device=DEV)
    for b in range(B):
        at = s.tables[b, (j // PAGE)].long() * PAGE + j % PAGE
        kb, vb = pool[at, :G * maps * D].view(-1, G, maps, D), pool[at, G * maps * D:].view(-1, G, VDIM)
        qb = q[b * n:(b + 1) * n].view(n, H, maps, D)
        gate = _sigmoid(s.gate[b * n:(b + 1) * n].double())
        for r in range(0, n, 256):
            i = ctx + torch.arange(r, min(n, r + 256), device=DEV)
            qi, gi = qb[r:r + 256], gate[r:r + 256]
            back = i[:, None] - j[None]
            hide = back < 0
            if "window" in z:
                hide = hide | ((back >= z["window"]) & (j[None] >= z.get("keep", 0)))
            if "chunk" in z:
                hide = hide | (j[None] < (i[:, None] // z["chunk"]) * z["chunk"])
            sc = torch.einsum("ihmd,jhmd->hmij", qi, kb.repeat_interleave(rep, 1)) * D ** -0.5
            if form == "diff":
                a = torch.einsum("hmij,jhd->ihmd", torch.softmax(sc.masked_fill(hide, float("-inf")), -1), vb.repeat_interleave(rep, 1))
                o = _rms(a[:, :, 0] - DIFF[0] * a[:, :, 1], DIFF[2]) * DIFF[1] * gi[..., None]
            else:
                sc = sc[:, 0]
                if form == "capped":
                    sc = 30.0 * torch.tanh(sc / 30.0)
                if form == "talk":
                    sc = torch.einsum("hg,gij->hij", s.talk.double(), sc)
                if form == "window":
                    sc = sc * s.temp.double()[:, None, None]
                if form == "chunk":
                    sc = sc + s.bias.double().T[:, back.clamp(0, 511)]
                sc = sc.masked_fill(hide, float("-inf"))
                if form in ("talk", "chunk"):
                    p = torch.softmax(torch.cat([sc, s.sink.double()[:, None, None].expand(H, len(i), 1)], -1), -1)[..., :-1]
                else:
                    p = torch.softmax(sc, -1)
                if form == "window":
                    p = torch.einsum("hg,gij->hij", s.talk.double(), p)
                o = torch.einsum("hij,jhd->ihd", p, vb.repeat_interleave(rep, 1))
                if form in ("capped", "chunk"):
                    o = o * gi[..., None]
            out[b * n + r:b * n + r + len(i)] = o
    return [out.view(T, -1), pool]


def _attention_work(c):
    z, (B, n, ctx, H, G) = ATT[c["form"]], (c[k] for k in ("seqs", "rows", "context", "heads", "kv_heads"))
    maps = 2 if c["form"] == "diff" else 1
    row = G * (maps * z["dim"] + VDIM)
    pairs, seen = 0, set()
    for p in range(ctx, ctx + n):
        lo = (p // z["chunk"]) * z["chunk"] if "chunk" in z else max(0, p - z["window"] + 1) if "window" in z else 0
        pairs += p + 1 - lo + min(lo, z.get("keep", 0))
    first = max(0, ctx - z["window"] + 1) if "window" in z else (ctx // z["chunk"]) * z["chunk"] if "chunk" in z else 0
    keys = ctx + n - first + min(first, z.get("keep", 0))
    return dict(bytes=2.0 * B * (keys + n) * row + 2.0 * B * n * ((H + G) * maps * z["dim"] + H * VDIM),
                flops=2.0 * B * pairs * H * (maps * z["dim"] + maps * VDIM))


# ---- recurrent mixers ----------------------------------------------------------------------------------------
def _scan_inputs(c, seed):
    g, s, form = _gen(seed), State(), c["form"]
    B, n, W = c["seqs"], c["rows"], c["width"]
    T, H = B * n, W // 128
    s.seqs = torch.tensor([(b * n, n, c["context"], b) for b in range(B)], dtype=torch.int32, device=DEV)
    if form == "ssd":
        s.H, s.P, s.N, s.G = 2 * W // 64, 64, 128, 8
        s.u = _silu(torch.randn(T, 2 * W + 2 * s.G * s.N, generator=g, device=DEV)).to(BF)   # x | B | C behind their convolution
        wide = _randn(g, T, 2 * W + s.H)
        s.z, s.dt = wide[:, :2 * W], wide[:, 2 * W:]
        s.dt_bias = _rand(g, s.H, lo=-4.6, hi=-2.3)
        s.A_log = torch.log(_rand(g, s.H, lo=1.0, hi=16.0))
        s.D = 1 + 0.1 * torch.randn(s.H, generator=g, device=DEV)
        shape = (s.H, s.P, s.N)
    else:
        s.H, shape = H, (H, 128, 128)
        s.u = _randn(g, T, 4 * W)
        s.decay = torch.tensor([1.0 - 2.0 ** (-1.0 - 9.0 * i / H) for i in range(H)], device=DEV)
        s.bias = 1 + torch.randn(W, generator=g, device=DEV)
        s.lower = _rand(g, W, lo=0.0, hi=0.9)
        s.ab = _randn(g, T, 2 * H)
        s.A_log, s.dt_bias = torch.log(_rand(g, H, lo=1.0, hi=8.0)), _rand(g, H, lo=-4.6, hi=-2.3)
    s.state = torch.randn(B, *shape, generator=g, device=DEV)
    return s


def _scan_prepare(c, seed):
    from vila_b200 import ops
    s, form, W = _scan_inputs(c, seed), c["form"], c["width"]
    hd = dict(heads=s.H, dim=128, vdim=128)

    def step(s):
        part = [s.u[:, i * W:(i + 1) * W] for i in range(4)] if form != "ssd" else None
        if form == "ssd":
            o = ops.ssd_scan(s.u, s.dt, s.z, s.state, s.seqs, heads=s.H, vdim=s.P, nstate=s.N, groups=s.G, dt_bias=s.dt_bias,
                             A_log=s.A_log, D=s.D)
        elif form == "decay":
            o = ops.decay_scan(*part[:3], s.state, s.seqs, decay=s.decay, silu=True, **hd)
        elif form == "gla":
            o = ops.gla_scan(*part, s.state, s.seqs, q_scale=128 ** -0.5, tau=8.0, z_bias=s.bias, **hd)
        elif form == "delta":
            o = ops.delta_scan(s.u[:, :2 * W], s.ab[:, :s.H], s.ab[:, s.H:], s.state, s.seqs, kv_heads=s.H // 2, A_log=s.A_log,
                               dt_bias=s.dt_bias, q_scale=128 ** -0.5, **hd)
        else:
            o = ops.hgrn2_scan(s.u, s.state, s.seqs, q_off=0, f_off=W, v_off=2 * W, f_bias=s.bias, lower=s.lower, **hd)
        return [o, s.state]
    if c["rows"] == 1:
        s.step = _captured(lambda: step(s))
        s.state.copy_(_scan_inputs(c, seed).state)   # what the capture's trial run advanced
    else:
        s.step = step
    return s


def _scan_exact(c, seed):
    s, form, W, B, n = _scan_inputs(c, seed), c["form"], c["width"], c["seqs"], c["rows"]
    u, H = s.u.double().view(B, n, -1), s.H
    head = lambda t: t.reshape(B, n, -1, 128)
    beta = extra = None
    scale = 1.0
    if form == "ssd":
        P, N, G = s.P, s.N, s.G
        x, k, q = u[..., :2 * W].view(B, n, H, P), u[..., 2 * W:2 * W + G * N].view(B, n, G, N), u[..., 2 * W + G * N:].view(B, n, G, N)
        k, q = (t.repeat_interleave(H // G, 2) for t in (k, q))
        dt = F.softplus(s.dt.double().view(B, n, H) + s.dt_bias.double())
        keep = torch.exp(-torch.exp(s.A_log.double()) * dt)[..., None].expand(B, n, H, N)
        v, extra = x * dt[..., None], s.D.double()[:, None] * x
    elif form == "decay":
        q, k, v = (head(_silu(u[..., i * W:(i + 1) * W])) for i in range(3))
        keep = s.decay.double()[:, None].expand(B, n, H, 128)
    elif form == "gla":
        q, k, v = (head(u[..., i * W:(i + 1) * W]) for i in range(3))
        keep, scale = head(_sigmoid(u[..., 3 * W:] + s.bias.double()).pow(1 / 8.0)), 128 ** -0.5
    elif form == "delta":
        q, k = (head(u[..., i * W // 2:(i + 1) * W // 2]).repeat_interleave(2, 2) for i in range(2))
        q, k = (t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        v, scale = head(u[..., W:2 * W]), 128 ** -0.5
        a, beta = s.ab[:, :H].double().view(B, n, H), _sigmoid(s.ab[:, H:].double()).view(B, n, H)
        keep = torch.exp(-torch.exp(s.A_log.double()) * F.softplus(a + s.dt_bias.double()))[..., None].expand(B, n, H, 128)
    else:
        q, v = head(_silu(u[..., :W])), head(u[..., 2 * W:3 * W])
        lo = s.lower.double()
        keep = head(lo + (1 - lo) * _sigmoid(u[..., W:2 * W] + s.bias.double()))
        k = 1 - keep
    S = s.state.double()                       # [B, H, vdim, dim], hgrn2: [B, H, dim, vdim]
    S = S if form == "hgrn2" else S.transpose(2, 3)
    S = S * (1.0 if c["context"] else 0.0)
    o = torch.empty(B, n, H, v.shape[-1], device=DEV, dtype=torch.float64)
    for t in range(n):
        S = keep[:, t, ..., None] * S
        w = v[:, t] if beta is None else beta[:, t, :, None] * (v[:, t] - torch.einsum("bhde,bhd->bhe", S, k[:, t]))
        S = S + k[:, t, ..., None] * w[:, :, None]
        o[:, t] = torch.einsum("bhde,bhd->bhe", S, q[:, t]) * scale
    if form == "ssd":
        o = (o + extra) * _silu(s.z.double()).view(B, n, H, s.P)
    return [o.reshape(B * n, -1), (S if form == "hgrn2" else S.transpose(2, 3)).contiguous()]


def _scan_work(c):
    W, T = c["width"], c["seqs"] * c["rows"]
    state = 2 * W * 128 if c["form"] == "ssd" else W * 128
    cols = {"ssd": 4 * W + 2 * 1024, "decay": 3 * W, "gla": 4 * W, "delta": 2 * W, "hgrn2": 3 * W}[c["form"]]
    out = 2 * W if c["form"] == "ssd" else W
    return dict(bytes=T * (2.0 * cols + 4 * out) + c["seqs"] * state * (8.0 if c["context"] else 4.0),
                flops=(6.0 if c["form"] == "delta" else 4.0) * T * state)


# ---- output head -----------------------------------------------------------------------------------------------
def _head_inputs(c, seed):
    g, s = _gen(seed), State()
    s.x = torch.randn(c["rows"], c["width"], generator=g, device=DEV) * 3
    s.norm = 1 + 0.1 * torch.randn(c["width"], generator=g, device=DEV)
    s.w = _randn(g, c["vocab"], c["width"], std=c["width"] ** -0.5)
    return s


def _head_prepare(c, seed):
    from vila_b200 import ops
    s = _head_inputs(c, seed)

    def step(s):
        return ops.glinear(ops.rmsnorm_rows(s.x, s.norm, EPS, out_dtype=BF), s.w, out_dtype=torch.float32)
    s.step = _captured(lambda: step(s))
    return s


def _head_exact(c, seed):
    s = _head_inputs(c, seed)
    return _rms(s.x.double(), EPS) * s.norm.double() @ s.w.double().T


def _head_work(c):
    return dict(bytes=2.0 * c["vocab"] * c["width"] + 4.0 * c["rows"] * (c["width"] + c["vocab"]), flops=2.0 * c["rows"] * c["vocab"] * c["width"])


# ---- the interface -----------------------------------------------------------------------------------------------
_PREPARE = dict(vision=_vision_prepare, prefill=_prefill_prepare, decode=_decode_prepare, serve=_serve_prepare, experts=_experts_prepare,
                attention=_attention_prepare, scan=_scan_prepare, head=_head_prepare)
_EXACT = dict(vision=_vision_exact, prefill=_prefill_exact, decode=_decode_exact, serve=_serve_exact, experts=_experts_exact,
              attention=_attention_exact, scan=_scan_exact, head=_head_exact)
_WORK = dict(vision=_vision_work, prefill=_prefill_work, decode=_decode_work, serve=_serve_work, experts=_experts_work,
             attention=_attention_work, scan=_scan_work, head=_head_work)


def prepare(case, seed):
    gc.collect()   # a graph that dies while another is captured would end the capture
    with torch.no_grad():
        return _PREPARE[case["part"]](case, int(seed) % (1 << 30))


def run(state):
    return state.step(state)


def work(case):
    return _WORK[case["part"]](case)


# About four times the distance between a path's results and exact(): bf16 roundings between the layers (vision, prefill,
# decode, serve), of one operand or of the output (experts, attention, head), fp32 sums of up to thousands of terms (scan).
_REL = dict(vision=0.025, prefill=0.03, decode=0.022, serve=0.028, experts=0.007, attention=0.008, scan=4e-6, head=0.007)


def tolerance(case):
    return {"rel": _REL[case["part"]]}


def exact(case, seed):
    with torch.no_grad():
        return _EXACT[case["part"]](case, int(seed) % (1 << 30))
