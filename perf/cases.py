"""What a user of this library has it do, as cases to be timed and checked.

Every case is one call of a served model: a prompt batch goes through a decoder and some greedy tokens come
back, with the logits behind the prompt and behind the last token.  The models are the shapes this
repository is benchmarked and tested on (`synth`, `layered`): the whole Llama-3.2-1B shape, slices of the
first layers of the Llama-3-8B, Gemma-2-2B and Qwen3-30B-A3B shapes at full width and vocabulary, and two of the
designs built layer by layer, whose rows may differ in length.  One case replays the reference's own op stream
through the trait methods in f32, as the interpreter does.

Weights are random: matrices N(0, 0.02^2) rounded to bf16 as in the benchmark, but with an embedding of the size
of what a few layers add to it and a head that reads it (the same matrix where the shape ties them, else with
its rows moved on), so that the greedy choice is as clear as a trained model's and a sequence does not depend on
the last bits of a sum.
"""
from __future__ import annotations

import dataclasses
import functools
import importlib
import math
import zlib

import numpy as np
import torch

cg = importlib.import_module("catgrad-rs_b200")
layered = importlib.import_module("catgrad-rs_b200.layered")
synth = cg.synth

MODELS = {
    "llama1b": synth.LLAMA_32_1B,
    "llama8b": dataclasses.replace(synth.LLAMA_3_8B, num_hidden_layers=4),
    "gemma2": dataclasses.replace(synth.GEMMA_2_2B, num_hidden_layers=4),
    "qwen3moe": dataclasses.replace(synth.QWEN3_30B_A3B, num_hidden_layers=4),
    "ralapel": layered.RALAPEL_W2048,
    "segedra": layered.SEGEDRA_W2048,
    "trait": synth.TINY_LLAMA,
}
NEXT = 7919  # an untied head answers token t with t + NEXT


def listed():
    def case(name, model, batch, prompt, decode, ragged=False):
        return {"name": name, "model": model, "batch": batch, "prompt": prompt, "decode": decode, "ragged": ragged}

    return [
        # one chat turn of a small model: launches and latency are all there is
        case("llama1b-turn", "llama1b", 1, 37, 24),
        # the batch the benchmark is quoted on: decode steps that stream the weights
        case("llama1b-batch8", "llama1b", 8, 512, 128),
        # an odd batch of odd prompts, a few tokens each: classification, extraction
        case("llama1b-odd", "llama1b", 13, 389, 5),
        # many users at once on wide layers: the decode GEMMs' largest token count
        case("llama8b-batch32", "llama8b", 32, 509, 48),
        # one long document with a short answer: prompt GEMMs and attention over a long context
        case("llama8b-document", "llama8b", 1, 8191, 8),
        # heads of 256 with capped scores, gelu units, a vocabulary of 256 000
        case("gemma2-batch4", "gemma2", 4, 2048, 64),
        # experts: a batch in which each expert sees a few rows per step, and a single row
        case("qwen3moe-batch8", "qwen3moe", 8, 1024, 48),
        case("qwen3moe-turn", "qwen3moe", 1, 333, 32),
        # recurrent and latent layers in a loop: the benchmark's batch, and rows as requests come in
        case("ralapel-batch8", "ralapel", 8, 512, 64),
        case("ralapel-requests", "ralapel", 5, 300, 16, True),
        # windows, sinks, four residual streams and experts, rows as requests come in
        case("segedra-requests", "segedra", 8, 800, 32, True),
        # the reference's op stream through the trait methods, f32
        case("trait-f32", "trait", 1, 61, 0),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(list(MODELS))
    if model == "trait":
        return {"model": model, "batch": 1, "prompt": spread(17, 160), "decode": 0, "ragged": False}
    batch = spread(1, 32 if model == "llama8b" else 13 if model == "llama1b" else 8)
    most = {"llama1b": 5100, "llama8b": 16000, "gemma2": 8192, "qwen3moe": 8192, "ralapel": 4096, "segedra": 6400}[model]
    longest = min(8191 if model == "llama8b" else 2048, most // batch)
    return {"model": model, "batch": batch, "prompt": spread(24, longest), "decode": spread(4, 64),
            "ragged": model in ("ralapel", "segedra") and rng.random() < 0.5}


# ---------------------------------------------------------------- inputs


def shapes_of(cfg):
    return synth.param_shapes(cfg)


def weight(cfg, name, shape, seed):
    """One tensor of the checkpoint, f32 on the GPU; matrices of bf16 models hold bf16 values."""
    gen = torch.Generator(device="cuda").manual_seed((seed << 20) ^ zlib.crc32(name.encode()))

    def normal(std=1.0, mean=0.0):
        return torch.randn(shape, generator=gen, device="cuda") * std + mean

    design = cfg.design if cfg.arch == "layered" else None
    if name in ("model.embed_tokens.weight", "embed"):
        # scaled up by the model where it says so
        w = normal(0.02 if cfg.arch == "gemma" or (design and cfg.embed_scale != 1.0) else 1.0)
    elif name in ("lm_head.weight", "head"):
        embed = "embed" if design else "model.embed_tokens.weight"
        w = torch.roll(weight(cfg, embed, shape, seed), NEXT % shape[0], 0)
    elif name in ("model.norm.weight", "final.norm"):
        # logits of about one: the head's rows are as long as the embedding's
        w = torch.full(shape, 0.0 if cfg.arch == "gemma" or (design and design.norm_plus_one) else 0.02, device="cuda")
    elif name == "loop.in":
        eye = torch.eye(shape[0], device="cuda") * 0.5   # a pass starts from the mean of its two inputs, nearly
        w = normal(0.002) + torch.cat([eye, eye], 1)
    elif name.endswith((".hc1.mix", ".hc2.mix")):
        w = normal(0.05 / shape[0]) + torch.eye(shape[0], device="cuda")   # streams stay apart, nearly
    elif name.endswith((".hc1.out", ".hc2.out")):
        w = normal(0.2, 1.0)
    elif design:
        mean, std = cfg.synthetic(name)
        w = normal(std, mean)
    elif len(shape) == 1:
        w = torch.full(shape, 0.0 if cfg.arch == "gemma" else 1.0, device="cuda")
    else:
        w = normal(0.02)
    return w.bfloat16().float() if cfg.dtype == "bf16" and len(shape) > 1 else w


def lengths(case):
    """Prompt lengths of the rows."""
    n, B = case["prompt"], case["batch"]
    if not case["ragged"]:
        return [n] * B
    return [max(1, int(n * (0.25 + 0.75 * ((7 * r + 3) % B + 1) / B))) for r in range(B)]


def prompts(case, cfg, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, cfg.vocab_size, n).astype(np.uint32) for n in lengths(case)]


_last = {}


def backend(case):
    """The program's backend; a program of another case has another one, and this one's memory is given back."""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    if _last.get("key") != key:
        if _last:
            _last["backend"].close()
        trait = case["model"] == "trait"
        b = cg.CudaBackend(0, cg.PREC_F32 if trait else cg.PREC_BF16)
        if trait:
            b.set_option("lazy", 1)   # the trait's calls are recorded and run fused, with unchanged results
        _last.update(key=key, backend=b)
    return _last["backend"]


@functools.lru_cache(1)
def staging(n):
    return torch.empty(n, pin_memory=True)


def upload(B, w):
    """The trait's upload of a host array."""
    n = w.numel()
    host = staging(1 << 20 if n <= 1 << 20 else 600_000_000)[:n]
    host.copy_(w.reshape(-1))
    t = B.ndarray_from_vec_f32(host.numpy(), tuple(w.shape))
    B.sync()
    return t


def prepare(case, seed):
    cfg = MODELS[case["model"]]
    B = backend(case)
    rows = prompts(case, cfg, seed)
    named = ((name, weight(cfg, name, shape, seed)) for name, shape in sorted(shapes_of(cfg).items(), key=lambda s: np.prod(s[1])))
    if case["model"] == "trait":
        return {"B": B, "cfg": cfg, "params": {name: upload(B, w) for name, w in named}, "ids": rows[0][None]}
    dec = cg.Decoder(B, cfg, max_seq=case["prompt"] + case["decode"] + 1, max_batch=case["batch"])
    for name, w in named:
        dec.set_param(name, upload(B, w))
    dec.finalize()
    return {"B": B, "dec": dec, "rows": rows, "decode": case["decode"], "ragged": case["ragged"]}


def run(state):
    B = state["B"]
    if "params" in state:
        ids = B.ndarray_from_vec_u32(state["ids"], state["ids"].shape)
        best, logits = cg.graphs.llama.forward(B, state["cfg"], state["params"], ids, ids.shape[1], want_logits=True)
        return {"tokens": B.to_numpy(best).astype(np.int64), "logits": B.to_numpy(logits)}
    dec, rows = state["dec"], state["rows"]
    if state["ragged"]:
        slots = [dec.open_sequence() for _ in rows]
        try:
            first = dec.run(list(zip(slots, rows)), want=[(r, len(t) - 1) for r, t in enumerate(rows)], greedy=True)
            last = dec.decode(state["decode"], want_logits=True)
            tokens = dec.tokens()
        finally:
            for s in slots:
                dec.close_sequence(s)
    else:
        first = dec.prefill(B.from_numpy(np.stack(rows)), want_logits=True)
        last = dec.decode(state["decode"], want_logits=True)
        tokens = dec.tokens()
    return {"tokens": tokens.astype(np.int64), "first": B.to_numpy(first), "last": B.to_numpy(last)}


# ---------------------------------------------------------------- what a pass cannot do without


def matrix_values(cfg, rows):
    """(values of all matrices a step of `rows` tokens reads, values one token is multiplied with); of the experts
    those that independent choices reach."""
    read = used = 0.0
    shapes = shapes_of(cfg)
    if cfg.arch != "layered":
        H = cfg.hidden_size
        for name, s in shapes.items():
            n = float(np.prod(s))
            if ".experts." in name:
                read += n * (1.0 - (1.0 - cfg.num_experts_per_tok / s[0]) ** rows)
                used += n * cfg.num_experts_per_tok / s[0]
            elif len(s) > 1 and name != "model.embed_tokens.weight":
                read, used = read + n, used + n
        tied = cfg.vocab_size * H if cfg.tie_word_embeddings else 0
        return read + tied, used + tied
    for i in cfg.layer_runs():
        e = cfg.layers[i].experts
        for name, s in shapes.items():
            if name.startswith(f"l{i}.") and len(s) > 1:
                n = float(np.prod(s))
                expert = e and ".mlp.e" in name
                read += n * (1.0 - (1.0 - e.top / e.count) ** rows) if expert else n
                used += n * e.top / e.count if expert else n
    extra = cfg.vocab_size * cfg.hidden_size + (cfg.loop[2] * np.prod(shapes["loop.in"]) if "loop.in" in shapes else 0)
    return read + extra, used + extra


def attention_layers(cfg):
    """(query heads, key heads, size of keys, of values, tokens seen) of every layer run with attention."""
    if cfg.arch != "layered":
        seen = [cfg.sliding_window if cfg.sliding_window and i % 2 == 0 else 1 << 30 for i in range(cfg.num_hidden_layers)]
        return [(cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.head_dim, w) for w in seen]
    out = []
    for i in cfg.layer_runs():
        m, kind = cfg.layers[i].sizes, cfg.layers[i].mixer
        if kind == "attention":
            out.append((m["heads"], m["kv_heads"], m["dim"], m["vdim"], cfg.layers[i].window or 1 << 30))
        elif kind == "latent_attention":
            out.append((m["heads"], 1, m["dim"] + m["rot_dim"], m["vdim"], 1 << 30))
    return out


def state_values(cfg):
    """Values of the matrix states of one sequence over all layer runs."""
    if cfg.arch != "layered":
        return 0
    m = [cfg.layers[i].sizes for i in cfg.layer_runs() if cfg.layers[i].mixer in ("delta", "mamba2")]
    return sum(s["heads"] * s["vdim"] * s.get("state", s.get("dim", 0)) for s in m)


def work(case):
    cfg = MODELS[case["model"]]
    lens, T, elem = lengths(case), case["decode"], 4 if case["model"] == "trait" else 2
    B, n = len(lens), sum(lengths(case))
    read_prompt, used = matrix_values(cfg, n)
    read_step, _ = matrix_values(cfg, B)
    head = cfg.vocab_size * cfg.hidden_size
    heads_run = n if case["model"] == "trait" else B
    flops = 2.0 * (used - head) * (n + T * B) + 2.0 * head * (heads_run + T * B)
    cache = 0.0
    for H, G, d, dv, seen in attention_layers(cfg):
        for s in lens:
            pairs = sum(min(p + 1, seen) for p in range(s + T))
            flops += 2.0 * pairs * H * (d + dv)
            cache += elem * G * (d + dv) * (s + sum(min(s + t + 1, seen) for t in range(T)))
    logits = 4.0 * cfg.vocab_size * (n if case["model"] == "trait" else 2 * B)
    states = 4.0 * B * state_values(cfg) * (1 + 2 * T)
    return {"bytes": float(elem * (read_prompt + T * read_step) + cache + states + logits), "flops": float(flops)}


def tolerance(case):
    """Measured against `exact`: 3e-7 in f32; in bf16 0.5 to 0.9 % where layers are dense, 1.0 to 1.3 % where they
    are recurrent and where a token stands between two experts.  Two implementations are off independently."""
    if case["model"] == "trait":
        return {"rel": 2e-6}
    return {"rel": 0.03 if case["model"] in ("ralapel", "segedra", "qwen3moe") else 0.02, "max": 0.25}


# ---------------------------------------------------------------- the same in 64 bits


def rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


silu = torch.nn.functional.silu


def turn_halves(x, base):
    """x [B, T, heads, d]: component i turns with component i + d / 2.  The angles are those of the reference's
    tables, which it makes in 32 bits."""
    T, d = x.shape[1], x.shape[-1]
    inv = 1.0 / torch.pow(torch.tensor(base, dtype=torch.float32), torch.arange(0, d, 2, dtype=torch.float32) / d)
    a = (torch.arange(T, dtype=torch.float32)[:, None] * inv).double().to(x.device)[None, :, None]
    u, v = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def turn_pairs(x, base, dims):
    """x [B, T, heads, d]: of the first `dims` components each turns with its neighbour."""
    a = torch.arange(x.shape[1], device=x.device).double()[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device).double() / dims)
    a = a[None, :, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2), x[..., dims:]], -1)


def attend(q, k, v, scale, window=0, cap=0.0, sink=None):
    """q [B, T, H, d], k, v [B, T, G, d]: causal attention, some heads of one row at a time."""
    B, T, H, _ = q.shape
    per = H // k.shape[2]
    t = torch.arange(T, device=q.device)
    hidden = t[None, :] > t[:, None]
    if window:
        hidden |= t[None, :] <= t[:, None] - window
    out = torch.empty(B, T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    some = max(1, min(H, int(1e9 / 8 / T / T)))
    for b in range(B):
        for lo in range(0, H, some):
            hs = torch.arange(lo, min(H, lo + some), device=q.device)
            s = torch.einsum("thd,jhd->htj", q[b][:, hs], k[b][:, hs // per]) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[hs, None, None].expand(-1, T, 1)], 2)
            s = torch.softmax(s, 2)[..., :T]
            out[b][:, hs] = torch.einsum("htj,jhd->thd", s, v[b][:, hs // per])
    return out


def chosen_experts(scores, top):
    return torch.zeros_like(scores).scatter_(-1, scores.topk(top, -1).indices, 1.0)


def attention_only(cfg, W, x):
    """The layers of the Llama, Qwen3 and Gemma shapes on x [B, T, width]."""
    B, T, _ = x.shape
    H, G, d, eps = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.rms_norm_eps
    gemma = cfg.arch == "gemma"

    def norm(x, name):
        w = W(name)
        return rms(x, eps) * (1.0 + w if gemma else w)

    if gemma:
        x = x * float(np.sqrt(np.float32(cfg.hidden_size)))
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        q, k, v = ((h @ W(p + f"self_attn.{n}_proj.weight").T).view(B, T, -1, d) for n in "qkv")
        if cfg.arch == "qwen3":
            q, k = norm(q, p + "self_attn.q_norm.weight"), norm(k, p + "self_attn.k_norm.weight")
        q, k = turn_halves(q, cfg.rope_theta), turn_halves(k, cfg.rope_theta)
        window = cfg.sliding_window if i % 2 == 0 else 0
        y = attend(q, k, v, d ** -0.5, window, cfg.attn_logit_softcap).flatten(2) @ W(p + "self_attn.o_proj.weight").T
        x = x + (norm(y, p + "post_attention_layernorm.weight") if gemma else y)
        h = norm(x, p + ("pre_feedforward_layernorm.weight" if gemma else "post_attention_layernorm.weight"))
        if cfg.num_local_experts > 1:
            prob = torch.softmax(h @ W(p + "mlp.gate.weight").T, -1)
            prob = prob * chosen_experts(prob, cfg.num_experts_per_tok)
            prob = prob / prob.sum(-1, keepdim=True)
            gate, up, down = (W(p + f"mlp.experts.{n}_proj.weight") for n in ("gate", "up", "down"))
            y = torch.zeros_like(x)
            for e in range(cfg.num_local_experts):
                at = prob[..., e] > 0
                y[at] += prob[..., e][at][:, None] * ((silu(h[at] @ gate[e].T) * (h[at] @ up[e].T)) @ down[e].T)
        else:
            unit = gelu if gemma else silu
            y = (unit(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
        x = x + (norm(y, p + "post_feedforward_layernorm.weight") if gemma else y)
    return norm(x, "model.norm.weight")


def convolved(x, w, bias=None):
    """Causal convolution of every channel of x [B, T, ch] with its taps w [ch, taps], then silu."""
    return silu(torch.nn.functional.conv1d(torch.nn.functional.pad(x.transpose(1, 2), (w.shape[1] - 1, 0)), w[:, None], bias,
                                           groups=w.shape[0]).transpose(1, 2))


def latent(h, P, m, eps):
    B, T, _ = h.shape
    H, d, r, R = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    q, down = (h @ P("q").T).view(B, T, H, d + r), h @ P("dkv").T
    c = rms(down[..., :R], eps) * P("dkv.norm")
    turned = turn_pairs(down[..., None, R:], m["rot"]["base"], r).expand(B, T, H, r)
    q = torch.cat([q[..., :d], turn_pairs(q[..., d:], m["rot"]["base"], r)], -1)
    k = torch.cat([(c @ P("uk").T).view(B, T, H, d), turned], -1)
    return attend(q, k, (c @ P("uv").T).view(B, T, H, -1), m["scale"]).flatten(2) @ P("o").T


def delta(h, P, m, eps):
    B, T, _ = h.shape
    H, K, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (convolved(h @ P(n).T, P(n + ".conv")).view(B, T, -1, s) for n, s in (("q", d), ("k", d), ("v", dv)))
    q, k = (torch.repeat_interleave(x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6), H // K, 2) for x in (q * 1.0, k))
    q = q * d ** -0.5
    beta = torch.sigmoid(h @ P("b").T)[..., None, None]
    decay = torch.exp(-torch.exp(P("A_log")) * torch.nn.functional.softplus(h @ P("a").T + P("dt_bias")))[..., None, None]
    S, out = h.new_zeros(B, H, d, dv), torch.empty_like(v)
    for t in range(T):
        S = decay[:, t] * S
        S = S + k[:, t, :, :, None] @ (beta[:, t] * (v[:, t, :, None] - k[:, t, :, None] @ S))
        out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    return (rms(out, eps) * P("norm") * silu(h @ P("g").T).view(B, T, H, dv)).flatten(2) @ P("o").T


def mamba2(h, P, m, eps):
    B, T, _ = h.shape
    H, dv, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * dv
    z, xbc, dt = (h @ P("in").T).split([inner, inner + 2 * G * N, H], -1)
    x, b, c = convolved(xbc, P("conv"), P("conv.b")).split([inner, G * N, G * N], -1)
    x = x.reshape(B, T, H, dv)
    b, c = (torch.repeat_interleave(y.reshape(B, T, G, N), H // G, 2) for y in (b, c))
    dt = torch.nn.functional.softplus(dt + P("dt_bias"))
    decay = torch.exp(-torch.exp(P("A_log")) * dt)[..., None, None]
    S, y = h.new_zeros(B, H, N, dv), torch.empty_like(x)
    for t in range(T):
        S = decay[:, t] * S + b[:, t, :, :, None] * (dt[:, t, :, None] * x[:, t])[:, :, None]
        y[:, t] = (c[:, t, :, None] @ S)[:, :, 0]
    y = (y + P("D")[:, None] * x).flatten(2) * silu(z)
    return (rms(y.view(B, T, m["norm_groups"], -1), eps).flatten(2) * P("norm")) @ P("o").T


def ralapel(cfg, W, x):
    eps = cfg.rms_norm_eps
    x = x0 = rms(x, eps) * W("embed.norm")
    a, b, times = cfg.loop
    runs = cfg.layer_runs()
    for n, i in enumerate(runs):
        L, p = cfg.layers[i], f"l{i}."
        if a <= n < a + times * (b - a) and i == a:
            x = torch.cat([x, x0], -1) @ W("loop.in").T
        mix = {"latent_attention": latent, "delta": delta, "mamba2": mamba2}[L.mixer]
        y = mix(rms(x, eps) * W(p + "norm1"), lambda n: W(p + "mix." + n), L.sizes, eps)
        x = x + rms(y, eps) * W(p + "norm1b")
        if L.ffn:
            h = rms(x, eps) * W(p + "norm2")
            y = (gelu(h @ W(p + "mlp.gate").T) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T
            x = x + rms(y, eps) * W(p + "norm2b")
    return rms(x, eps) * W("final.norm")


def segedra(cfg, W, x):
    eps = cfg.rms_norm_eps
    B, T, _ = x.shape

    def norm(x, w):
        return rms(x, eps) * (1.0 + w)

    def mixed(h, P, L):
        m = L.sizes
        q, k, v = h @ P("q").T, h @ P("k").T, (h @ P("v").T).view(B, T, m["kv_heads"], m["vdim"])
        q = (rms(q, eps) * P("q.norm")).view(B, T, m["heads"], m["dim"])
        k = (rms(k, eps) * P("k.norm")).view(B, T, m["kv_heads"], m["dim"])
        q, k = (turn_pairs(y, m["rot"]["base"], m["rot"]["dims"]) for y in (q, k))
        return attend(q, k, v, m["scale"], L.window, sink=P("sink")).flatten(2) @ P("o").T

    def fed(h, P, L):
        if not L.experts:
            return torch.relu(h @ P("up").T).square() @ P("down").T
        s = torch.softmax(h @ P("router").T, -1)
        s = s * chosen_experts(s + P("correction"), L.experts.top) * L.experts.scale
        y = torch.zeros_like(h)
        for e in range(L.experts.count):
            at = s[..., e] > 0
            g = (h[at] @ P(f"e{e}.gate").T).clamp(max=L.experts.limit)
            u = (h[at] @ P(f"e{e}.up").T).clamp(-L.experts.limit, L.experts.limit)
            y[at] += s[..., e][at][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ P(f"e{e}.down").T)
        return y

    x = (x * cfg.embed_scale)[None].repeat(cfg.streams, 1, 1, 1)
    for i in cfg.layer_runs():
        L, p = cfg.layers[i], f"l{i}."
        for q, part, f in ((1, "mix.", mixed), (2, "mlp.", fed)):
            u = torch.einsum("s,sbtw->btw", W(p + f"hc{q}.in"), x)
            y = f(norm(u, W(p + f"norm{q}")), lambda n: W(p + part + n), L)
            x = torch.einsum("sr,sbtw->rbtw", W(p + f"hc{q}.mix"), x) + W(p + f"hc{q}.out")[:, None, None, None] * y
    return norm(x.sum(0), W("final.norm"))


def exact_row(cfg, W, ids, T):
    """(tokens [B, 1 + T], logits behind the prompt and behind the last token fed) of prompts ids [B, n]: the whole
    sequence in one pass, repeated until the tokens that it assumed are the ones that it answers with."""
    layered_ = cfg.arch == "layered"
    embed = W("embed" if layered_ else "model.embed_tokens.weight")
    tied = cfg.design.tied_head if layered_ else cfg.tie_word_embeddings
    head = embed if tied else W("head" if layered_ else "lm_head.weight")
    walk = attention_only if not layered_ else ralapel if cfg.loop and "loop.in" in shapes_of(cfg) else segedra
    n = ids.shape[1]
    step = torch.arange(1, T + 1, device=ids.device)
    new = (ids[:, -1:] + (0 if tied else NEXT) * step) % cfg.vocab_size
    for _ in range(T + 1):
        x = walk(cfg, W, embed[torch.cat([ids, new], 1)])[:, n - 1:]
        cap = getattr(cfg, "final_logit_softcap", 0.0)
        logits = [(cap * torch.tanh(y / cap) if cap else y) for y in (x[:, t] @ head.T for t in range(T + 1))]
        said = torch.stack([y.argmax(-1) for y in logits], 1)
        if torch.equal(said[:, :T], new):
            break
        new = said[:, :T]
    return said, logits[0], logits[-1]


def exact(case, seed):
    cfg = MODELS[case["model"]]
    if case["model"] == "ralapel" and case["ragged"] and sum(lengths(case)) > 4000:
        return None   # token after token, row after row
    shapes = shapes_of(cfg)

    @functools.lru_cache(None)
    def kept(name):
        return weight(cfg, name, shapes[name], seed)

    def W(name):
        return kept(name).double()

    rows = [torch.from_numpy(r.astype(np.int64)).cuda()[None] for r in prompts(case, cfg, seed)]
    if case["model"] == "trait":
        x = attention_only(cfg, W, W("model.embed_tokens.weight")[rows[0]])
        logits = x @ W("lm_head.weight").T
        return {"tokens": logits.argmax(-1, keepdim=True), "logits": logits}
    got = [exact_row(cfg, W, r, case["decode"]) for r in (rows if case["ragged"] else [torch.cat(rows)])]
    return {k: torch.cat([g[i] for g in got]) for i, k in enumerate(("tokens", "first", "last"))}
