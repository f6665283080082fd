"""One cached step against the prompt kernels: the logits behind token n + 1 are the same whether that token comes as a
step or as the end of a prompt.  The two ways share no attention, norm or GEMM kernel.

Query and key weights are scaled up so that a few keys decide; which ones is left to chance, so that these tests see the
kernels' sums and sizes, not every key.  That each cached key is seen, and none behind the new token, is what
test_each_cached_key asks, against a plain restatement.  Both ways round the same values to bf16 (2^-9 each) in another order: after
one or two layers logits differ by some 2^-7 of their scale, and 2^-5 is asked for.
"""
import numpy as np
import pytest

from conftest import cg

gpu = pytest.mark.gpu
synth = cg.synth


def shape(D, nh, nkv, hidden=256, ffn=512, layers=1, arch="llama", **kw):
    return synth.ModelConfig("step", hidden, ffn, layers, nh, nkv, 512, head_dim=D, rms_norm_eps=1e-5, rope_theta=10000.0,
                             tie_word_embeddings=True, dtype="bf16", arch=arch, **kw)


def check(C, cfg, batch, lengths, max_seq, spread=12.0):
    dec = cg.Decoder(C, cfg, max_seq=max_seq, max_batch=batch)
    for name, w in synth.make_weights(cfg, 0):
        dec.set_param(name, C.from_numpy(w * np.float32(spread if "q_proj" in name or "k_proj" in name else 1.0)))
    dec.finalize()
    for n in lengths:
        ids = synth.make_tokens(cfg, batch, n + 1, seed=n)
        dec.reset()
        want = C.to_numpy(dec.prefill(C.from_numpy(ids), want_logits=True))
        dec.reset()
        dec.prefill(C.from_numpy(ids[:, :n].copy()))
        got = C.to_numpy(dec.step_with(C.from_numpy(ids[:, n].copy()), want_logits=True))
        assert np.isfinite(got).all()
        err = np.abs(got - want).max() / np.abs(want).max()
        assert err <= 2.0 ** -5, (n, err)
    dec.close()


# cached keys around a warp's chunk (16 or 32), all warps' chunks (64 or 128) and a slice
EDGES = [1, 15, 16, 31, 32, 33, 63, 64, 127, 128, 129, 255, 256, 300]


@gpu
@pytest.mark.parametrize("D,nh,nkv", [(64, 1, 1), (64, 6, 2), (64, 8, 1), (128, 2, 2), (128, 8, 1), (256, 2, 1), (256, 8, 1)])
@pytest.mark.parametrize("batch,max_seq", [(1, 310), (1, 4200), (2, 600), (40, 310), (230, 310)])
def test_attention_edges(cuda_bf16, D, nh, nkv, batch, max_seq):
    """1 to 16 slices of the context, most of them empty where the context is short; few CTAs and more than fit at once."""
    check(cuda_bf16, shape(D, nh, nkv), batch, EDGES if batch < 40 else [1, 15, 16, 33, 65, 129, 300], max_seq)


SOUGHT, STALE, ASKS, BOTH = range(508, 512)   # tokens: two whose keys stand out, one whose query looks for them, one with both


def seeking(cfg):
    """Weights under which ASKS and BOTH attend to SOUGHT, STALE and BOTH alone, wherever they stand: queries and keys have one component, of
    the pair that turns by less than 0.03 within 310 positions."""
    W = {n: w.astype(np.float64) for n, w in synth.make_weights(cfg, 0)}
    D = cfg.head_dim
    e = W["model.embed_tokens.weight"]
    h = {t: e[t] / np.sqrt(np.mean(e[t] ** 2) + cfg.rms_norm_eps) for t in range(508, 512)}
    q, k = (sum(h[t] / (h[t] @ h[t]) for t in ts) for ts in ((ASKS, BOTH), (SOUGHT, STALE, BOTH)))
    for name, row in (("q_proj", 16.0 * D ** 0.5 * q), ("k_proj", k)):
        w = np.zeros_like(W[f"model.layers.0.self_attn.{name}.weight"])
        w[D // 2 - 1::D] = row
        W[f"model.layers.0.self_attn.{name}.weight"] = w
    return {n: synth.bf16_round(w.astype(np.float32)) if w.ndim > 1 else w.astype(np.float32) for n, w in W.items()}


def last_logits(cfg, W, ids, hide=()):
    """Logits behind the last token of ids, one layer, plainly; its attention does not see the places `hide`."""
    D, nh, nkv, n, eps = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, len(ids), cfg.rms_norm_eps
    W = {k.removeprefix("model.layers.0."): v.astype(np.float64) for k, v in W.items()}
    def rms(v, g):
        return v / np.sqrt((v * v).mean(-1, keepdims=True) + eps) * g
    x = W["model.embed_tokens.weight"][ids]
    h = rms(x, W["input_layernorm.weight"])
    angle = np.arange(n)[:, None, None] * cfg.rope_theta ** (-np.arange(0, D, 2) / D)
    def turned(t):
        a, b = t[..., :D // 2], t[..., D // 2:]
        return np.concatenate([a * np.cos(angle) - b * np.sin(angle), b * np.cos(angle) + a * np.sin(angle)], -1)
    q, k, v = (h @ W[f"self_attn.{p}_proj.weight"].T for p in "qkv")
    q, k, v = turned(q.reshape(n, nh, D))[-1], np.repeat(turned(k.reshape(n, nkv, D)), nh // nkv, 1), np.repeat(v.reshape(n, nkv, D), nh // nkv, 1)
    s = np.einsum("hd,jhd->hj", q, k) / D ** 0.5
    s[:, list(hide)] = -np.inf
    p = np.exp(s - s.max(1, keepdims=True))
    x = x[-1] + np.einsum("hj,jhd->hd", p / p.sum(1, keepdims=True), v).reshape(-1) @ W["self_attn.o_proj.weight"].T
    h = rms(x, W["post_attention_layernorm.weight"])
    g = h @ W["mlp.gate_proj.weight"].T
    x = x + (g / (1 + np.exp(-g)) * (h @ W["mlp.up_proj.weight"].T)) @ W["mlp.down_proj.weight"].T
    return rms(x, W["model.norm.weight"]) @ W["model.embed_tokens.weight"].T


def off(got, want):
    return np.abs(got - want).max() / np.abs(want).max()


def sought_at(rng, n, at):
    """n + 1 tokens whose last one asks; the key that it looks for is at `at`, at its own place if that is n."""
    ids = rng.integers(0, 508, n + 1).astype(np.uint32)
    ids[at], ids[n] = SOUGHT, BOTH if at == n else ASKS
    return ids


@pytest.mark.parametrize("D,nh,nkv", [(64, 1, 1), (64, 6, 2), (128, 8, 1), (256, 8, 1)])
@pytest.mark.parametrize("n", [1, 33, 300])
def test_a_key_too_few_or_too_many_would_show(D, nh, nkv, n):
    """With one key hidden, or one more that stands out, logits move by far more than the tolerance."""
    cfg = shape(D, nh, nkv)
    W = seeking(cfg)
    for at in (0, n // 2, n - 1, n):
        ids = sought_at(np.random.default_rng(n), n, at)
        want = last_logits(cfg, W, ids)
        assert off(last_logits(cfg, W, ids, (at,)), want) > 4 * 2.0 ** -5
        more = np.concatenate([[STALE], ids])
        assert off(last_logits(cfg, W, more.astype(np.uint32)), want) > 4 * 2.0 ** -5


@gpu
@pytest.mark.parametrize("D,nh,nkv", [(64, 1, 1), (64, 6, 2), (64, 8, 1), (128, 2, 2), (128, 8, 1), (256, 2, 1), (256, 8, 1)])
@pytest.mark.parametrize("batch,max_seq", [(1, 370), (2, 4200), (11, 4200), (40, 600), (230, 370)])
def test_each_cached_key(cuda_bf16, D, nh, nkv, batch, max_seq):
    """The key that decides stands at another place in every row; what the cache holds behind the new token is keys that would
    decide as well, left by the rows before."""
    C, cfg = cuda_bf16, shape(D, nh, nkv)
    W = seeking(cfg)
    dec = cg.Decoder(C, cfg, max_seq=max_seq, max_batch=batch)
    for name, w in W.items():
        dec.set_param(name, C.from_numpy(w))
    dec.finalize()
    for n in ([15, 33, 128, 300] if batch > 2 else [1, 31, 64, 129, 300]):
        places = np.unique(np.linspace(0, n, max(batch, 4)).astype(int))
        for first in range(0, len(places), batch):
            at = np.resize(places[first:first + batch], batch)
            ids = np.stack([sought_at(np.random.default_rng(int(a)), n, a) for a in at])
            dec.reset()
            dec.prefill(C.from_numpy(np.full((batch, n + 60), STALE, np.uint32)))
            dec.reset()
            dec.prefill(C.from_numpy(ids[:, :n].copy()))
            got = C.to_numpy(dec.step_with(C.from_numpy(ids[:, n].copy()), want_logits=True))
            for r in np.unique(at, return_index=True)[1]:
                assert off(got[r], last_logits(cfg, W, ids[r])) <= 2.0 ** -5, (n, at[r])
            assert all((got[r] == got[r % len(places)]).all() for r in range(len(places), batch))   # the same row, the same logits
    dec.close()


@gpu
@pytest.mark.parametrize("D,cap,window", [(64, 0.0, 40), (128, 0.0, 129), (256, 30.0, 0), (256, 50.0, 100)])
def test_attention_windows_and_soft_caps(cuda_bf16, D, cap, window):
    cfg = shape(D, 4, 2, layers=2, arch="gemma", attn_logit_softcap=cap, sliding_window=window)
    check(cuda_bf16, cfg, 2, [1, 39, 40, 41, 100, 129, 200, 299], 310, spread=6.0)


@gpu
@pytest.mark.parametrize("D,nh,nkv", [(64, 4, 4), (128, 8, 1), (128, 6, 2)])
def test_attention_head_norms(cuda_bf16, D, nh, nkv):
    check(cuda_bf16, shape(D, nh, nkv, arch="qwen3"), 2, [1, 31, 32, 128, 200], 310, spread=1.0)


@gpu
@pytest.mark.parametrize("kind,dk,dv,taps", [("mamba2", 128, 64, 4), ("mamba2", 24, 32, 2), ("mamba2", 128, 128, 3), ("delta", 128, 128, 4),
                                             ("delta", 128, 64, 4), ("delta", 16, 40, 3), ("delta", 40, 24, 2)])
def test_recurrences(cuda_bf16, kind, dk, dv, taps):
    """A block's convolutions: fewer channels than threads and more, values with and without padding."""
    if kind == "mamba2":
        sizes = {"heads": 4, "groups": 2, "state": dk, "vdim": dv, "norm_groups": 2, "conv": taps}
    else:
        sizes = {"heads": 4, "kv_heads": 2, "dim": dk, "vdim": dv, "conv": taps}
    cfg = cg.LayeredConfig("step-recurrent", 128, 512, [cg.LayerSpec(kind, sizes, 256 if kind == "delta" else 0)], None)
    check(cuda_bf16, cfg, 3, [1, 2, 3, 5, 70], 80)


@gpu
@pytest.mark.parametrize("hidden", [256, 2304, 4096, 4104, 8192])
def test_post_norms_of_many_rows(cuda_bf16, hidden):
    """297 rows and more take the residual norms' form for prompts, the step the one for few rows."""
    check(cuda_bf16, shape(64, 2, 1, hidden, 256, 1, arch="gemma"), 3, [99, 120], 130, spread=1.0)


@gpu
@pytest.mark.parametrize("hidden,ffn", [(128, 256), (256, 640), (512, 1024), (1024, 2048), (2048, 1152)])
@pytest.mark.parametrize("batch", [1, 4, 5, 8, 9, 16, 17, 31, 32])
def test_projections_by_slices_and_tokens(cuda_bf16, hidden, ffn, batch):
    """Clusters of 1 to 16 slices along k; 1 to 32 tokens, so a thread finishes 1 to 16 values of a row."""
    check(cuda_bf16, shape(64, hidden // 64, max(1, hidden // 256), hidden, ffn, 2), batch, [3], 8, spread=1.0)
