"""One cached step against the prompt kernels: the logits behind token n + 1 are the same whether that token comes as a
step or as the end of a prompt.  The two ways share no attention, norm or GEMM kernel.

Query and key weights are scaled up so that the scores spread over several units and a key too many or too few
would show.  Both ways round the same values to bf16 (2^-9 each) in another order: after one or two layers logits
differ by some 2^-7 of their scale, and 2^-5 is asked for.
"""
import numpy as np
import pytest

from conftest import cg

pytestmark = pytest.mark.gpu
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


@pytest.mark.parametrize("D,nh,nkv", [(64, 1, 1), (64, 6, 2), (64, 8, 1), (128, 2, 2), (128, 8, 1), (256, 2, 1), (256, 8, 1)])
@pytest.mark.parametrize("batch,max_seq", [(1, 310), (1, 4200), (2, 600), (40, 310), (230, 310)])
def test_attention_edges(cuda_bf16, D, nh, nkv, batch, max_seq):
    """1 to 16 slices of the context, most of them empty where the context is short; few CTAs and more than fit at once."""
    check(cuda_bf16, shape(D, nh, nkv), batch, EDGES if batch < 40 else [1, 15, 16, 33, 65, 129, 300], max_seq)


@pytest.mark.parametrize("D,cap,window", [(64, 0.0, 40), (128, 0.0, 129), (256, 30.0, 0), (256, 50.0, 100)])
def test_attention_windows_and_soft_caps(cuda_bf16, D, cap, window):
    cfg = shape(D, 4, 2, layers=2, arch="gemma", attn_logit_softcap=cap, sliding_window=window)
    check(cuda_bf16, cfg, 2, [1, 39, 40, 41, 100, 129, 200, 299], 310, spread=6.0)


@pytest.mark.parametrize("D,nh,nkv", [(64, 4, 4), (128, 8, 1), (128, 6, 2)])
def test_attention_head_norms(cuda_bf16, D, nh, nkv):
    check(cuda_bf16, shape(D, nh, nkv, arch="qwen3"), 2, [1, 31, 32, 128, 200], 310, spread=1.0)


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


@pytest.mark.parametrize("hidden", [256, 2304, 4096, 4104, 8192])
def test_post_norms_of_many_rows(cuda_bf16, hidden):
    """297 rows and more take the residual norms' form for prompts, the step the one for few rows."""
    check(cuda_bf16, shape(64, 2, 1, hidden, 256, 1, arch="gemma"), 3, [99, 120], 130, spread=1.0)


@pytest.mark.parametrize("hidden,ffn", [(128, 256), (256, 640), (512, 1024), (1024, 2048), (2048, 1152)])
@pytest.mark.parametrize("batch", [1, 4, 5, 8, 9, 16, 17, 31, 32])
def test_projections_by_slices_and_tokens(cuda_bf16, hidden, ffn, batch):
    """Clusters of 1 to 16 slices along k; 1 to 32 tokens, so a thread finishes 1 to 16 values of a row."""
    check(cuda_bf16, shape(64, hidden // 64, max(1, hidden // 256), hidden, ffn, 2), batch, [3], 8, spread=1.0)
