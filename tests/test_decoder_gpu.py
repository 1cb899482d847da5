"""A Qwen3-shaped dense decoder end to end on the GPU (palm-infra_b200/decoder.py: every
operator a libb200w4 kernel) against the same decoder computed on the CPU from the oracle's
pieces: greedy tokens must be identical over a prompt and a run of decode steps, with the
reference's activation rule (per 128 values for one row, per 32 for the prompt's rows).  The
matmuls are bit-exact on both sides; the norms, the attention scores and the softmax differ by
the rounding of reassociated fp32 sums, so identity rests on the top-1 margins, which the test
prints and requires to be far above that noise."""
import numpy as np
import pytest

import oracle_lib as ol
from __graft_entry__ import load_package

pkg = load_package()
pytestmark = pytest.mark.gpu


# Seeds are chosen on the CPU (the oracle decoder alone) for a comfortable smallest top-1 margin
# over the run: 5e-2 for the 64-step case.
@pytest.mark.parametrize("layers,hidden,heads,kv_heads,head_dim,inter,vocab,prompt_len,steps,"
                         "seed",
                         [(2, 256, 4, 2, 64, 512, 1000, 12, 64, 11),   # 64 greedy steps
                          (3, 512, 8, 2, 128, 1024, 2048, 33, 16, 20261128),
                          # benchmark configuration 3's widths (hidden 2560, 32 / 8 heads of 128,
                          # intermediate 9728, vocabulary 151936) at four layers: what the CPU
                          # decoder finishes in about a minute
                          (4, 2560, 32, 8, 128, 9728, 151936, 8, 6, 20261129)])
def test_greedy_tokens_identical_to_the_cpu_decoder(layers, hidden, heads, kv_heads, head_dim,
                                                   inter, vocab, prompt_len, steps, seed):
    dec = pkg.decoder
    cfg = dec.DecoderConfig(layers, hidden, heads, kv_heads, head_dim, inter, vocab)
    weights = dec.synthetic_weights(cfg, seed=seed)
    prompt = np.random.default_rng(11).integers(0, vocab, prompt_len).tolist()
    ol.set_exp_mode(True)
    try:
        want, margins = ol.dense_decoder_tokens(cfg, weights, prompt, steps)
    finally:
        ol.set_exp_mode(False)
    ctx = pkg.capi.Context(0)
    model = dec.DenseDecoder(ctx, cfg, weights, capacity=prompt_len + steps + 8)
    got = model.generate(prompt, steps)
    replayed = model.generate(prompt, steps, replay=True)  # one captured step, replayed
    model.free()
    model = dec.DenseDecoder(ctx, cfg, weights, capacity=prompt_len + steps + 8, fused_qkv=False)
    unfused = model.generate(prompt, steps)                # operator by operator
    model.free()
    ctx.close()
    print(f"tokens {got}\nminimum top-1 margin {min(margins):.3e}")
    assert got == want, (got, want, margins)
    assert replayed == want, (replayed, want)
    assert unfused == want, (unfused, want)
    assert min(margins) > 1e-2  # identity is not an accident of a near-tie


@pytest.mark.parametrize("layers,hidden,heads,kv_heads,head_dim,inter,vocab,experts,top_k,"
                         "prompt_len,steps,seed",
                         [(2, 256, 4, 2, 64, 128, 1000, 8, 2, 12, 64, 4),   # 64 greedy steps
                          # benchmark configuration 4's widths (hidden 2048, 32 / 4 heads of 128,
                          # 128 experts of width 768, 8 per token) at two layers
                          (2, 2048, 32, 4, 128, 768, 4096, 128, 8, 20, 6, 77 + 128)])
def test_mixture_of_experts_decoder_tokens_identical(layers, hidden, heads, kv_heads, head_dim,
                                                    inter, vocab, experts, top_k, prompt_len,
                                                    steps, seed):
    """The same identity with the MOE operator as the feed-forward block (router, selection,
    expert matmuls under the reference's per-expert activation rule, ordered combine): prompt
    rows give experts several rows each, decode steps one."""
    dec = pkg.decoder
    cfg = dec.DecoderConfig(layers, hidden, heads, kv_heads, head_dim, inter, vocab,
                            experts=experts, top_k=top_k)
    weights = dec.synthetic_weights(cfg, seed=seed)
    prompt = np.random.default_rng(5).integers(0, vocab, prompt_len).tolist()
    ol.set_exp_mode(True)
    try:
        want, margins = ol.dense_decoder_tokens(cfg, weights, prompt, steps)
    finally:
        ol.set_exp_mode(False)
    ctx = pkg.capi.Context(0)
    model = dec.DenseDecoder(ctx, cfg, weights, capacity=prompt_len + steps + 8)
    got = model.generate(prompt, steps)
    replayed = model.generate(prompt, steps, replay=True)
    model.free()
    ctx.close()
    print(f"tokens {got}\nminimum top-1 margin {min(margins):.3e}")
    assert got == want, (got, want, margins)
    assert replayed == want, (replayed, want)
    assert min(margins) > 1e-2


@pytest.mark.parametrize("hidden", [256, 2560, 4224])
def test_captured_step_outlives_grown_scratch(hidden):
    """A step captured behind one prompt and replayed behind another, of two to eight tokens, and
    after a matmul that needs far more of the context's scratch: rows that the step's matmuls
    cannot make inside (more than 4096 values) are in the decoder's own buffers."""
    import torch
    dec = pkg.decoder
    cfg = dec.DecoderConfig(2, hidden, 4, 2, 128, 1024, 2048)
    weights = dec.synthetic_weights(cfg, seed=hidden)
    rng = np.random.default_rng(hidden)
    prompts = [rng.integers(0, 2048, n).tolist() for n in (9, 5, 2)]
    ctx = pkg.capi.Context(0)
    model = dec.DenseDecoder(ctx, cfg, weights, capacity=40)
    want = [model.generate(p, 8) for p in prompts]
    model.free()
    ctx.close()
    ctx = pkg.capi.Context(0)
    model = dec.DenseDecoder(ctx, cfg, weights, capacity=40)
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, 1, 256, 9728), 256, 9728)
    got = []
    for i, p in enumerate(prompts):
        got.append(model.generate(p, 8, replay=True))  # captured with the first prompt
        rows = 300 * (i + 1)
        merged = torch.randn((rows, 2 * 9728), device="cuda")
        ctx.matmul_swiglu(w, merged, torch.zeros((rows, 256), device="cuda"))
        x = torch.randn((8, 9728), device="cuda")
        ctx.matmul_norm(w, x, None, torch.ones(9728, device="cuda"), 1e-6,
                        torch.zeros((8, 256), device="cuda"))
    w.free()
    model.free()
    ctx.close()
    assert got == want


def test_step_of_a_decoder_with_very_long_rows():
    """22528 hidden values: a gate and an up tile together are more than a block's memory, one tile
    is not.  The steps run, eager and captured, with the tokens of the operators in turn."""
    dec = pkg.decoder
    cfg = dec.DecoderConfig(1, 22528, 4, 2, 64, 128, 256)
    weights = dec.synthetic_weights(cfg, seed=3)
    ctx = pkg.capi.Context(0)
    tokens = []
    for fused in (False, None):
        model = dec.DenseDecoder(ctx, cfg, weights, capacity=16, fused_qkv=fused)
        tokens += [model.generate([7], 6), model.generate([7], 6, replay=True)]
        model.free()
    ctx.close()
    assert tokens[1:] == tokens[:-1]
