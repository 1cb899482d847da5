"""The decoder driver with a context that has the fused entries (b2w4_step_matmul,
b2w4_attention_step, b2w4_matmul_norm, b2w4_matmul_swiglu), on the CPU: the tokens of the driver
that runs operator by operator, and no call that would have a row of up to eight made in the
context's scratch.  A decode step is captured once and replayed later; scratch that it holds is
freed when a larger call grows it."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from cpu_context import OracleContext
from __graft_entry__ import load_package

pkg = load_package()
dec, capi = pkg.decoder, pkg.capi


class FusedOracleContext(OracleContext):
    def step_matmul(self, w, residual, update, norm_weight, eps, residual_out, y=None,
                    tokens=None, hidden_out=None, swiglu=False):
        inside = tokens is None and w.k <= 4096 and (update is not None or w.k > 256)
        assert inside or hidden_out is not None, f"a row of {w.k} values in the context's scratch"
        assert (tokens is None) != (y is None)
        assert not swiglu or w.k <= 20480, "more than a gate and an up tile of a block's memory"
        hidden = torch.empty((1, w.k)) if hidden_out is None else hidden_out
        if update is None:
            self.rms_norm(residual, norm_weight, eps, hidden)
            if residual_out is not None:
                residual_out.copy_(residual)
        else:
            total = residual.clone()
            self.add_rms_norm(total, update, norm_weight, eps, hidden)
            assert residual_out.data_ptr() not in (residual.data_ptr(), update.data_ptr())
            residual_out.copy_(total)
        if tokens is not None:
            self.matmul_argmax(w, hidden, tokens)
        elif swiglu:
            merged = torch.empty((1, w.n))
            self.matmul(w, hidden, merged)
            self.swiglu(merged, y)
        else:
            self.matmul(w, hidden, y)

    def attention_step(self, qkv, heads, kv_heads, dim, q_weight, k_weight, eps, cos, sin, past,
                       q_work, k_cache, v_cache, out, capacity, scale, past_dev=None):
        self.qkv_prepare(qkv, 1, heads, kv_heads, dim, q_weight, k_weight, eps, cos, sin, past,
                         q_work, k_cache, v_cache, capacity, past_dev)
        self.attention(q_work, None, None, k_cache, v_cache, out, 1, heads, kv_heads, dim, past,
                       capacity, scale, past_dev)

    def matmul_norm(self, w, residual, update, norm_weight, eps, y, rule=ol.ACT_G128):
        assert residual.shape[0] > 8, "rows in the context's scratch"
        hidden = torch.empty_like(residual)
        if update is None:
            self.rms_norm(residual, norm_weight, eps, hidden)
        else:
            self.add_rms_norm(residual, update, norm_weight, eps, hidden)
        self.matmul(w, hidden, y, rule=rule)

    def matmul_swiglu(self, w, merged, y, rule=ol.ACT_G128):
        assert merged.shape[0] > 8, "rows in the context's scratch"
        act = torch.empty((merged.shape[0], w.k))
        self.swiglu(merged, act)
        self.matmul(w, act, y, rule=rule)


@pytest.mark.parametrize("experts", [0, 4])
@pytest.mark.parametrize("hidden", [256, 384, 4224, 22528])
@pytest.mark.parametrize("prompt_len", [5, 9])
def test_fused_driver_gives_the_tokens_and_holds_no_scratch(hidden, prompt_len, experts):
    cfg = dec.DecoderConfig(2, hidden, 4, 2, 64, 128, 256, experts=experts,
                            top_k=2 if experts else 0)
    weights = dec.synthetic_weights(cfg, seed=hidden + prompt_len)
    prompt = np.random.default_rng(hidden).integers(0, 256, prompt_len).tolist()
    tokens = []
    for ctx in (OracleContext(), FusedOracleContext()):
        model = dec.DenseDecoder(ctx, cfg, weights, capacity=prompt_len + 12, device="cpu")
        assert model.fused_step == isinstance(ctx, FusedOracleContext)
        tokens.append(model.generate(prompt, 6))
    assert tokens[0] == tokens[1]
