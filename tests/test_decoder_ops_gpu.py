"""The operators between a decoder layer's matmuls (b2w4_rms_norm, b2w4_add_rms_norm,
b2w4_swiglu, b2w4_elementwise, b2w4_rope, b2w4_attention, b2w4_embed_rows) through the C ABI
against the CPU oracle, which is pinned bit for bit against the reference's own CPU operators
(tests/test_oracle_pins.py).  Element-wise arithmetic must be bit-exact; operators that sum
over a row (norms, attention scores, softmax) use tree reductions where the reference's loops
are sequential, and are held to the rounding error of a reassociated fp32 sum: 2e-6 relative
for the norms, 1e-5 relative L2 for attention."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle_lib as ol
from golden_util import rel_l2
from __graft_entry__ import load_package

pkg = load_package()
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    ol.set_exp_mode(True)  # the device takes exp in double and rounds once
    c = pkg.capi.Context(0)
    yield c
    c.close()
    ol.set_exp_mode(False)


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("rows,dim", [(1, 2560), (7, 2560), (256, 2560), (64, 128), (5, 4096),
                                      (3, 200)])
def test_rms_norm(ctx, rows, dim):
    import torch
    rng = np.random.default_rng(rows * 1000 + dim)
    x = rng.normal(0, 1.7, (rows, dim)).astype(np.float32)
    w = rng.normal(1, 0.2, dim).astype(np.float32)
    out = torch.zeros((rows, dim), dtype=torch.float32, device="cuda")
    ctx.rms_norm(_dev(x), _dev(w), 1e-6, out)
    ctx.sync()
    want = ol.rms_norm(x, w, 1e-6)
    got = out.cpu().numpy()
    assert np.max(np.abs(got - want) / (np.abs(want) + 1e-30)) < 2e-6


def test_add_rms_norm_writes_the_sum_back(ctx):
    import torch
    rng = np.random.default_rng(5)
    x = rng.normal(0, 1, (9, 2560)).astype(np.float32)
    u = rng.normal(0, 1, (9, 2560)).astype(np.float32)
    w = rng.normal(1, 0.2, 2560).astype(np.float32)
    res = _dev(x)
    out = torch.zeros((9, 2560), dtype=torch.float32, device="cuda")
    ctx.add_rms_norm(res, _dev(u), _dev(w), 1e-6, out)
    ctx.sync()
    want_res, want = ol.add_rms_norm(x, u, w, 1e-6)
    assert res.cpu().numpy().tobytes() == want_res.tobytes()  # one rounded add per element
    got = out.cpu().numpy()
    assert np.max(np.abs(got - want) / (np.abs(want) + 1e-30)) < 2e-6


def test_swiglu_add_mul_rope_embedding_are_bit_exact(ctx):
    import torch
    rng = np.random.default_rng(6)
    m = rng.normal(0, 2.5, (6, 2 * 9728)).astype(np.float32)
    out = torch.zeros((6, 9728), dtype=torch.float32, device="cuda")
    ctx.swiglu(_dev(m), out)
    a = rng.normal(0, 1, (4, 2560)).astype(np.float32)
    b = rng.normal(0, 1, (4, 2560)).astype(np.float32)
    s_add = torch.zeros((4, 2560), dtype=torch.float32, device="cuda")
    s_mul = torch.zeros((4, 2560), dtype=torch.float32, device="cuda")
    ctx.add(_dev(a), _dev(b), s_add)
    ctx.add(_dev(a), _dev(b), s_mul, multiply=True)
    q = rng.normal(0, 1, (5, 8, 128)).astype(np.float32)
    ang = rng.uniform(0, 6.28, (5, 64)).astype(np.float32)
    c, s = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    qd = _dev(q)
    r_out = torch.zeros_like(qd)
    ctx.rope(qd, r_out, 5, 8, 128, _dev(c), _dev(s), 128)
    r_part = torch.zeros_like(qd)
    ctx.rope(qd, r_part, 5, 8, 128, _dev(c[:, :32]), _dev(s[:, :32]), 64)  # rope_dim < dim
    ctx.rope(qd, qd, 5, 8, 128, _dev(c), _dev(s), 128)                     # in place
    table = rng.normal(0, 0.02, (1000, 256)).astype(np.float16)
    ids = np.array([3, 999, 0, 3], dtype=np.int32)
    emb = torch.zeros((4, 256), dtype=torch.float32, device="cuda")
    ctx.embed_rows(_dev(table.view(np.int16)), _dev(ids), emb)
    ctx.sync()
    assert out.cpu().numpy().tobytes() == ol.swiglu(m).tobytes()
    assert s_add.cpu().numpy().tobytes() == (a + b).tobytes()
    assert s_mul.cpu().numpy().tobytes() == (a * b).tobytes()
    assert r_out.cpu().numpy().tobytes() == ol.rope(q, c, s, 128).tobytes()
    assert r_part.cpu().numpy().tobytes() == ol.rope(q, c[:, :32], s[:, :32], 64).tobytes()
    assert qd.cpu().numpy().tobytes() == ol.rope(q, c, s, 128).tobytes()
    assert emb.cpu().numpy().tobytes() == table[ids].astype(np.float32).tobytes()


@pytest.mark.parametrize("tokens,past,heads,kv_heads", [(1, 37, 8, 2), (33, 0, 8, 2),
                                                        (5, 300, 32, 8), (1, 0, 4, 4)])
def test_attention_over_the_cache(ctx, tokens, past, heads, kv_heads):
    """Causal attention of new tokens over a cache that already holds `past` tokens: the new
    keys and values land at their positions (exact copies) and the output agrees with the
    x86 reference's (full-row softmax, P*V key by key) within 1e-5: the cluster and tile kernels
    take the softmax over parts of the keys."""
    import torch
    dim, capacity = 128, 512
    rng = np.random.default_rng(tokens * 31 + past)
    k_hist = rng.normal(0, 1, (past, kv_heads, dim)).astype(np.float32)
    v_hist = rng.normal(0, 1, (past, kv_heads, dim)).astype(np.float32)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k = rng.normal(0, 1, (tokens, kv_heads, dim)).astype(np.float32)
    v = rng.normal(0, 1, (tokens, kv_heads, dim)).astype(np.float32)
    kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    vc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    kc[:, :past] = k_hist.transpose(1, 0, 2)
    vc[:, :past] = v_hist.transpose(1, 0, 2)
    kcd, vcd = _dev(kc), _dev(vc)
    out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
    scale = dim ** -0.5
    ctx.attention(_dev(q), _dev(k), _dev(v), kcd, vcd, out, tokens, heads, kv_heads, dim, past,
                  capacity, scale)
    ctx.sync()
    k_all = np.concatenate([k_hist, k])
    v_all = np.concatenate([v_hist, v])
    assert kcd.cpu().numpy()[:, :past + tokens].tobytes() == \
        np.ascontiguousarray(k_all.transpose(1, 0, 2)).tobytes()
    assert vcd.cpu().numpy()[:, :past + tokens].tobytes() == \
        np.ascontiguousarray(v_all.transpose(1, 0, 2)).tobytes()
    want = ol.causal_attention(q, k_all, v_all, heads, kv_heads, past, scale)
    assert rel_l2(out.cpu().numpy(), want) < 1e-5
    # the same call with the position read from device memory gives the same bits
    kcd2, vcd2 = _dev(kc), _dev(vc)
    out2 = torch.zeros_like(out)
    past_dev = torch.full((1,), past, dtype=torch.int32, device="cuda")
    ctx.attention(_dev(q), _dev(k), _dev(v), kcd2, vcd2, out2, tokens, heads, kv_heads, dim, 0,
                  capacity, scale, past_dev)
    ctx.sync()
    assert out2.cpu().numpy().tobytes() == out.cpu().numpy().tobytes()
    assert kcd2.cpu().numpy().tobytes() == kcd.cpu().numpy().tobytes()
    with pytest.raises(pkg.capi.B200W4Error):  # the cache is full
        ctx.attention(_dev(q), _dev(k), _dev(v), kcd, vcd, out, tokens, heads, kv_heads, dim,
                      capacity - tokens + 1, capacity, scale)


def test_position_on_the_device(ctx):
    """Rotary rows taken at first_position + t or at *position_dev + t agree with the oracle
    on those rows of the table; b2w4_advance records the token and moves the counter."""
    import torch
    rng = np.random.default_rng(11)
    q = rng.normal(0, 1, (3, 4, 64)).astype(np.float32)
    ang = rng.uniform(0, 6.28, (40, 32)).astype(np.float32)
    c, s = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    cd, sd, qd = _dev(c), _dev(s), _dev(q)
    a = torch.zeros_like(qd)
    b = torch.zeros_like(qd)
    pos = torch.full((1,), 17, dtype=torch.int32, device="cuda")
    ctx.rope(qd, a, 3, 4, 64, cd, sd, 64, 17)
    ctx.rope(qd, b, 3, 4, 64, cd, sd, 64, 0, pos)
    hist = torch.full((40,), -1, dtype=torch.int32, device="cuda")
    tok = torch.full((1,), 1234, dtype=torch.int32, device="cuda")
    ctx.advance(pos, 1, tok, hist)
    ctx.advance(pos, 2)
    ctx.sync()
    want = ol.rope(q, c[17:20], s[17:20], 64)
    assert a.cpu().numpy().tobytes() == want.tobytes()
    assert b.cpu().numpy().tobytes() == want.tobytes()
    assert int(pos.item()) == 20
    h = hist.cpu().numpy()
    assert h[17] == 1234 and (np.delete(h, 17) == -1).all()


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [(1, 9, 8, 2, 128), (7, 0, 4, 4, 64),
                                                            (3, 20, 2, 1, 256)])
def test_fused_qkv_step_equals_the_separate_operators(ctx, tokens, past, heads, kv_heads, dim):
    """b2w4_qkv_prepare (per-head norm + rotary embedding + cache append in one launch) leaves
    the same bits in q and in the caches as rms_norm, rope and the append of b2w4_attention
    run one after the other; attention without an append then gives the same output."""
    import torch
    capacity = 64
    rng = np.random.default_rng(dim + tokens)
    width = (heads + 2 * kv_heads) * dim
    qkv = rng.normal(0, 1, (tokens, width)).astype(np.float32)
    qw = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    kw = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    ang = rng.uniform(0, 6.28, (capacity, dim // 2)).astype(np.float32)
    c, s = _dev(np.cos(ang).astype(np.float32)), _dev(np.sin(ang).astype(np.float32))
    hist = rng.normal(0, 1, (2, kv_heads, capacity, dim)).astype(np.float32)
    qkv_d, qw_d, kw_d = _dev(qkv), _dev(qw), _dev(kw)
    scale = dim ** -0.5
    # operator by operator
    q = _dev(qkv[:, :heads * dim].reshape(tokens * heads, dim))
    k = _dev(qkv[:, heads * dim:(heads + kv_heads) * dim].reshape(tokens * kv_heads, dim))
    v = _dev(qkv[:, (heads + kv_heads) * dim:])
    kc1, vc1 = _dev(hist[0]), _dev(hist[1])
    out1 = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
    ctx.rms_norm(q, qw_d, 1e-6, q)
    ctx.rms_norm(k, kw_d, 1e-6, k)
    ctx.rope(q, q, tokens, heads, dim, c, s, dim, past)
    ctx.rope(k, k, tokens, kv_heads, dim, c, s, dim, past)
    ctx.attention(q, k, v, kc1, vc1, out1, tokens, heads, kv_heads, dim, past, capacity, scale)
    # fused, once with the position as an argument and once from device memory
    for past_dev in (None, torch.full((1,), past, dtype=torch.int32, device="cuda")):
        kc2, vc2 = _dev(hist[0]), _dev(hist[1])
        q2 = torch.zeros((tokens * heads, dim), dtype=torch.float32, device="cuda")
        out2 = torch.zeros_like(out1)
        arg_past = past if past_dev is None else 0
        ctx.qkv_prepare(qkv_d, tokens, heads, kv_heads, dim, qw_d, kw_d, 1e-6, c, s, arg_past, q2,
                        kc2, vc2, capacity, past_dev)
        ctx.attention(q2, None, None, kc2, vc2, out2, tokens, heads, kv_heads, dim, arg_past,
                      capacity, scale, past_dev)
        ctx.sync()
        assert q2.cpu().numpy().tobytes() == q.cpu().numpy().tobytes()
        assert kc2.cpu().numpy().tobytes() == kc1.cpu().numpy().tobytes()
        assert vc2.cpu().numpy().tobytes() == vc1.cpu().numpy().tobytes()
        assert out2.cpu().numpy().tobytes() == out1.cpu().numpy().tobytes()


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [(33, 0, 8, 2, 128),
                                                            (256, 0, 32, 8, 128),
                                                            (40, 100, 4, 4, 64),
                                                            (17, 5, 6, 2, 256),
                                                            (64, 300, 32, 4, 128)])
def test_tile_attention_equals_the_row_kernel(ctx, tokens, past, heads, kv_heads, dim):
    """A run of tokens takes the tile kernel (a block per kv head and tile of query tokens);
    it must leave the same bits as the one-row kernel, and agree with the oracle."""
    import os
    import torch
    os.environ["B2W4_ATTN"] = "row"
    try:
        ctx_row = pkg.capi.Context(0)
    finally:
        del os.environ["B2W4_ATTN"]
    capacity = past + tokens + 3
    rng = np.random.default_rng(tokens + dim)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    vc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    kc[:, :past + tokens] = k_all.transpose(1, 0, 2)
    vc[:, :past + tokens] = v_all.transpose(1, 0, 2)
    kcd, vcd, qd = _dev(kc), _dev(vc), _dev(q)
    scale = dim ** -0.5
    outs = []
    for c, past_dev in ((ctx_row, None), (ctx, None),
                        (ctx, torch.full((1,), past, dtype=torch.int32, device="cuda"))):
        out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
        c.attention(qd, None, None, kcd, vcd, out, tokens, heads, kv_heads, dim,
                    past if past_dev is None else 0, capacity, scale, past_dev)
        c.sync()
        outs.append(out.cpu().numpy())
    ctx_row.close()
    assert outs[1].tobytes() == outs[0].tobytes()
    assert outs[2].tobytes() == outs[0].tobytes()
    want = ol.causal_attention(q, k_all, v_all, heads, kv_heads, past, scale)
    assert rel_l2(outs[1], want) < 1e-5


def _attention_fp64(q, k_all, v_all, heads, kv_heads, past, scale):
    """Causal attention in 64 bits, key rows with a vanishing probability left out."""
    tokens, rep = q.shape[0], heads // kv_heads
    out = np.zeros(q.shape)
    for t in range(tokens):
        for h in range(heads):
            k = k_all[:past + t + 1, h // rep].astype(np.float64)
            s = (k @ q[t, h].astype(np.float64)) * scale
            p = np.exp(s - s.max())
            seen = p > 0
            v = v_all[:past + t + 1, h // rep][seen].astype(np.float64)
            out[t, h] = (p[seen] / p.sum()) @ v
    return out


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (1, 0, 4, 4, 64), (1, 14, 8, 8, 64), (1, 15, 12, 2, 64), (2, 16, 6, 2, 128),
    (1, 127, 4, 1, 128), (7, 1000, 10, 2, 128), (1, 4100, 2, 2, 128), (3, 31, 2, 2, 256),
    (1, 777, 6, 2, 256)])
def test_split_attention_of_a_few_tokens(ctx, tokens, past, heads, kv_heads, dim):
    """Up to seven query tokens: the keys are split over a cluster of blocks (ranges of zero,
    one or many keys, head groups that do not fill a block's rows).  Tolerance: the fp32 dot
    product of 256 terms, 2^-24 * (16 adds in sequence) * sum |q k| * scale <= 1e-5, is the
    relative error of a probability.  Then with a key whose probability underflows to zero and
    whose value row is NaN: nothing of it may reach the output."""
    import torch
    capacity, scale = past + tokens + 5, dim ** -0.5
    rng = np.random.default_rng(past + dim)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    for hole in (None, past // 2):
        if hole is not None:
            if past == 0 or tokens > 1 or heads != kv_heads:
                continue
            k_all[hole] = -1e30 * np.sign(q[0])
            v_all[hole] = np.nan
        kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
        vc = np.full((kv_heads, capacity, dim), np.nan, dtype=np.float32)  # past the position
        kc[:, :past + tokens] = k_all.transpose(1, 0, 2)
        vc[:, :past + tokens] = v_all.transpose(1, 0, 2)
        kcd, vcd, qd = _dev(kc), _dev(vc), _dev(q)
        outs = []
        for past_dev in (None, torch.full((1,), past, dtype=torch.int32, device="cuda")):
            out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
            ctx.attention(qd, None, None, kcd, vcd, out, tokens, heads, kv_heads, dim,
                          past if past_dev is None else 0, capacity, scale, past_dev)
            ctx.sync()
            outs.append(out.cpu().numpy())
        assert outs[1].tobytes() == outs[0].tobytes()
        assert rel_l2(outs[0], _attention_fp64(q, k_all, v_all, heads, kv_heads, past,
                                               scale)) < 1e-5


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (8, 0, 64, 1, 64), (9, 1600, 8, 2, 128), (31, 33, 3, 1, 128), (70, 0, 5, 5, 256),
    (2, 70, 4, 2, 80), (1, 300, 3, 3, 20), (12, 40, 2, 1, 96), (9, 3, 65, 1, 64)])
def test_tile_and_row_attention(ctx, tokens, past, heads, kv_heads, dim):
    """Runs of eight or more tokens (tile kernel: several softmax blocks, head groups that do
    not fill a tile, more keys than a block's scores would hold) and the shapes that only the
    one-row kernel takes (other head sizes, more heads per kv head than a tile has rows),
    against 64 bits; tolerance as for the split kernel.  Value rows past the last position are
    NaN, and so is the last token's: the earlier tokens do not see them."""
    import torch
    capacity, scale = past + tokens + 40, dim ** -0.5
    rng = np.random.default_rng(past + dim)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all[-1] = np.nan
    kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    vc = np.full((kv_heads, capacity, dim), np.nan, dtype=np.float32)
    kc[:, :past + tokens] = k_all.transpose(1, 0, 2)
    vc[:, :past + tokens] = v_all.transpose(1, 0, 2)
    out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
    ctx.attention(_dev(q), None, None, _dev(kc), _dev(vc), out, tokens, heads, kv_heads, dim,
                  past, capacity, scale)
    ctx.sync()
    got = out.cpu().numpy()
    assert np.isnan(got[-1]).all()
    if tokens > 1:
        want = _attention_fp64(q, k_all, v_all, heads, kv_heads, past, scale)
        assert rel_l2(got[:-1], want[:-1]) < 1e-5


def _row_context():
    """A context whose attention keeps one block per (token, head)."""
    import os
    os.environ["B2W4_ATTN"] = "row"
    try:
        return pkg.capi.Context(0)
    finally:
        del os.environ["B2W4_ATTN"]


@pytest.mark.parametrize("past,heads,kv_heads,dim", [(0, 4, 2, 128), (31, 2, 2, 64),
                                                     (300, 8, 2, 128), (97, 6, 2, 256)])
def test_row_switch_holds_for_a_single_token(ctx, past, heads, kv_heads, dim):
    """B2W4_ATTN=row keeps the one-row kernel for single tokens too: the last token of a run
    through the tile kernel and that token alone through the row switch leave the same bits
    (one arithmetic), and the default form of the single token agrees with both (tolerance as
    for the split kernel)."""
    import torch
    tokens, scale = 9, dim ** -0.5
    capacity = past + tokens + 2
    rng = np.random.default_rng(past + dim)
    q = _dev(rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32))
    kc, vc = (_dev(rng.normal(0, 1, (kv_heads, capacity, dim)).astype(np.float32))
              for _ in range(2))
    run, row, one = (torch.zeros((n, heads, dim), dtype=torch.float32, device="cuda")
                     for n in (tokens, 1, 1))
    ctx_row = _row_context()
    last = q[-1:].contiguous()
    ctx.attention(q, None, None, kc, vc, run, tokens, heads, kv_heads, dim, past, capacity, scale)
    ctx_row.attention(last, None, None, kc, vc, row, 1, heads, kv_heads, dim,
                      past + tokens - 1, capacity, scale)
    ctx.attention(last, None, None, kc, vc, one, 1, heads, kv_heads, dim, past + tokens - 1,
                  capacity, scale)
    ctx.sync()
    ctx_row.sync()
    ctx_row.close()
    assert row.cpu().numpy().tobytes() == run[-1:].contiguous().cpu().numpy().tobytes()
    assert rel_l2(one.cpu().numpy(), row.cpu().numpy()) < 1e-5


def _staged(rng, heads, kv_heads, dim, keys, levels):
    """q of one token and a cache whose scores (scale 1) are levels[i] in the i-th part of the
    keys, the same for every head: feature 0 carries the score, the others are zero."""
    q = np.zeros((1, heads, dim), dtype=np.float32)
    q[:, :, 0] = 1.0
    k = np.zeros((keys, kv_heads, dim), dtype=np.float32)
    for i, part in enumerate(np.array_split(np.arange(keys), len(levels))):
        k[part, :, 0] = levels[i]
    v = rng.normal(0, 1, (keys, kv_heads, dim)).astype(np.float32)
    return q, k, v


@pytest.mark.parametrize("row", [False, True])
@pytest.mark.parametrize("tokens,heads,kv_heads,dim", [
    (1, 2, 2, 64), (1, 4, 2, 64), (1, 8, 2, 128), (1, 2, 1, 256), (3, 3, 1, 128),
    (12, 8, 2, 128), (12, 2, 2, 64), (9, 2, 1, 256), (1, 4, 2, 80), (10, 4, 2, 80)])
def test_attention_ignores_value_rows_of_zero_probability(ctx, tokens, heads, kv_heads, dim, row):
    """Scores of 0, 80 and 160 in the three parts of the cache: a key of the first part has
    the probability e^-160 = 0, but e^-80 > 0 against the middle part, and 1 against its own
    neighbours.  Its value row is NaN (then infinite): nothing of it may reach the output, in
    whatever order or split the keys are taken.  Then value rows near the largest number under
    equal scores: a sum before the division would overflow, the result does not.  Tolerance:
    300 terms summed in fp32 at most one after the other, 300 * 2^-24 = 2e-5 of their
    magnitudes; the mean of 1e38 rows keeps 1e-5 since all terms have one sign."""
    import torch
    rng = np.random.default_rng(dim + tokens)
    keys = 300 + tokens
    q1, k, v = _staged(rng, heads, kv_heads, dim, keys, [0.0, 80.0, 160.0])
    q = np.repeat(q1, tokens, axis=0)
    c = _row_context() if row else ctx
    capacity = keys + 3

    def run():
        kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
        vc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
        kc[:, :keys], vc[:, :keys] = k.transpose(1, 0, 2), v.transpose(1, 0, 2)
        out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
        c.attention(_dev(q), None, None, _dev(kc), _dev(vc), out, tokens, heads, kv_heads, dim,
                    keys - tokens, capacity, 1.0)
        c.sync()
        return out.cpu().numpy()

    clean = _attention_fp64(q, k, np.where(np.arange(keys)[:, None, None] < 100, 0, v), heads,
                            kv_heads, keys - tokens, 1.0)
    for bad in (np.nan, np.inf, -np.inf):
        v[3] = bad
        v[50, :, dim // 2] = bad
        got = run()
        assert np.isfinite(got).all()
        assert rel_l2(got, clean) < 2e-5
    k[:] = 0.0
    v[:] = 3e38 * rng.uniform(0.5, 1.0, v.shape)
    got = run()
    want = _attention_fp64(q, k, v, heads, kv_heads, keys - tokens, 1.0)
    assert np.isfinite(got).all()
    assert rel_l2(got / 3e38, want / 3e38) < 1e-5
    k[:] = 0.0
    v[:] = rng.normal(0, 1, v.shape)
    v[7] = np.nan  # seen: every feature is NaN, as the sum has it
    assert np.isnan(run()).all()
    if row:
        c.close()


@pytest.mark.parametrize("cluster", [0, 1, 3, 4, 8, 16])
@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (1, 94, 8, 2, 64), (3, 94, 4, 2, 128), (2, 126, 3, 3, 128), (7, 126, 6, 1, 256),
    (1, 1500, 8, 2, 128), (5, 700, 5, 5, 64), (12, 1200, 4, 2, 64)])
def test_split_attention_on_either_side_of_one_range(ctx, tokens, past, heads, kv_heads, dim,
                                                     cluster):
    """Runs whose tokens see 95 .. 133 keys, the last counts that one block takes alone and the
    first that a cluster splits, and longer ones; clusters of every size that a device may
    allow, and none (one block per (token, head), or tiles).  Position on the host or on the device: the
    same bits.  Tolerance as for the split kernel."""
    import os
    import torch
    capacity, scale = 1600, dim ** -0.5
    rng = np.random.default_rng(past + dim + cluster)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    kc = np.zeros((kv_heads, capacity, dim), dtype=np.float32)
    vc = np.full((kv_heads, capacity, dim), np.nan, dtype=np.float32)
    kc[:, :past + tokens] = k_all.transpose(1, 0, 2)
    vc[:, :past + tokens] = v_all.transpose(1, 0, 2)
    kcd, vcd, qd = _dev(kc), _dev(vc), _dev(q)
    os.environ["B2W4_ATTN_CLUSTER"] = str(cluster)
    try:
        c = pkg.capi.Context(0)
    finally:
        del os.environ["B2W4_ATTN_CLUSTER"]
    outs = []
    for past_dev in (None, torch.full((1,), past, dtype=torch.int32, device="cuda")):
        out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
        c.attention(qd, None, None, kcd, vcd, out, tokens, heads, kv_heads, dim,
                    past if past_dev is None else 0, capacity, scale, past_dev)
        c.sync()
        outs.append(out.cpu().numpy())
    c.close()
    want = _attention_fp64(q, k_all, v_all, heads, kv_heads, past, scale)
    assert rel_l2(outs[0], want) < 1e-5
    if cluster >= 4:
        assert outs[1].tobytes() == outs[0].tobytes()
    else:  # few keys known to the host need no cluster; the device's position does
        assert rel_l2(outs[1], want) < 1e-5


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (8, 376, 8, 2, 128), (9, 1600, 3, 1, 64), (16, 3000, 2, 2, 256), (33, 4090, 4, 2, 128),
    (64, 500, 32, 8, 64), (200, 300, 6, 2, 128)])
def test_short_runs_behind_a_context(ctx, tokens, past, heads, kv_heads, dim):
    """Runs of eight or more tokens on a cache of at least 384 rows whose tiles would leave
    most of the chip idle go to the split kernel: some tokens within one block's range of keys
    and some beyond.  The position on the device leaves the same bits.  Tolerance as for the
    split kernel."""
    import torch
    capacity, scale = past + tokens, dim ** -0.5
    rng = np.random.default_rng(past + dim)
    q = rng.normal(0, 1, (tokens, heads, dim)).astype(np.float32)
    k_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    v_all = rng.normal(0, 1, (past + tokens, kv_heads, dim)).astype(np.float32)
    kcd, vcd = (_dev(np.ascontiguousarray(x.transpose(1, 0, 2))) for x in (k_all, v_all))
    qd = _dev(q)
    outs = []
    for past_dev in (None, torch.full((1,), past, dtype=torch.int32, device="cuda")):
        out = torch.zeros((tokens, heads, dim), dtype=torch.float32, device="cuda")
        ctx.attention(qd, None, None, kcd, vcd, out, tokens, heads, kv_heads, dim,
                      past if past_dev is None else 0, capacity, scale, past_dev)
        ctx.sync()
        outs.append(out.cpu().numpy())
    assert outs[1].tobytes() == outs[0].tobytes()
    some = [0, 1, tokens // 2, tokens - 1]
    for t in some:
        want = _attention_fp64(q[t:t + 1], k_all, v_all, heads, kv_heads, past + t, scale)
        assert rel_l2(outs[0][t:t + 1], want) < 1e-5


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (31, 0, 8, 8, 64), (260, 90, 20, 20, 64), (600, 100, 8, 8, 128), (700, 0, 33, 1, 64),
    (640, 0, 32, 8, 64), (1300, 0, 16, 8, 64), (500, 3, 16, 4, 256)])
def test_tile_variants_equal_the_row_arithmetic(ctx, tokens, past, heads, kv_heads, dim):
    """Tiles of 32 and 64 rows, one or two per multiprocessor, grids of one wave and of several,
    ragged last tiles: the bits of the one-row form, row by row."""
    import torch
    capacity, scale = past + tokens, dim ** -0.5
    g = torch.Generator(device="cuda").manual_seed(tokens + dim)
    q = torch.randn((tokens, heads, dim), device="cuda", generator=g)
    kc, vc = (torch.randn((kv_heads, capacity, dim), device="cuda", generator=g)
              for _ in range(2))
    ctx_row = _row_context()
    outs = []
    for c in (ctx, ctx_row):
        out = torch.zeros_like(q)
        c.attention(q, None, None, kc, vc, out, tokens, heads, kv_heads, dim, past, capacity,
                    scale)
        c.sync()
        outs.append(out.cpu().numpy())
    ctx_row.close()
    assert np.isfinite(outs[0]).all()
    assert outs[0].tobytes() == outs[1].tobytes()


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [
    (1, 40, 8, 2, 128), (25, 50, 32, 8, 128), (70, 300, 16, 8, 64), (600, 0, 16, 4, 128),
    (300, 7, 16, 4, 256)])
def test_attention_on_unaligned_rows(ctx, tokens, past, heads, kv_heads, dim):
    """q, the caches and the output one float past a 16-byte boundary: runs take the tile
    kernel with narrow copies (the bits of the one-row form), few rows one block per (token,
    head) (tolerance as for the split kernel)."""
    import torch
    capacity, scale = past + tokens + 1, dim ** -0.5
    g = torch.Generator(device="cuda").manual_seed(tokens + dim)

    def odd(*shape):
        n = int(np.prod(shape))
        return torch.randn(n + 1, device="cuda", generator=g)[1:].view(*shape)

    q, out = odd(tokens, heads, dim), odd(tokens, heads, dim)
    kc, vc = odd(kv_heads, capacity, dim), odd(kv_heads, capacity, dim)
    row = torch.zeros((tokens, heads, dim), device="cuda")
    assert q.data_ptr() % 16 and out.data_ptr() % 16 and kc.data_ptr() % 16
    ctx_row = _row_context()
    ctx.attention(q, None, None, kc, vc, out, tokens, heads, kv_heads, dim, past, capacity, scale)
    ctx_row.attention(q, None, None, kc, vc, row, tokens, heads, kv_heads, dim, past, capacity,
                      scale)
    ctx.sync()
    ctx_row.sync()
    ctx_row.close()
    got, want = out.cpu().numpy(), row.cpu().numpy()
    if tokens >= 8:
        assert got.tobytes() == want.tobytes()
    assert rel_l2(got, want) < 1e-5


@pytest.mark.parametrize("past,heads,kv_heads,dim", [(0, 4, 2, 128), (31, 16, 2, 128),
                                                     (300, 32, 8, 128), (127, 8, 2, 64),
                                                     (500, 6, 6, 64), (1000, 4, 2, 256),
                                                     (40, 6, 2, 192)])
@pytest.mark.parametrize("on_device", [False, True])
def test_attention_step_equals_prepare_and_attention(ctx, past, heads, kv_heads, dim, on_device):
    """One token's norm, rotary embedding, cache append and attention in one launch (or, for a
    head size that is not split, in the two launches): the bits of the separate operators."""
    import torch
    rng = np.random.default_rng(past + dim)
    cap = past + 70
    qkv = _dev(rng.normal(0, 1, (1, (heads + 2 * kv_heads) * dim)).astype(np.float32))
    qw, kw = (_dev(rng.normal(1, 0.1, dim).astype(np.float32)) for _ in range(2))
    cos, sin = (_dev(t) for t in pkg.decoder.rope_tables(range(cap), dim, 1e6))
    cache = [_dev(rng.normal(0, 1, (kv_heads, cap, dim)).astype(np.float32)) for _ in range(2)]
    pos = torch.tensor([past], dtype=torch.int32, device="cuda") if on_device else None
    host_past = 0 if on_device else past
    want_kv = [c.clone() for c in cache]
    q, want, got = (torch.zeros((1, heads * dim), device="cuda") for _ in range(3))
    ctx.qkv_prepare(qkv, 1, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, host_past, q,
                    *want_kv, cap, pos)
    ctx.attention(q, None, None, *want_kv, want, 1, heads, kv_heads, dim, host_past, cap,
                  dim ** -0.5, pos)
    ctx.attention_step(qkv, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, host_past,
                       torch.zeros_like(q), *cache, got, cap, dim ** -0.5, pos)
    ctx.sync()
    for a, b in zip(cache, want_kv):
        assert torch.equal(a, b) and torch.equal(got, want)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n,k", [(16, 128), (272, 2560), (4864, 4096), (2560, 9728),
                                 (19456, 2560)])
@pytest.mark.parametrize("with_update", [False, True])
def test_step_matmul_equals_its_operators(ctx, n, k, with_update):
    """The matmul with the residual add and norm in front and SwiGLU or the greedy token behind:
    the bits of the operators in turn (rows up to and beyond the 4096 values that stay in
    registers)."""
    import torch
    rng = np.random.default_rng(n + k)
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
    x, u, g = (_dev(rng.normal(m, s, (1, k)).astype(np.float32))
               for m, s in ((0, 2), (0, 1), (1, 0.2)))
    upd = u if with_update else None
    res, hid = (torch.zeros((1, k), device="cuda") for _ in range(2))
    y, want = (torch.zeros((1, n), device="cuda") for _ in range(2))
    act, want_act = (torch.zeros((1, n // 2), device="cuda") for _ in range(2))
    tok, want_tok = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    ctx.step_matmul(w, x, upd, g, 1e-6, res, y=y, hidden_out=hid)
    ctx.step_matmul(w, x, upd, g, 1e-6, res, y=act, swiglu=True)
    ctx.step_matmul(w, x, upd, g, 1e-6, res, tokens=tok)
    want_res, want_hid = x.clone(), torch.zeros((1, k), device="cuda")
    ctx.add_rms_norm(want_res, u if with_update else torch.zeros_like(x), g, 1e-6, want_hid)
    ctx.matmul(w, want_hid, want, rule=ol.ACT_G128)
    ctx.swiglu(want, want_act)
    ctx.matmul_argmax(w, want_hid, want_tok)
    ctx.sync()
    assert torch.equal(res, want_res) and torch.equal(hid, want_hid)
    assert torch.equal(y, want) and torch.equal(act, want_act) and torch.equal(tok, want_tok)
    w.free()


def test_step_matmul_refuses_what_it_cannot_take(ctx):
    """The new residual in the old one's place, both or no outputs, rows off 16 bytes."""
    import torch
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, 1, 24, 128), 24, 128)
    x, u, g, r = (torch.ones((1, 128), device="cuda") for _ in range(4))
    y = torch.zeros((1, 24), device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    for kw in (dict(residual_out=x, y=y), dict(residual_out=u, y=y), dict(residual_out=None, y=y),
               dict(residual_out=r), dict(residual_out=r, y=y, tokens=tok),
               dict(residual_out=r, y=y, swiglu=True),
               dict(residual_out=torch.ones(129, device="cuda")[1:], y=y)):
        with pytest.raises(pkg.capi.B200W4Error):
            ctx.step_matmul(w, x, u, g, 1e-6, **kw)
    w.free()


@pytest.mark.parametrize("rows,dim,off", [(1, 2560, 0), (3, 1026, 0), (2, 1024, 1), (70000, 8, 0)])
def test_embedding_rows_of_any_size(ctx, rows, dim, off):
    """Rows that four features divide and that they do not, off the store's alignment, and more
    rows than a grid's second dimension holds."""
    import torch
    table = torch.randn((50, dim), device="cuda").half()
    ids = torch.randint(0, 50, (rows,), dtype=torch.int32, device="cuda")
    out = torch.zeros(rows * dim + off, device="cuda")[off:].view(rows, dim)
    ctx.embed_rows(table, ids, out)
    ctx.sync()
    assert torch.equal(out, table.float()[ids.long()])


@pytest.mark.parametrize("rule", [ol.ACT_G32, ol.ACT_G128])
@pytest.mark.parametrize("m,n,k", [(1, 72, 384), (6, 72, 640), (9, 264, 2560), (33, 136, 5120),
                                   (150, 264, 5376), (40, 48, 256), (12, 40, 12416)])
def test_matmuls_that_make_their_rows(ctx, m, n, k, rule):
    """Residual add + norm, or SwiGLU, in the matmul's quantiser (and, for row counts, weights and
    row lengths that it does not take, in scratch): the bits of the two calls."""
    import torch
    rng = np.random.default_rng(m + k)
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
    dev = lambda *shape: _dev(rng.normal(0, 1, shape).astype(np.float32))
    x, u, g, merged = dev(m, k), dev(m, k), _dev(rng.normal(1, 0.2, k).astype(np.float32)), \
        dev(m, 2 * k)
    got, want, h, act = (torch.zeros((m, c), device="cuda") for c in (n, n, k, k))
    ctx.matmul_swiglu(w, merged, got, rule=rule)
    ctx.swiglu(merged, act)
    ctx.matmul(w, act, want, rule=rule)
    ctx.sync()
    assert torch.equal(got, want)
    for update in (None, u):
        a, b = x.clone(), x.clone()
        ctx.matmul_norm(w, a, update, g, 1e-6, got, rule=rule)
        if update is None:
            ctx.rms_norm(b, g, 1e-6, h)
        else:
            ctx.add_rms_norm(b, update, g, 1e-6, h)
        ctx.matmul(w, h, want, rule=rule)
        ctx.sync()
        assert torch.equal(a, b) and torch.equal(got, want)
    w.free()


@pytest.mark.parametrize("n,k", [(272, 128), (272, 2560), (4864, 4096), (272, 4224)])
def test_step_matmul_reads_norm_weights_that_were_just_written(ctx, n, k):
    """A norm weight made by the operator in front (1 + w, as some packages store it): read when
    that operator is done, as b2w4_add_rms_norm reads it."""
    import torch
    rng = np.random.default_rng(n + k)
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
    x, u, g = (_dev(rng.normal(0, s, (1, k)).astype(np.float32)) for s in (2, 1, 0.2))
    one = torch.ones((1, k), device="cuda")
    made = [torch.zeros((1, k), device="cuda") for _ in range(12)]
    res, hid, want_hid = (torch.zeros((1, k), device="cuda") for _ in range(3))
    y = torch.zeros((len(made), n), device="cuda")
    want = torch.zeros((1, n), device="cuda")
    # (the many rows keep the kernels in front from being done early)
    wide = [torch.zeros((4096, k), device="cuda") for _ in range(2)]
    for i, weight in enumerate(made):
        ctx.copy_rows(wide[0], wide[1], 4096, k)
        ctx.add(g, one, weight)
        ctx.step_matmul(w, x, u, weight, 1e-6, res, y=y[i:i + 1], hidden_out=hid)
    ctx.add_rms_norm(x.clone(), u, one + g, 1e-6, want_hid)
    ctx.matmul(w, want_hid, want, rule=ol.ACT_G128)
    ctx.sync()
    assert torch.equal(hid, want_hid) and torch.equal(y, want.expand_as(y))
    w.free()


@pytest.mark.parametrize("where", ["residual", "update", "both", "weight", "new residual",
                                   "half", "in place", "in place of update"])
@pytest.mark.parametrize("k", [2560, 4224])
def test_step_matmul_outputs_over_rows_that_are_read(ctx, k, where):
    """y over the rows the call reads (the very row, the end of one and the start of the next, or
    its second half), over the new residual, and the normalised row in the place of the one it is
    made from: the operators in turn, whose inputs are read before their outputs are stored."""
    import torch
    n = k
    rng = np.random.default_rng(k)
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
    first = rng.normal(0, 1, (5, k)).astype(np.float32)  # residual, update, weight, new, spare
    rows = _dev(first)
    x, u, g, res, spare = (rows[i:i + 1] for i in range(5))
    flat = rows.view(-1)
    y = {"residual": x, "update": u, "weight": g, "new residual": res,
         "both": flat[k // 2:k // 2 + n].view(1, n), "half": flat[3 * k // 2:][:n].view(1, n),
         "in place": spare, "in place of update": spare}[where]
    hid = {"in place": x, "in place of update": u}.get(where)
    want_res, want_hid = _dev(first[:1]), torch.zeros((1, k), device="cuda")
    want = torch.zeros((1, n), device="cuda")
    ctx.add_rms_norm(want_res, _dev(first[1:2]), _dev(first[2:3]), 1e-6, want_hid)
    ctx.matmul(w, want_hid, want, rule=ol.ACT_G128)
    ctx.step_matmul(w, x, u, g, 1e-6, res, y=y, hidden_out=hid)
    ctx.sync()
    assert torch.equal(y, want)
    if where != "new residual":
        assert torch.equal(res, want_res)
    if hid is not None:
        assert torch.equal(hid, want_hid)
    w.free()


@pytest.mark.parametrize("k", [128, 4224])
def test_step_matmul_refuses_rows_that_overlap(ctx, k):
    """The new residual over a part of a row that is read, the normalised row over another output
    or over a part of a row that is read."""
    import torch
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, 1, 24, k), 24, k)
    rows = torch.ones(8 * k, device="cuda")
    row = lambda at: rows[at:at + k].view(1, k)
    x, u, g, r = (row(i * k) for i in range(4))
    y = torch.zeros((1, 24), device="cuda")
    for kw in (dict(residual_out=row(4), y=y), dict(residual_out=row(2 * k - 4), y=y),
               dict(residual_out=row(2 * k), y=y),
               dict(residual_out=r, y=y, hidden_out=row(4)),
               dict(residual_out=r, y=y, hidden_out=row(k + 4)),
               dict(residual_out=r, y=y, hidden_out=g),
               dict(residual_out=r, y=y, hidden_out=r),
               dict(residual_out=r, y=y, hidden_out=row(4 * k - 4)),
               dict(residual_out=r, y=rows[5 * k:5 * k + 24].view(1, 24), hidden_out=row(5 * k))):
        with pytest.raises(pkg.capi.B200W4Error, match="overlap"):
            ctx.step_matmul(w, x, u, g, 1e-6, **kw)
    ctx.step_matmul(w, x, u, g, 1e-6, r, y=y, hidden_out=row(4 * k))  # side by side: accepted
    ctx.sync()
    w.free()


@pytest.mark.parametrize("k", [128, 256, 384])
def test_step_matmul_of_a_short_row_alone(ctx, k):
    """No update: the sum of squares in b2w4_rms_norm's order, one warp up to 256 values."""
    import torch
    n = 64
    w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
    rng = np.random.default_rng(k)
    for _ in range(20):
        x, g = (_dev(rng.normal(0, 1, (1, k)).astype(np.float32)) for _ in range(2))
        hid, hid_t, res, want_hid = (torch.zeros((1, k), device="cuda") for _ in range(4))
        y, want = (torch.zeros((1, n), device="cuda") for _ in range(2))
        tok, want_tok = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
        ctx.step_matmul(w, x, None, g, 1e-6, res, y=y, hidden_out=hid)
        ctx.step_matmul(w, x, None, g, 1e-6, None, tokens=tok, hidden_out=hid_t)
        ctx.rms_norm(x, g, 1e-6, want_hid)
        ctx.matmul(w, want_hid, want, rule=ol.ACT_G128)
        ctx.matmul_argmax(w, want_hid, want_tok)
        ctx.sync()
        assert torch.equal(hid, want_hid) and torch.equal(hid_t, want_hid)
        assert torch.equal(y, want) and torch.equal(tok, want_tok) and torch.equal(res, x)
    w.free()


@pytest.mark.parametrize("past,heads,kv_heads,dim", [(40, 4, 2, 128), (1000, 32, 8, 128),
                                                     (300, 6, 6, 64)])
@pytest.mark.parametrize("at", [0, 64])
def test_attention_step_over_its_own_rows(ctx, past, heads, kv_heads, dim, at):
    """The result in the place of the query rows, or over the later ones and the keys, as the two
    calls allow: they have read every row before the first value is stored."""
    import torch
    rng = np.random.default_rng(past + dim + at)
    cap = past + 70
    first = rng.normal(0, 1, (1, (heads + 2 * kv_heads) * dim)).astype(np.float32)
    qw, kw = (_dev(rng.normal(1, 0.1, dim).astype(np.float32)) for _ in range(2))
    cos, sin = (_dev(t) for t in pkg.decoder.rope_tables(range(cap), dim, 1e6))
    first_kv = [rng.normal(0, 1, (kv_heads, cap, dim)).astype(np.float32) for _ in range(2)]
    want_kv, cache = [_dev(c) for c in first_kv], [_dev(c) for c in first_kv]
    q, want = (torch.zeros((1, heads * dim), device="cuda") for _ in range(2))
    ctx.qkv_prepare(_dev(first), 1, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, past, q,
                    *want_kv, cap)
    ctx.attention(q, None, None, *want_kv, want, 1, heads, kv_heads, dim, past, cap, dim ** -0.5)
    qkv = _dev(first)
    out = qkv.view(-1)[at:at + heads * dim].view(1, -1)
    ctx.attention_step(qkv, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, past,
                       torch.zeros_like(q), *cache, out, cap, dim ** -0.5)
    ctx.sync()
    for a, b in zip(cache, want_kv):
        assert torch.equal(a, b)
    assert torch.equal(out, want)


@pytest.mark.parametrize("f32", [False, True])
def test_step_matmul_swiglu_longest_rows(ctx, f32):
    """The longest row that the header names, and one that is refused before anything is written."""
    import torch
    for k in (20480, 22016):
        n = 32
        blocks = np.array(pkg.synth.bg128_weight(3, n + k, n, k), copy=True)
        if f32:  # scales that fp16 cannot hold
            blocks.reshape(-1, 544)[:, :32].view(np.float32)[:] *= np.float32(1.0001)
        w = ctx.upload_weight(blocks, n, k)
        x, u, g = (torch.randn((1, k), device="cuda") for _ in range(3))
        res, hid, y = torch.zeros((1, k), device="cuda"), torch.zeros((1, k), device="cuda"), \
            torch.zeros((1, n // 2), device="cuda")
        if k == 20480:
            merged, want = torch.zeros((1, n), device="cuda"), torch.zeros_like(y)
            ctx.step_matmul(w, x, u, g, 1e-6, res, y=y, swiglu=True, hidden_out=hid)
            ctx.matmul(w, hid, merged, rule=ol.ACT_G128)
            ctx.swiglu(merged, want)
            ctx.sync()
            assert torch.equal(y, want) and bool(y.any())
        else:
            with pytest.raises(pkg.capi.B200W4Error, match="too long"):
                ctx.step_matmul(w, x, u, g, 1e-6, res, y=y, swiglu=True, hidden_out=hid)
            ctx.sync()
            assert not res.any() and not hid.any() and not y.any()
        w.free()


def _attention_fp64_cuda(q, kc, vc, past, scale):
    """_attention_fp64 on device tensors."""
    import torch
    tokens, heads, dim = q.shape
    kv_heads, keys = kc.shape[0], past + tokens
    out = torch.empty((tokens, heads, dim), dtype=torch.float64, device="cuda")
    hidden = torch.arange(keys, device="cuda")[None] > \
        past + torch.arange(tokens, device="cuda")[:, None]
    for h in range(heads):
        g = h // (heads // kv_heads)
        s = (q[:, h].double() @ kc[g, :keys].double().T) * scale
        p = torch.softmax(s.masked_fill_(hidden, float("-inf")), 1)
        v = torch.where((p > 0).any(0)[:, None], vc[g, :keys].double(), 0.0)
        out[:, h] = p @ v
    return out


LONG_RUNS = [  # tokens, past, heads, kv_heads, dim: the tensor-core kernel
    (256, 128, 24, 8, 128),   # the shortest, three heads per kv head: 126 of 128 rows in use
    (1473, 3, 32, 8, 128),    # ragged last tile and last block of keys
    (261, 700, 40, 1, 128),   # 40 heads per kv head: 120 rows
    (400, 64, 64, 1, 64), (1500, 1, 16, 16, 64), (640, 0, 40, 8, 64)]


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", LONG_RUNS)
def test_long_runs_on_tensor_cores(ctx, tokens, past, heads, kv_heads, dim):
    """Runs whose products go to the tensor cores in three bf16 pieces, against 64 bits, and no
    further from them than the one-row arithmetic in fp32 (a tenth more for the luck of one
    draw); the position on the device leaves the same bits; value rows past the position are NaN.
    Tolerance as for the split kernel."""
    import torch
    capacity, scale = max(384, past + tokens + 9), dim ** -0.5
    g = torch.Generator(device="cuda").manual_seed(tokens + dim)
    q = torch.randn((tokens, heads, dim), device="cuda", generator=g)
    kc, vc = (torch.randn((kv_heads, capacity, dim), device="cuda", generator=g)
              for _ in range(2))
    vc[:, past + tokens:] = float("nan")
    ctx_row = _row_context()
    outs = []
    for c, past_dev in ((ctx, None), (ctx_row, None),
                        (ctx, torch.full((1,), past, dtype=torch.int32, device="cuda"))):
        out = torch.zeros_like(q)
        c.attention(q, None, None, kc, vc, out, tokens, heads, kv_heads, dim,
                    past if past_dev is None else 0, capacity, scale, past_dev)
        c.sync()
        outs.append(out)
    ctx_row.close()
    want = _attention_fp64_cuda(q, kc, vc, past, scale)
    err, row_err = (float((o.double() - want).norm() / want.norm()) for o in outs[:2])
    assert err < 1e-5 and err < 1.1 * row_err
    assert torch.equal(outs[0], outs[2])
    assert not torch.equal(outs[0], outs[1])  # not the tile kernel, which has the row's bits


@pytest.mark.parametrize("tokens,heads,kv_heads,dim", [(256, 24, 8, 128), (640, 40, 8, 64)])
def test_long_runs_with_extreme_values(ctx, tokens, heads, kv_heads, dim):
    """Keys of probability zero whose value rows are not finite, values near the largest number,
    values so small that bf16 pieces would lose bits, a value row of NaN that is seen: as in
    test_attention_ignores_value_rows_of_zero_probability, tolerances from there (640 terms:
    4e-5).  Such tiles are done in fp32, the others are not touched by it."""
    import torch
    rng = np.random.default_rng(dim)
    keys = tokens + 300
    q1, k, v = _staged(rng, heads, kv_heads, dim, keys, [0.0, 80.0, 160.0])
    qd = _dev(np.repeat(q1, tokens, axis=0))
    k[:] = 0.0
    k[:100, :, 0] = -160.0  # probability zero against the rest
    kc, vc = (_dev(np.ascontiguousarray(x.transpose(1, 0, 2))) for x in (k, v))

    def run():
        out = torch.zeros((tokens, heads, dim), device="cuda")
        ctx.attention(qd, None, None, kc, vc, out, tokens, heads, kv_heads, dim, 300, keys, 1.0)
        ctx.sync()
        return out

    clean = vc.clone()
    clean[:, :100] = 0.0
    want = _attention_fp64_cuda(qd, kc, clean, 300, 1.0)
    for bad in (float("nan"), float("inf"), float("-inf")):
        vc[:, 3] = bad
        vc[:, 50, dim // 2] = bad
        got = run()
        assert torch.isfinite(got).all()
        assert float((got.double() - want).norm() / want.norm()) < 4e-5
    vc[:, :100] = 0.0
    for size, tol in ((3e38, 1e-5), (1e-34, 4e-5)):
        vc[:, 100:] = torch.rand_like(vc[:, 100:]) * 0.5 + 0.5
        want = _attention_fp64_cuda(qd, kc, vc, 300, 1.0)
        vc *= size
        got = run().double() / size
        assert float((got - want).norm() / want.norm()) < tol
    vc.normal_()
    vc[:, 300 + tokens // 2] = float("nan")  # seen by the second half
    got = run()
    assert torch.isnan(got[tokens // 2:]).all() and torch.isfinite(got[:tokens // 2]).all()


def _step_both_ways(ctx, qkv, heads, kv_heads, dim, qw, kw, cos, sin, past, cap, cache):
    """A decode step with its operators apart and in one launch, the position given by the host and
    on the device: the same bits in the caches and in the result, which is returned."""
    import torch
    pos = torch.tensor([past], dtype=torch.int32, device="cuda")
    for position, host in ((None, past), (pos, 0)):
        want_kv, got_kv = ([c.clone() for c in cache] for _ in range(2))
        q, want, got = (torch.zeros((1, heads * dim), device="cuda") for _ in range(3))
        ctx.qkv_prepare(qkv, 1, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, host, q, *want_kv,
                        cap, position)
        ctx.attention(q, None, None, *want_kv, want, 1, heads, kv_heads, dim, host, cap,
                      dim ** -0.5, position)
        ctx.attention_step(qkv, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, host,
                           torch.zeros_like(q), *got_kv, got, cap, dim ** -0.5, position)
        ctx.sync()
        for a, b in zip(got_kv, want_kv):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    return want


RING_STEPS = [  # past, heads, kv_heads, dim, cap
    (0, 8, 2, 128, 96), (3, 8, 2, 128, 96), (94, 4, 1, 64, 96),      # one block per kv head
    (127, 32, 8, 128, 800), (159, 32, 8, 128, 800), (703, 6, 6, 128, 800),
    (6015, 32, 8, 128, 6100), (5500, 16, 8, 64, 6100),               # the ring turns over
    (4095, 4, 1, 128, 4096), (2999, 2, 2, 64, 3001)]


@pytest.mark.parametrize("past,heads,kv_heads,dim,cap", RING_STEPS)
def test_attention_step_through_the_ring(ctx, past, heads, kv_heads, dim, cap):
    """A decode step whose blocks have a multiprocessor each brings the cache in through a ring:
    the bits of the separate operators at the edges of a slot's keys, with fewer keys than warps,
    with more slots than the ring has, and with the new key in the first and in the last slot.
    Rows past the position are NaN; all scores and results are finite, so what is compared is made
    of the rows that the ring brought."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(past + dim)
    qkv = torch.randn((1, (heads + 2 * kv_heads) * dim), device="cuda", generator=g)
    qw, kw = (torch.rand(dim, device="cuda", generator=g) + 0.5 for _ in range(2))
    cos, sin = (_dev(t) for t in pkg.decoder.rope_tables(range(cap), dim, 1e6))
    cache = [torch.randn((kv_heads, cap, dim), device="cuda", generator=g) for _ in range(2)]
    for c in cache:
        c[:, past + 1:] = float("nan")
    want = _step_both_ways(ctx, qkv, heads, kv_heads, dim, qw, kw, cos, sin, past, cap, cache)
    assert bool(torch.isfinite(want).all())


@pytest.mark.parametrize("past,heads,kv_heads,dim,cap", RING_STEPS[2:])
def test_ring_ignores_value_rows_of_zero_probability(ctx, past, heads, kv_heads, dim, cap):
    """Keys at both ends of the cache that point away from every query head of their kv head, which
    are alike: probability zero for all of them, so their value rows of NaN count for nothing and
    the result stays the one that the ring's rows give, against 64 bits too."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(past + dim + 1)
    rep = heads // kv_heads
    qkv = torch.randn((1, (heads + 2 * kv_heads) * dim), device="cuda", generator=g)
    rows = qkv.view(heads + 2 * kv_heads, dim)
    alike = rows[:kv_heads].repeat_interleave(rep, 0).clone()
    rows[:heads] = alike + 0.1 * rows[:heads]
    qw, kw = (torch.rand(dim, device="cuda", generator=g) + 0.5 for _ in range(2))
    cos, sin = (_dev(t) for t in pkg.decoder.rope_tables(range(cap), dim, 1e6))
    cache = [torch.randn((kv_heads, cap, dim), device="cuda", generator=g) for _ in range(2)]
    q = torch.zeros((1, heads * dim), device="cuda")
    kv = [c.clone() for c in cache]
    ctx.qkv_prepare(qkv, 1, heads, kv_heads, dim, qw, kw, 1e-6, cos, sin, past, q, *kv, cap)
    ctx.sync()
    away = -100.0 * q.view(kv_heads, rep, dim).mean(1)
    for key in (5, past - 1):
        cache[0][:, key], cache[1][:, key] = away, float("nan")
    for c in cache:
        c[:, past + 1:] = float("nan")
    want = _step_both_ways(ctx, qkv, heads, kv_heads, dim, qw, kw, cos, sin, past, cap, cache)
    assert bool(torch.isfinite(want).all())
    for c, new in zip(cache, kv):
        c[:, past] = new[:, past]
    cache[1][:, [5, past - 1]] = 0.0
    ref = _attention_fp64_cuda(q.view(1, heads, dim), *cache, past, dim ** -0.5)
    got = want.view(1, heads, dim).double()
    assert float((got - ref).norm() / ref.norm()) < 1e-5


@pytest.mark.parametrize("n,k,f32", [(18960, 2560, True), (9600, 4224, False), (37920, 1280, False),
                                     (19456, 384, False)])
def test_step_matmul_with_twice_the_warps(ctx, n, k, f32):
    """SwiGLU over more pairs of tiles than two blocks per multiprocessor hold: one block of twice
    the warps, with the norm inside and (rows beyond 4096 values) in front, fp32 scales, a last
    block with fewer pairs; and short rows, whose copy is larger than the sums it lies over."""
    import torch
    rng = np.random.default_rng(n + k)
    blocks = pkg.synth.bg128_weight(3, n + k, n, k)
    if f32:
        blocks = np.array(blocks, copy=True)
        s = blocks.reshape(-1, 544)[:, :32].copy().view(np.float32)
        blocks.reshape(-1, 544)[:, :32] = (s * np.float32(1.0000001)).view(np.uint8)
    w = ctx.upload_weight(blocks, n, k)
    x, u, g = (_dev(rng.normal(m, s, (1, k)).astype(np.float32))
               for m, s in ((0, 2), (0, 1), (1, 0.2)))
    res, hid = (torch.zeros((1, k), device="cuda") for _ in range(2))
    want = torch.zeros((1, n), device="cuda")
    act, want_act = (torch.zeros((1, n // 2), device="cuda") for _ in range(2))
    ctx.step_matmul(w, x, u, g, 1e-6, res, y=act, swiglu=True)
    want_res = x.clone()
    ctx.add_rms_norm(want_res, u, g, 1e-6, hid)
    ctx.matmul(w, hid, want, rule=ol.ACT_G128)
    ctx.swiglu(want, want_act)
    ctx.sync()
    assert torch.equal(res, want_res) and torch.equal(act, want_act)
    w.free()


def test_shared_memory_just_below_the_default_limit():
    """A first call whose dynamic part is below 48 KiB and whose whole is not (SwiGLU of two tiles of
    [4096, 4736]: 49 000 bytes and 768): in a process of its own, where no larger call came before."""
    code = """
import sys; sys.path.insert(0, %r)
import torch
from __graft_entry__ import load_package
pkg = load_package()
ctx = pkg.capi.Context(0)
n, k = 4096, 4736
w = ctx.upload_weight(pkg.synth.bg128_weight(3, 1, n, k), n, k)
x = torch.randn((1, k), device="cuda")
out = [torch.zeros((1, s), device="cuda") for s in (k, n // 2, k, n, n // 2)]
one = torch.ones(k, device="cuda")
ctx.step_matmul(w, x, None, one, 1e-6, out[0], y=out[1], swiglu=True)
ctx.rms_norm(x, one, 1e-6, out[2])
ctx.matmul(w, out[2], out[3], rule=128)
ctx.swiglu(out[3], out[4])
ctx.sync()
assert torch.equal(out[1], out[4])
""" % os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("tokens,heads,dim", [(600, 64, 128), (1000, 64, 64)])
def test_long_runs_take_exp_in_64_bits(ctx, tokens, heads, dim):
    """The tensor-core kernel's probabilities are exp in 64 bits rounded once.  Two keys count, of
    scores 0 and x <= 0 (both exact), with values that show p / (1 + p) and 1 / (1 + p); all further
    scores are -1000.  Its exp is within 2^-43 of e^x, 2^-18 of a unit in the last place: of the
    results, 2^-17 are expected to be rounded to the neighbour, 1e-4 are allowed (an exp in 32 bits
    has some in a hundred).  From -69 on, as results below 2^-100 send a tile to the fp32 form."""
    import torch
    rng = np.random.default_rng(dim)
    n, past, keys = tokens * heads, 64, 64 + tokens
    x = np.where(rng.random(n) < 0.5, rng.uniform(-69, 0, n), -10.0 ** rng.uniform(-7, 1.8, n))
    x = x.astype(np.float32)
    q = np.zeros((tokens, heads, dim), np.float32)
    q[..., 0], q[..., 1] = x.reshape(tokens, heads), 1.0
    k, v = (np.zeros((1, max(384, keys), dim), np.float32) for _ in range(2))
    k[0, 1, 0], k[0, 2:, 1] = 1.0, -1000.0
    v[0, 0, 0], v[0, 1, 1] = 1.0, 1.0
    out = torch.zeros((tokens, heads, dim), device="cuda")
    ctx.attention(_dev(q), None, None, _dev(k), _dev(v), out, tokens, heads, 1, dim, past,
                  k.shape[1], 1.0)
    ctx.sync()
    p = np.exp(x.astype(np.float64)).astype(np.float32)
    total = np.float32(1.0) + p
    want = np.stack([np.float32(1.0) / total, p / total], 1)
    got = out.cpu().numpy().reshape(n, dim)
    assert not got[:, 2:].any()
    assert (got[:, :2] != want).mean() < 1e-4
    assert np.abs(got[:, :2] - want).max() < 2.0 ** -23


@pytest.mark.parametrize("tokens,heads,kv_heads,dim", [(256, 24, 8, 128), (640, 40, 8, 64)])
def test_long_runs_whose_pieces_lose_bits(ctx, tokens, heads, kv_heads, dim):
    """Queries, keys, values and probabilities with bits below 2^-133, which three bf16 pieces drop:
    as precise as in fp32.  Keys or queries near 2^-124 against rows near 2^124 (tolerance of the
    forms); values near 2^-138 averaged (they and the result are multiples of 2^-149); one key with
    probability p and value v, where a key of value zero has all the rest: a product of three
    roundings, 2^-22, and half of 2^-149 where it is not a normal number."""
    import torch
    past, g = 300, torch.Generator(device="cuda").manual_seed(dim)
    keys = past + tokens

    def rand(*shape):
        return torch.randn(shape, device="cuda", generator=g)

    def run(q, kc, vc):
        out = torch.full((tokens, heads, dim), 7.0, device="cuda")
        ctx.attention(q, None, None, kc, vc, out, tokens, heads, kv_heads, dim, past, keys, 1.0)
        ctx.sync()
        return out.double(), _attention_fp64_cuda(q, kc, vc, past, 1.0)

    q, kc, vc = rand(tokens, heads, dim), rand(kv_heads, keys, dim), rand(kv_heads, keys, dim)
    q *= dim ** -0.5
    for up, down in ((q, kc), (kc, q)):
        a, b = up * 2.0 ** 124, down * 2.0 ** -124
        got, want = run(*((a, b) if up is q else (b, a)), vc)
        assert float((got - want).norm() / want.norm()) < 1e-5
    got, want = run(torch.zeros_like(q), kc, (torch.rand_like(vc) + 0.5) * 2.0 ** -138)
    assert float((got - want).abs().max()) <= 2.0 ** -149 and bool(got.all())

    q[:], kc[:], vc[:] = 0.0, 0.0, 0.0
    q[..., 0] = kc[:, 1, 0] = 1.0
    kc[:, 2:, 0] = -1000.0
    for x, v in ((-85.0, 1e38), (-80.0, 3e33), (-86.0, 2.0 ** 30), (-84.5, 2.0 ** 30),
                 (-74.2, 2.0 ** -21), (-60.0, 2.0 ** -50), (-74.2, 2.0 ** -39), (-103.0, 1e30)):
        kc[:, 1, 0] = x
        vc[:, 1, ::2] = v
        got, want = run(q, kc, vc)
        # exp(-103) in 32 bits is 1.3e-45 or 2^-149
        p = float(np.float32(np.exp(np.float64(x))))
        want *= p / np.exp(x)
        assert float((got - want).abs().max()) <= 2.0 ** -22 * float(want.max()) + 2.0 ** -149
        assert not got[..., 1::2].any()
    # probabilities that lose bits and count for nothing: in pieces, with zeros and without
    kc[:, 1, 0] = -80.0
    vc.copy_(rand(*vc.shape))
    got, want = run(q, kc, vc)
    assert float((got - want).norm() / want.norm()) < 1e-5
    vc[:, 0, ::2] = 0.0
    got, want = run(q, kc, vc)
    assert float((got - want).norm() / want.norm()) < 1e-5
    tiny = float((got - want)[..., ::2].norm() / want[..., ::2].norm())
    assert tiny < 1e-5


@pytest.mark.parametrize("tokens,past,heads,kv_heads,dim", [(256, 128, 24, 8, 128), (640, 0, 40, 8, 64),
                                                            (2000, 6000, 4, 1, 128)])
@pytest.mark.parametrize("kind", ["values of one sign", "flat", "sharp", "large scores"])
def test_long_runs_on_other_inputs(ctx, tokens, past, heads, kv_heads, dim, kind):
    """The tensor-core kernel is nearer to 64 bits than the one-row arithmetic in fp32 where its
    truncated sums are all of one sign, where every key counts or only a few do, and where all scores
    are large."""
    import torch
    keys, scale = past + tokens, dim ** -0.5
    g = torch.Generator(device="cuda").manual_seed(tokens + dim + 1)
    q = torch.randn((tokens, heads, dim), device="cuda", generator=g)
    kc, vc = (torch.randn((kv_heads, max(384, keys), dim), device="cuda", generator=g)
              for _ in range(2))
    if kind == "values of one sign":
        vc = torch.rand_like(vc) * 0.5 + 0.5
    elif kind == "flat":
        q, vc = q * 0.01, vc.abs()
    elif kind == "sharp":
        q = q * 30.0
    else:
        q, kc = (q * 0.2).clamp(-0.9, 0.9) + 8.0, (kc * 0.2).clamp(-0.9, 0.9) + 1.0
    ctx_row = _row_context()
    outs = []
    for c in (ctx, ctx_row):
        out = torch.zeros_like(q)
        c.attention(q, None, None, kc, vc, out, tokens, heads, kv_heads, dim, past, kc.shape[1],
                    scale)
        c.sync()
        outs.append(out)
    ctx_row.close()
    want = _attention_fp64_cuda(q, kc, vc, past, scale)
    err, row_err = (float((o.double() - want).norm() / want.norm()) for o in outs)
    assert err < row_err < 1e-5


def test_step_matmul_keeps_the_cap_on_tiles():
    """B2W4_GEMV_TPC caps the tiles of a block, also where a SwiGLU would else take blocks of twice
    the warps: one pair of tiles each, the default's bits."""
    import torch
    driver = pytest.importorskip("cuda.bindings.driver")
    n, k, stream = 9728, 2560, torch.cuda.Stream()
    blocks = pkg.synth.bg128_weight(3, n + k, n, k)
    x, one = torch.randn((1, k), device="cuda"), torch.ones(k, device="cuda")
    results, grids = [], []
    for cap in (None, "2"):
        if cap:
            os.environ["B2W4_GEMV_TPC"] = cap
        try:
            c = pkg.capi.Context(0)
        finally:
            os.environ.pop("B2W4_GEMV_TPC", None)
        w = c.upload_weight(blocks, n, k)
        res, y = torch.zeros((1, k), device="cuda"), torch.zeros((1, n // 2), device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph, stream=stream):
            c.set_stream(torch.cuda.current_stream().cuda_stream)
            c.step_matmul(w, x, None, one, 1e-6, res, y=y, swiglu=True)
        raw = driver.CUgraph(init_value=graph.raw_cuda_graph())
        count = driver.cuGraphGetNodes(raw)[-1]
        assert count == 1
        node = driver.cuGraphGetNodes(raw, count)[1][0]
        grids.append(driver.cuGraphKernelNodeGetParams(node)[1].gridDimX)
        graph.instantiate()
        graph.replay()
        torch.cuda.synchronize()
        results.append(y)
        del graph
        c.set_stream(torch.cuda.current_stream().cuda_stream)
        w.free()
        c.close()
    assert grids[1] == n // 16 and grids[0] < grids[1]
    assert torch.equal(*results)
