"""GPU parity of the W4G128 matmul path (through the C ABI) against the CPU oracle:
int32 group accumulators and fp32 outputs bit-exact, on the reference's own golden cases,
on seeded synthetic shapes, and at the benchmark's full size through properties."""
import numpy as np
import pytest

import oracle_lib as ol
from golden_util import MATMUL_CASES, case, rel_l2
from __graft_entry__ import load_package

pkg = load_package()
pytestmark = pytest.mark.gpu


def _forced_ctx(kind):
    import os
    os.environ["B2W4_GEMM"] = kind
    try:
        return pkg.capi.Context(0)
    finally:
        del os.environ["B2W4_GEMM"]


@pytest.fixture(scope="module")
def ctx_tc():
    """A context that sends every many-row matmul to the tcgen05 kernel."""
    c = _forced_ctx("tc")
    yield c
    c.close()


@pytest.fixture(scope="module")
def ctx_mma():
    """A context that sends every many-row matmul that fits to the mma.sync kernel."""
    c = _forced_ctx("mma")
    yield c
    c.close()


@pytest.fixture(scope="module")
def ctx():
    c = pkg.capi.Context(0)
    yield c
    c.close()


def run_gpu(ctx, blocks, n, k, x, rule=ol.ACT_G128, act=0, begin=0, length=-1, sums=True,
            pad=0):
    import torch
    m = x.shape[0]
    w = ctx.upload_weight(blocks, n, k)
    xd = torch.zeros((m, k + pad), dtype=torch.float32, device="cuda")
    xd[:, :k] = torch.from_numpy(x)
    yd = torch.full((m, n + pad), -7.0, dtype=torch.float32, device="cuda")
    ctx.matmul(w, xd, yd, rule=rule, act=act, act_begin=begin, act_len=length)
    out_s = None
    if sums:
        per = k // 128 if rule == ol.ACT_G128 else k // 32
        sd = torch.zeros((m, n, per), dtype=torch.int32, device="cuda")
        ctx.group_sums(w, xd, sd, rule=rule)
        ctx.sync()
        out_s = sd.cpu().numpy()
    ctx.sync()
    y = yd.cpu().numpy()
    if pad:
        assert (y[:, n:] == -7.0).all(), "wrote past N"
    w.free()
    return y[:, :n], out_s


@pytest.mark.parametrize("name", MATMUL_CASES)
@pytest.mark.parametrize("rule", [ol.ACT_G128, ol.ACT_G32])
def test_golden_cases_bit_exact(ctx, name, rule):
    c = case(name)
    n, k = c["q"].shape
    y_ref, s_ref = ol.matmul_w4(c["blocks"], n, k, c["a"], rule=rule, want_sums=True)
    y, s = run_gpu(ctx, c["blocks"], n, k, c["a"], rule=rule, pad=3)
    assert (s == s_ref).all()
    assert y.tobytes() == y_ref.tobytes()
    # and inside the reference CUDA test's own bound against its W4A32 answer
    assert np.max(np.abs(y - c["y_ref_w4a32"])) < 5e-2


def test_quantiser_bit_exact(ctx):
    import torch
    c = case("quant_edge")
    x = np.stack([c["x"], case("synth_m5_k512_n72")["a"][2]])
    xd = torch.from_numpy(x).cuda()
    for rule in (ol.ACT_G128, ol.ACT_G32):
        q = torch.zeros((2, 512), dtype=torch.int8, device="cuda")
        s = torch.zeros((2, 512 // rule), dtype=torch.float32, device="cuda")
        ctx.quantize(xd, q, s, rule=rule)
        ctx.sync()
        for r in range(2):
            if rule == ol.ACT_G128:
                q_ref, s_ref = ol.quantize_g128(x[r])
            else:
                q_ref, s_ref = ol.quantize_g32(x[r:r + 1])
                q_ref, s_ref = q_ref[0], s_ref[0]
            assert (q[r].cpu().numpy() == q_ref).all()
            assert s[r].cpu().numpy().tobytes() == s_ref.tobytes()


@pytest.mark.parametrize("m,n,k", [(1, 8, 128), (1, 7, 128), (2, 13, 256), (3, 264, 512),
                                   (4, 1000, 768), (5, 72, 512), (9, 40, 1280),
                                   (1, 2560, 9728), (4, 520, 4096), (6, 328, 640),
                                   (7, 8, 128), (8, 1304, 2560), (8, 2560, 9728)])
@pytest.mark.parametrize("rule", [ol.ACT_G128, ol.ACT_G32])
def test_synthetic_shapes_bit_exact(ctx, m, n, k, rule):
    if rule == ol.ACT_G32 and k > 4096:
        pytest.skip("per-32 rule is exercised at smaller K")
    blocks = pkg.synth.bg128_weight(20261125, n + k, n, k)
    x = pkg.synth.activations(7, m, m, k)
    x[0, :128] = 0.0  # an all-zero activation group (scale 1, codes 0)
    y_ref, s_ref = ol.matmul_w4(blocks, n, k, x, rule=rule, want_sums=True)
    y, s = run_gpu(ctx, blocks, n, k, x, rule=rule, pad=5)
    assert (s == s_ref).all()
    assert y.tobytes() == y_ref.tobytes()


def test_fp32_scale_plane_when_not_fp16_exact(ctx):
    n, k, m = 64, 256, 2
    blocks = pkg.synth.bg128_weight(3, 3, n, k).copy()
    b = blocks.reshape(-1, 544)
    b[:, :32].view(np.float32)[:] *= np.float32(1.0001)  # no longer fp16-representable
    x = pkg.synth.activations(7, 5, m, k)
    w = ctx.upload_weight(blocks, n, k)
    assert not w.scales_fp16
    w.free()
    y, s = run_gpu(ctx, blocks, n, k, x)
    y_ref, s_ref = ol.matmul_w4(blocks, n, k, x, want_sums=True)
    assert (s == s_ref).all() and y.tobytes() == y_ref.tobytes()


@pytest.mark.parametrize("act,begin,length", [(1, 0, -1), (1, 8, 40), (3, 16, 8), (4, 0, 72),
                                              (2, 0, -1), (1, 5, 0)])
def test_fused_activation_range(ctx, act, begin, length):
    c = case("synth_m5_k512_n72")
    y, _ = run_gpu(ctx, c["blocks"], 72, 512, c["a"], act=act, begin=begin, length=length,
                   sums=False)
    y_ref = ol.apply_activation(ol.matmul_w4(c["blocks"], 72, 512, c["a"]), act, begin, length)
    if act == 2:  # GELU goes through tanh: tolerance, 1e-6 relative
        assert rel_l2(y, y_ref) < 1e-6
    else:
        assert y.tobytes() == y_ref.tobytes()


def test_host_entry_point_and_weight_copy_ownership(ctx):
    """matmul_host stages host tensors itself; the uploaded weight is a copy, so zeroing
    the caller's blocks afterwards must not change results (the reference CUDA test does
    the same, tests/test_cuda_backend.cpp:1259-1261)."""
    n, k, m = 200, 384, 3
    blocks = pkg.synth.bg128_weight(11, 4, n, k)
    x = pkg.synth.activations(7, 6, m, k)
    y_ref = ol.matmul_w4(blocks, n, k, x)
    w = ctx.upload_weight(blocks, n, k)
    blocks[:] = 0
    y = np.zeros((m, n), dtype=np.float32)
    ctx.matmul_host(w, x, y)
    assert y.tobytes() == y_ref.tobytes()
    w.free()


@pytest.mark.parametrize("m", [1, 24])
def test_repeated_pinned_host_calls(ctx, m):
    """A host call repeated through a bound closure on the same pinned buffers: the buffers'
    current contents are used every time, also after a larger call in between has moved the
    context's staging buffers, and after the weight was freed and another one uploaded."""
    import torch
    n, k = 328, 640
    blocks = pkg.synth.bg128_weight(11, 9, n, k)
    w = ctx.upload_weight(blocks, n, k)
    xh = torch.zeros((m, k), dtype=torch.float32).pin_memory()
    yh = torch.zeros((m, n), dtype=torch.float32).pin_memory()
    call = ctx.bind_matmul_host(w, xh.numpy(), yh.numpy())
    for step in range(5):
        x = pkg.synth.activations(7, 500 + step, m, k)
        xh.numpy()[:] = x
        yh.zero_()
        call()
        assert yh.numpy().tobytes() == ol.matmul_w4(blocks, n, k, x).tobytes(), step
        if step == 2:  # a larger host call in between moves the staging buffers
            big_n, big_m = 2048, 64
            wb = ctx.upload_weight(pkg.synth.bg128_weight(11, 10, big_n, k), big_n, k)
            xb = pkg.synth.activations(7, 600, big_m, k)
            yb = np.zeros((big_m, big_n), dtype=np.float32)
            ctx.matmul_host(wb, xb, yb)
            wb.free()
    w.free()
    # the same buffers with another weight
    blocks2 = pkg.synth.bg128_weight(11, 11, n, k)
    w2 = ctx.upload_weight(blocks2, n, k)
    call2 = ctx.bind_matmul_host(w2, xh.numpy(), yh.numpy())
    for _ in range(3):
        call2()
        assert yh.numpy().tobytes() == ol.matmul_w4(blocks2, n, k, xh.numpy()).tobytes()
    w2.free()


def test_bad_arguments_are_errors(ctx):
    import torch
    blocks = pkg.synth.bg128_weight(1, 1, 8, 128)
    with pytest.raises(pkg.capi.B200W4Error):
        ctx.upload_weight(blocks, 8, 100)           # K not a multiple of 128
    w = ctx.upload_weight(blocks, 8, 128)
    x = torch.zeros((1, 128), device="cuda")
    y = torch.zeros((1, 8), device="cuda")
    with pytest.raises(pkg.capi.B200W4Error):
        ctx.matmul(w, x, y, rule=16)                # reference rejects group size 16 too
    with pytest.raises(pkg.capi.B200W4Error):
        ctx.matmul(w, x, y, lda=64)
    ctx.matmul(w, x, y)                             # the context stays usable
    ctx.sync()
    w.free()


def test_config1_full_size_properties(ctx):
    """M=1, K=2560, N=9728 (benchmark configuration 1).  The oracle runs the whole case in
    well under a second, so this is a direct bit-exact check, plus the size-independent
    properties: homogeneity under power-of-two scaling of x (quantisation is scale
    invariant for exact scalings) and block-row independence."""
    n, k = 9728, 2560
    blocks = pkg.synth.bg128_weight(20261125, 1, n, k)
    x = pkg.synth.activations(7, 0, 1, k)
    y_ref, s_ref = ol.matmul_w4(blocks, n, k, x, want_sums=True)
    y, s = run_gpu(ctx, blocks, n, k, x)
    assert (s == s_ref).all()
    assert y.tobytes() == y_ref.tobytes()
    y2, s2 = run_gpu(ctx, blocks, n, k, x * 4.0)
    assert (s2 == s).all() and (y2 == y * 4.0).all()
    half = ol.bg128_bytes(n // 2, k)
    y_top, _ = run_gpu(ctx, blocks[:half].copy(), n // 2, k, x, sums=False)
    assert y_top.tobytes() == y[:, :n // 2].tobytes()


@pytest.mark.parametrize("m", [4, 8, 16, 33, 64])
def test_config2_decode_sweep(ctx, m):
    n, k = 9728, 2560
    blocks = pkg.synth.bg128_weight(20261125, 1, n, k)
    x = pkg.synth.activations(7, m, m, k)
    y, _ = run_gpu(ctx, blocks, n, k, x, sums=False)
    y_ref = ol.matmul_w4(blocks, n, k, x)
    assert y.tobytes() == y_ref.tobytes()


@pytest.mark.parametrize("m,n,k", [(129, 72, 256), (300, 200, 512), (256, 1000, 1280),
                                   (37, 2560, 9728)])
@pytest.mark.parametrize("kind", ["mma", "tc"])
def test_many_row_paths_shapes_bit_exact(ctx_mma, ctx_tc, kind, m, n, k):
    """More than eight activation rows go to the mma.sync GEMM (register accumulators) or,
    when forced or when the shape does not fit it, to the tcgen05 GEMM: ragged token counts,
    several launches of 256 tokens, ragged row tiles, large K."""
    ctx = ctx_tc if kind == "tc" else ctx_mma
    blocks = pkg.synth.bg128_weight(20261125, n + k + m, n, k)
    x = pkg.synth.activations(7, m + 1, m, k)
    x[m // 2, 128:256] = 0.0
    y, _ = run_gpu(ctx, blocks, n, k, x, sums=False, pad=4)
    y_ref = ol.matmul_w4(blocks, n, k, x)
    assert y.tobytes() == y_ref.tobytes()


@pytest.mark.parametrize("m,n,k", [(24, 72, 10368), (260, 40, 10368), (12, 264, 16384)])
def test_many_rows_beyond_the_tcgen05_kernels_k_limit(ctx, m, n, k):
    """K above 10240 (more than 80 groups) cannot go to the tcgen05 kernel: the mma.sync
    kernel takes it, resident or through its activation ring, 256 rows per launch."""
    blocks = pkg.synth.bg128_weight(20261125, n + k + m, n, k)
    x = pkg.synth.activations(7, m + 3, m, k)
    y, _ = run_gpu(ctx, blocks, n, k, x, sums=False)
    y_ref = ol.matmul_w4(blocks, n, k, x)
    assert y.tobytes() == y_ref.tobytes()


@pytest.mark.parametrize("kind", ["tc", "mma"])
@pytest.mark.parametrize("m,n,k", [(24, 264, 1280), (9, 40, 640), (256, 520, 2560),
                                   (300, 72, 512), (40, 72, 10368), (129, 2560, 1024),
                                   (128, 392, 640), (200, 6144, 256)])
def test_per32_rule_many_rows_bit_exact(ctx_mma, ctx_tc, kind, m, n, k):
    """The reference's M > 1 rule (one int8 scale per 32 values, kernels/matmul_w4.cpp:785-901)
    for more than eight rows, on both many-row kernels: tcgen05 with one tensor-memory
    accumulator per 32-k block (32 / 48 / 64 weight rows per CTA, one or several token blocks,
    ragged last tiles), and mma.sync with one tensor instruction, bias and scale per block
    (resident and ring mode, several launches of 256 rows)."""
    blocks = pkg.synth.bg128_weight(20261125, n + k + m + 1, n, k)
    x = pkg.synth.activations(7, m + 9, m, k)
    x[m // 3, 32:64] = 0.0  # an all-zero 32-block
    y, _ = run_gpu(ctx_tc if kind == "tc" else ctx_mma, blocks, n, k, x, rule=ol.ACT_G32,
                   sums=False, pad=4 if n % 16 else 0)
    y_ref = ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32)
    assert y.tobytes() == y_ref.tobytes()


@pytest.mark.parametrize("m,n,k", [(33, 8, 128), (128, 11832, 256), (300, 4100, 384),
                                   (130, 9472, 512), (1000, 4100, 640), (97, 7104, 1664),
                                   (160, 1184, 10240)])
def test_per32_tensor_core_tiles_bit_exact(ctx_tc, m, n, k):
    """The per-32 tcgen05 kernel in each of its tile widths (32, 48 and 64 columns), one and
    several rounds of CTAs, ragged tokens and weight rows, fewer groups than pipeline stages
    and the largest K, with codes at both ends of the range: its sums arrive as 16 D."""
    blocks = pkg.synth.bg128_weight(20261125, n + k + m + 2, n, k)
    x = pkg.synth.activations(7, m + 11, m, k)
    x[m // 2] = np.sign(x[m // 2])  # every code +-127: the largest sums
    y, _ = run_gpu(ctx_tc, blocks, n, k, x, rule=ol.ACT_G32, sums=False, pad=4 if n % 16 else 0)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32).tobytes()


def _tiny_products(exponent, m=70, n=40, k=512):
    """fp32 weight scales and activations whose scale products lie in 2^exponent times [1, 4)."""
    rng = np.random.default_rng(-exponent)
    q = rng.integers(-8, 8, (n, k)).astype(np.int8)
    ws = (rng.uniform(1, 2, (n, k // 128)) * 2.0 ** -60).astype(np.float32)
    x = rng.uniform(-1, 1, (m, k // 32, 32))
    x /= np.abs(x).max(axis=2, keepdims=True)
    x *= 127 * rng.uniform(1, 2, (m, k // 32, 1)) * 2.0 ** (exponent + 60)
    return ol.bg128_encode(q, ws), np.ascontiguousarray(x.reshape(m, k).astype(np.float32)), n, k


def test_per32_tensor_core_scales_near_the_smallest_normal(ctx_tc):
    """The per-32 tcgen05 kernel stages weight scales as w / 16 and sums as 16 D: the oracle's
    bits while every w * a / 16 is a normal number (2^-126 and up).  Below, the product loses
    bits, at most 2^-150 each: with |16 D| <= 16 * 32 * 8 * 127 that is 2^19 * 2^-150 per
    32-block, beside 2^15 * 2^-150 for the oracle's own product and fp32 rounding of the sum."""
    blocks, x, n, k = _tiny_products(-122)
    y, _ = run_gpu(ctx_tc, blocks, n, k, x, rule=ol.ACT_G32, sums=False)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32).tobytes()
    blocks, x, n, k = _tiny_products(-126)
    y, _ = run_gpu(ctx_tc, blocks, n, k, x, rule=ol.ACT_G32, sums=False)
    want = ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32).astype(np.float64)
    bound = (k // 32) * (2.0 ** 19 + 2.0 ** 15) * 2.0 ** -150 + \
        2 * (k // 32) * 2.0 ** -24 * (k // 32) * 2.0 ** 15 * 2.0 ** -124
    assert np.max(np.abs(y - want)) <= bound
    assert np.max(np.abs(want)) > 50 * bound  # the results are far above it


@pytest.mark.parametrize("tiles", [3, 5, 7, 9, 12, 14, 15, 16])
def test_per32_tensor_core_wide_tiles_bit_exact(ctx_tc, tiles):
    """One round of CTAs whose tiles are 32 to 128 columns wide (multiples of 16, whole and with
    a last one that is not full), 33 tokens: all warps of one lane quarter and one lane of the
    next have a token."""
    n, k, m = 148 * 8 * tiles - 8, 384, 33
    blocks = pkg.synth.bg128_weight(20261125, n + k + 3, n, k)
    x = pkg.synth.activations(7, tiles, m, k)
    y, _ = run_gpu(ctx_tc, blocks, n, k, x, rule=ol.ACT_G32, sums=False)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32).tobytes()


@pytest.mark.parametrize("rule", [ol.ACT_G32, ol.ACT_G128])
@pytest.mark.parametrize("m,n,k", [(9, 8, 128), (16, 24, 384), (17, 4100, 512), (24, 1000, 640),
                                   (25, 11848, 256), (32, 9728, 2560), (12, 72, 10368)])
def test_few_rows_bit_exact(ctx, m, n, k, rule):
    """9 to 32 rows: one and two column blocks per warp, a last block that is not full, a missing
    second tile of a pair, fewer groups than are in flight, one to five pairs per CTA, K beyond
    the tcgen05 kernels'."""
    blocks = pkg.synth.bg128_weight(20261125, n + k + m + 4, n, k)
    x = pkg.synth.activations(7, m + 13, m, k)
    x[m // 3, 32:64] = 0.0  # an all-zero 32-block
    y, _ = run_gpu(ctx, blocks, n, k, x, rule=rule, sums=False, pad=4 if n % 16 else 0)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=rule).tobytes()


def test_config2_prefill_m256_reference_rule(ctx):
    """M=256, K=2560, N=9728 (benchmark configuration 2, prefill) under the reference's rule
    for several rows (per 32 values), the kernel the library picks by itself: bit-exact
    against the oracle, and within 1e-2 relative L2 of the exact dequantised product."""
    n, k, m = 9728, 2560, 256
    blocks = pkg.synth.bg128_weight(20261125, 1, n, k)
    x = pkg.synth.activations(7, 256, m, k)
    y, _ = run_gpu(ctx, blocks, n, k, x, rule=ol.ACT_G32, sums=False)
    y_ref = ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32)
    assert y.tobytes() == y_ref.tobytes()
    rows = [0, 100, 255]
    exact = ol.matmul_w4(blocks, n, k, x[rows], rule=ol.ACT_F64)
    assert rel_l2(y[rows], exact) < 1e-2


def test_config2_prefill_m256(ctx):
    """M=256, K=2560, N=9728 (benchmark configuration 2, prefill): bit-exact against the
    row-by-row W4A8 oracle, and within 1e-2 relative L2 of the exact dequantised product
    (the W4A8-vs-W4A32 gap itself is ~6e-3 on these distributions)."""
    n, k, m = 9728, 2560, 256
    blocks = pkg.synth.bg128_weight(20261125, 1, n, k)
    x = pkg.synth.activations(7, 256, m, k)
    y, _ = run_gpu(ctx, blocks, n, k, x, sums=False)
    y_ref = ol.matmul_w4(blocks, n, k, x)
    assert y.tobytes() == y_ref.tobytes()
    rows = [0, 100, 255]
    exact = ol.matmul_w4(blocks, n, k, x[rows], rule=ol.ACT_F64)
    assert rel_l2(y[rows], exact) < 1e-2


def test_gemv_and_tensor_core_paths_agree(ctx):
    """The same rows through the dp4a GEMV (one at a time) and through the tensor-core
    kernel (all at once) give identical bits."""
    import torch
    n, k, m = 520, 1024, 24
    blocks = pkg.synth.bg128_weight(5, 5, n, k)
    x = pkg.synth.activations(7, 77, m, k)
    w = ctx.upload_weight(blocks, n, k)
    xd = torch.from_numpy(x).cuda()
    y_all = torch.zeros((m, n), device="cuda")
    y_one = torch.zeros((m, n), device="cuda")
    ctx.matmul(w, xd, y_all)
    for r in range(m):
        ctx.matmul(w, xd[r:r + 1], y_one[r:r + 1])
    ctx.sync()
    assert torch.equal(y_all, y_one)
    w.free()


@pytest.mark.parametrize("n,k,m", [(64, 128, 1), (1024, 512, 1), (9728, 2560, 1), (1024, 512, 2),
                                   (2048, 1024, 4), (9728, 2560, 5), (4096, 640, 8),
                                   (151936, 2560, 1), (151936, 2560, 3)])
def test_matmul_argmax_picks_the_oracle_token(ctx, n, k, m):
    """b2w4_matmul_argmax: the token of every row equals argmax_token over the oracle's
    logits (which the device logits match bit for bit), with and without the logits written,
    and again on a second call (the reduction cells are cleared by the launch itself)."""
    import torch
    blocks = pkg.synth.bg128_weight(41, 3, n, k)
    w = ctx.upload_weight(blocks, n, k)
    for call in range(2):
        x = pkg.synth.activations(90 + call, 1, m, k)
        xd = torch.from_numpy(x).cuda()
        ref = ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G128)
        want = [ol.argmax_token(ref[i]) for i in range(m)]
        tok = torch.full((m,), -1, dtype=torch.int32, device="cuda")
        y = torch.zeros((m, n), dtype=torch.float32, device="cuda")
        ctx.matmul_argmax(w, xd, tok, y)
        ctx.sync()
        assert tok.cpu().tolist() == want
        assert np.array_equal(y.cpu().numpy().view(np.uint32), ref.view(np.uint32))
        tok.fill_(-1)
        ctx.matmul_argmax(w, xd, tok)        # logits not written at all
        ctx.sync()
        assert tok.cpu().tolist() == want
    w.free()


@pytest.mark.parametrize("m", [1, 4])
def test_matmul_argmax_equal_logits_go_to_the_lowest_index(ctx, m):
    """Every 8-row tile of the weight is the same tile, so row r and rows r+8, r+16, ... give
    identical logits in different CTAs: the first of them must win."""
    import torch
    k, tiles = 512, 600
    one = pkg.synth.bg128_weight(42, 1, 8, k)
    blocks = np.tile(one, tiles)
    n = 8 * tiles
    w = ctx.upload_weight(blocks, n, k)
    x = pkg.synth.activations(95, 2, m, k)
    ref = ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G128)
    want = [ol.argmax_token(ref[i]) for i in range(m)]
    assert all(t < 8 for t in want)
    tok = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    ctx.matmul_argmax(w, torch.from_numpy(x).cuda(), tok)
    ctx.sync()
    assert tok.cpu().tolist() == want
    w.free()


def test_matmul_argmax_bad_arguments(ctx):
    import torch
    w = ctx.upload_weight(pkg.synth.bg128_weight(43, 1, 64, 128), 64, 128)
    tok = torch.zeros((9,), dtype=torch.int32, device="cuda")
    with pytest.raises(pkg.capi.B200W4Error):
        ctx.matmul_argmax(w, torch.zeros((9, 128), device="cuda"), tok)   # more than 8 rows
    with pytest.raises(pkg.capi.B200W4Error):
        ctx.matmul_argmax(w, torch.zeros((1, 128), device="cuda"), tok,
                          torch.zeros((1, 32), device="cuda"))           # logits row too short
    w.free()


@pytest.mark.parametrize("n,k,f32", [(8, 6144, False), (2560, 9728, False), (1003, 6272, True),
                                     (40, 12160, False), (2072, 6144, True)])
def test_long_rows_split_over_a_cluster(ctx, n, k, f32):
    """One row against long weight rows, whose groups a cluster shares: group counts that four
    divides and does not, ragged last tiles and clusters, fp32 scales, a fused activation; the
    oracle's bits."""
    blocks = pkg.synth.bg128_weight(20261125, n + k, n, k)
    if f32:  # scales that fp16 cannot hold
        blocks = np.array(blocks, copy=True)
        s = blocks.reshape(-1, 544)[:, :32].copy().view(np.float32)
        blocks.reshape(-1, 544)[:, :32] = (s * np.float32(1.0000001) + np.float32(1e-9) *
                                           (s != 0)).astype(np.float32).view(np.uint8)
    x = pkg.synth.activations(7, n, 1, k)
    x[0, 128:256] = 0.0  # a group of zeros
    y, _ = run_gpu(ctx, blocks, n, k, x, sums=False)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x).tobytes()


@pytest.mark.parametrize("rule", [ol.ACT_G32, ol.ACT_G128])
@pytest.mark.parametrize("m,pairs,k", [(16, 1, 768), (12, 2, 640), (13, 3, 384), (16, 4, 1152),
                                       (17, 1, 128), (24, 2, 896), (32, 1, 256), (25, 2, 2560),
                                       (8, 7, 1024), (9, 5, 512)])
def test_few_rows_with_few_pairs_per_multiprocessor(ctx, m, pairs, k, rule):
    """Two or four warps share the chain of a pair of tiles: 1 to 20 groups (whole stages of four
    and cut ones), the last pair with one tile, up to the largest number of chains per block (eight:
    16 rows of four pairs under the per-128 rule, 25 of two; seven of eight rows) and one past it."""
    n = 148 * 16 * pairs - 8
    blocks = pkg.synth.bg128_weight(20261125, n + k + m, n, k)
    x = pkg.synth.activations(7, m + 5, m, k)
    x[m // 2, :128] = 0.0
    y, _ = run_gpu(ctx, blocks, n, k, x, rule=rule, sums=False, pad=4)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=rule).tobytes()


BOTH, G32, G128 = (ol.ACT_G32, ol.ACT_G128), (ol.ACT_G32,), (ol.ACT_G128,)
PER_SM = 148 * 16  # weight rows that give every multiprocessor one pair of tiles


def _fp32_scales(blocks):
    """The same blocks with scales that fp16 cannot hold."""
    blocks = np.array(blocks, copy=True)
    s = blocks.reshape(-1, 544)[:, :32].copy().view(np.float32)
    blocks.reshape(-1, 544)[:, :32] = (s * np.float32(1.0000001) + np.float32(1e-9) *
                                       (s != 0)).astype(np.float32).view(np.uint8)
    return blocks


# streamed: the rules under which the call goes to the kernel of 9 to 32 rows (a quantiser's launch
# and the matmul's); else it is one launch of the kernel that quantises inside
@pytest.mark.parametrize("rule", BOTH)
@pytest.mark.parametrize("m,n,k,streamed,f32", [
    (2, 16392, 256, (), False), (3, 4104, 512, (), False), (8, 6152, 640, G32, False),
    (5, 1608, 384, (), False), (2, 1608, 6272, (), False), (2, 16392, 1024, G32, False),
    (4, PER_SM * 8 - 8, 640, (), False),
    (7, 1603, 6144, BOTH, False),             # one pair per multiprocessor, four warps a chain
    (3, 2568, 6272, BOTH, False), (7, 4104, 512, G32, False),       # two pairs
    (8, 6152, 2048, BOTH, False),             # three; per 32 a warp per pair, six stages
    (7, PER_SM * 5 - 8, 2176, BOTH, True), (8, PER_SM * 7 - 8, 1024, BOTH, False),  # two warps
    (2, PER_SM * 8 - 8, 1024, G32, False), (8, PER_SM * 8 - 8, 2048, BOTH, False),  # five stages
    (5, PER_SM * 12 - 8, 1024, BOTH, False),  # two blocks per multiprocessor, three stages
    (8, PER_SM * 12 - 3, 1152, BOTH, True)])
def test_two_to_eight_rows_on_the_streamed_kernel(ctx, m, n, k, streamed, f32, rule):
    """Row counts and weights on both sides of the line between the two kernels, and each form of
    the streamed one with a single column block: chains shared by four and by two warps, a warp per
    pair with six, five and three stages, fp16 and fp32 scales; the oracle's bits."""
    import torch
    blocks = pkg.synth.bg128_weight(20261125, n + k + m + 5, n, k)
    if f32:
        blocks = _fp32_scales(blocks)
    x = pkg.synth.activations(7, m + 17, m, k)
    pad = 4 if n % 16 else 0
    w = ctx.upload_weight(blocks, n, k)
    xd = torch.zeros((m, k + pad), device="cuda")
    xd[:, :k] = torch.from_numpy(x)
    yd = torch.full((m, n + pad), -7.0, device="cuda")
    assert _launches_of(ctx, lambda: ctx.matmul(w, xd, yd, rule=rule)) == (
        2 if rule in streamed else 1)
    ctx.sync()
    w.free()
    assert bool((yd[:, n:] == -7.0).all())
    assert yd[:, :n].cpu().numpy().tobytes() == ol.matmul_w4(blocks, n, k, x, rule=rule).tobytes()


# (rows, weight, rule) that the streamed kernel of gemm_rows.cu takes below nine rows
STREAMED = [(2, 9728, 6272, ol.ACT_G32), (4, 9728, 2560, ol.ACT_G32), (8, 9728, 2560, ol.ACT_G128)]


def _launches_of(ctx, call):
    before = ctx.launches
    call()
    return ctx.launches - before


@pytest.mark.parametrize("m,n,k,rule", STREAMED)
def test_few_rows_captured_hold_no_scratch(m, n, k, rule):
    """Two to eight rows as a context's very first matmul, inside a capture; then calls that need
    far more of the context's scratch; then the graph again, on other rows.  What a graph holds
    must be neither grown nor freed: the captured call is one launch that quantises inside."""
    import torch
    blocks = pkg.synth.bg128_weight(20261125, n + k + m, n, k)
    ctx = pkg.capi.Context(0)
    w = ctx.upload_weight(blocks, n, k)
    xs = [pkg.synth.activations(7, i, m, k) for i in (1, 2)]
    x, y = torch.from_numpy(xs[0]).cuda(), torch.zeros((m, n), device="cuda")
    torch.cuda.synchronize()
    side, other, g = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x2, y2 = x.clone(), torch.zeros_like(y)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        with torch.cuda.graph(g, stream=side):
            ctx.set_stream(side.cuda_stream)
            assert _launches_of(ctx, lambda: ctx.matmul(w, x, y, rule=rule)) == 1
            # on another stream while the capture is open: not captured, and does not spoil it
            ctx.set_stream(other.cuda_stream)
            assert _launches_of(ctx, lambda: ctx.matmul(w, x2, y2, rule=rule)) == 2
    ctx.sync()
    want = ol.matmul_w4(blocks, n, k, xs[0], rule=rule)
    assert y2.cpu().numpy().tobytes() == want.tobytes() and not y.any()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    for rows in (9, 40, 700):
        big = torch.randn((rows, k), device="cuda")
        for r in (ol.ACT_G32, ol.ACT_G128):
            ctx.matmul(w, big, torch.zeros((rows, n), device="cuda"), rule=r)
    ctx.sync()
    for host in xs:
        x.copy_(torch.from_numpy(host))
        g.replay()
        torch.cuda.synchronize()
        want = ol.matmul_w4(blocks, n, k, host, rule=rule)
        assert y.cpu().numpy().tobytes() == want.tobytes()
    w.free()
    ctx.close()


@pytest.mark.parametrize("m,n,k,rule", STREAMED)
def test_few_rows_on_several_streams(m, n, k, rule):
    """One context used on 18 streams in turn, nothing ordered between them: every call's rows are
    its own.  Sixteen streams have buffers (a quantiser's launch and the matmul's), the others take
    the kernel that quantises inside."""
    import torch
    blocks = pkg.synth.bg128_weight(20261125, n + k + m, n, k)
    ctx = pkg.capi.Context(0)
    w = ctx.upload_weight(blocks, n, k)
    streams = [torch.cuda.Stream() for _ in range(18)]
    xs = torch.randn((len(streams), m, k), device="cuda") * torch.arange(
        1, len(streams) + 1, device="cuda").view(-1, 1, 1)
    want, ys = (torch.zeros((len(streams), m, n), device="cuda") for _ in range(2))
    assert len({s.cuda_stream for s in streams}) == len(streams)
    ctx.set_stream(0)
    for i in range(len(streams)):  # one row after another
        for r in range(m):
            ctx.matmul(w, xs[i, r:r + 1], want[i, r:r + 1], rule=rule)
    ctx.sync()
    torch.cuda.synchronize()
    for _ in range(5):
        ys.zero_()
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            ctx.set_stream(s.cuda_stream)
            assert _launches_of(ctx, lambda: ctx.matmul(w, xs[i], ys[i], rule=rule)) == (
                2 if i < 16 else 1)
        torch.cuda.synchronize()
        assert torch.equal(ys, want)
    ctx.set_stream(0)
    w.free()
    ctx.close()


@pytest.mark.parametrize("m,rule,longest", [(1, ol.ACT_G128, 39552), (1, ol.ACT_G32, 30464),
                                            (2, ol.ACT_G128, 33280), (4, ol.ACT_G32, 17152),
                                            (8, ol.ACT_G128, 15360), (8, ol.ACT_G32, 10112),
                                            (12, ol.ACT_G128, 26368), (32, ol.ACT_G32, 25216)])
def test_longest_rows(ctx, m, rule, longest):
    """The longest row of a call does not depend on the number of weight rows, which decides
    between kernels with and without a limit: the last length that is taken (a row of the result
    against the oracle) and the first that is refused, before anything is written."""
    import torch
    for n in (8, 2568):
        for k in (longest, longest + 128):
            w = ctx.upload_weight(pkg.synth.bg128_weight(3, n + k, n, k), n, k)
            x = pkg.synth.activations(7, m, m, k)
            xd, y = torch.from_numpy(x).cuda(), torch.full((m, n), -1.0, device="cuda")
            res, one = torch.ones((m, k), device="cuda"), torch.ones(k, device="cuda")
            if k == longest:
                ctx.matmul(w, xd, y, rule=rule)
                ctx.sync()
                rows = pkg.synth.bg128_weight(3, n + k, n, k)[:k // 128 * 544]  # the first tile
                want = ol.matmul_w4(rows, 8, k, x, rule=rule)
                assert y[:, :8].cpu().numpy().tobytes() == want.tobytes()
            else:
                for call in (lambda: ctx.matmul(w, xd, y, rule=rule),
                             lambda: ctx.matmul_norm(w, res, xd, one, 1e-6, y, rule=rule)):
                    with pytest.raises(pkg.capi.B200W4Error, match="K="):
                        call()
                assert bool((y == -1).all()) and bool((res == 1).all())
            w.free()


@pytest.mark.parametrize("n,k,f32", [(70001, 128, False), (99993, 384, True), (66305, 1152, False),
                                     (40961, 2560, False), (30011, 4224, True)])
def test_many_rows_on_persistent_blocks(ctx, n, k, f32):
    """One row against weights of many rows, whose blocks take chunks of tiles through a ring: one
    group and counts that four does not divide, chunks of 3 to 16 tiles, ragged last chunks and
    tiles, fp32 scales, a row that is not 16-byte aligned, a fused activation, the greedy token with
    and without the logits; the oracle's bits."""
    import torch
    blocks = pkg.synth.bg128_weight(20261125, n + k, n, k)
    if f32:  # scales that fp16 cannot hold
        blocks = np.array(blocks, copy=True)
        s = blocks.reshape(-1, 544)[:, :32].copy().view(np.float32)
        blocks.reshape(-1, 544)[:, :32] = (s * np.float32(1.0000001) + np.float32(1e-9) *
                                           (s != 0)).astype(np.float32).view(np.uint8)
    x = pkg.synth.activations(91, n, 1, k)
    ref = ol.matmul_w4(blocks, n, k, x)
    w = ctx.upload_weight(blocks, n, k)
    at = torch.zeros(k + 4, device="cuda")
    for off in (0, 1):
        xd = at[off:off + k].view(1, k)
        xd.copy_(torch.from_numpy(x))
        y, logits = (torch.zeros((1, n), device="cuda") for _ in range(2))
        tok = torch.full((2,), -1, dtype=torch.int32, device="cuda")
        ctx.matmul(w, xd, y)
        ctx.matmul_argmax(w, xd, tok[:1], logits)
        ctx.matmul_argmax(w, xd, tok[1:])
        ctx.sync()
        assert y.cpu().numpy().tobytes() == ref.tobytes()
        assert logits.cpu().numpy().tobytes() == ref.tobytes()
        assert tok.tolist() == [ol.argmax_token(ref[0])] * 2
    act, begin, length = 3, n // 2, 1000
    ctx.matmul(w, torch.from_numpy(x).cuda(), y, act=act, act_begin=begin, act_len=length)
    ctx.sync()
    want = ol.apply_activation(ref.copy(), act, begin, length)
    assert y.cpu().numpy().tobytes() == want.tobytes()
    w.free()


@pytest.mark.parametrize("n,k,f32,tiles", [(21801, 4096, False, 2), (23001, 3584, True, 2),
                                           (16501, 5120, True, 1), (11101, 7680, False, 1)])
def test_persistent_blocks_of_few_tiles(ctx, n, k, f32, tiles):
    """Chunks of two tiles and of one, just above their line, plain and with the greedy token: the
    oracle's bits."""
    import ctypes as C
    import torch
    blocks = pkg.synth.bg128_weight(20261125, n + k, n, k)
    if f32:  # scales that fp16 cannot hold
        blocks = np.array(blocks, copy=True)
        s = blocks.reshape(-1, 544)[:, :32].copy().view(np.float32)
        blocks.reshape(-1, 544)[:, :32] = (s * np.float32(1.0000001) + np.float32(1e-9) *
                                           (s != 0)).astype(np.float32).view(np.uint8)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:  # four (up to 4096 values a row), three or two tiles in a block of the other kernel
        per = 4 if k <= 4096 else 3 if k <= 6144 else 2
        plan = C.CDLL(pkg.capi.LIB_PATH).b2w4_gemv_stream_plan
        assert plan(k // 128, not f32, -(-(-(-n // 8)) // per), sms) == tiles
    x = pkg.synth.activations(91, n, 1, k)
    ref = ol.matmul_w4(blocks, n, k, x)
    w = ctx.upload_weight(blocks, n, k)
    xd = torch.from_numpy(x).cuda()
    y, logits = (torch.zeros((1, n), device="cuda") for _ in range(2))
    tok = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    ctx.matmul(w, xd, y)
    ctx.matmul_argmax(w, xd, tok[:1], logits)
    ctx.matmul_argmax(w, xd, tok[1:])
    ctx.sync()
    assert y.cpu().numpy().tobytes() == ref.tobytes()
    assert logits.cpu().numpy().tobytes() == ref.tobytes()
    assert tok.tolist() == [ol.argmax_token(ref[0])] * 2
    w.free()


@pytest.mark.parametrize("m,n,k", [(900, 1068, 896), (500, 1900, 1152), (900, 1224, 384),
                                   (1000, 1380, 1024), (500, 2500, 1408)])
def test_per32_tensor_core_tiles_of_64_and_80_columns(ctx_tc, m, n, k):
    """The two tile widths between those of test_per32_tensor_core_tiles_bit_exact that take two
    groups a turn, with odd and even numbers of groups, fewer and more than pipeline stages."""
    blocks = pkg.synth.bg128_weight(20261125, n + k + m + 2, n, k)
    x = pkg.synth.activations(7, m + 11, m, k)
    x[m // 2] = np.sign(x[m // 2])  # every code +-127: the largest sums
    y, _ = run_gpu(ctx_tc, blocks, n, k, x, rule=ol.ACT_G32, sums=False, pad=4 if n % 16 else 0)
    assert y.tobytes() == ol.matmul_w4(blocks, n, k, x, rule=ol.ACT_G32).tobytes()


@pytest.mark.parametrize("n,k,split", [(8704, 6144, True), (9472, 6144, True), (9480, 6144, False),
                                       (20000, 6144, False), (2560, 9728, True)])
def test_split_rows_in_one_wave_of_clusters(ctx, n, k, split):
    """Long rows are split over clusters of four where all of them run at once (two blocks per
    multiprocessor); the oracle's bits on either side of the line."""
    import torch
    driver = pytest.importorskip("cuda.bindings.driver")
    blocks = pkg.synth.bg128_weight(20261125, n + k, n, k)
    x = pkg.synth.activations(91, n, 1, k)
    w = ctx.upload_weight(blocks, n, k)
    xd, y = torch.from_numpy(x).cuda(), torch.zeros((1, n), device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    try:
        with torch.cuda.graph(graph):
            ctx.set_stream(torch.cuda.current_stream().cuda_stream)
            ctx.matmul(w, xd, y)
    finally:
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    raw = driver.CUgraph(init_value=graph.raw_cuda_graph())
    count = driver.cuGraphGetNodes(raw)[-1]
    assert count == 1
    node = driver.cuGraphGetNodes(raw, count)[1][0]
    grid = driver.cuGraphKernelNodeGetParams(node)[1].gridDimX
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        per = 3 if k == 6144 else 2  # tiles in a block of the kernel that does not split
        other = 2 * sms if n == 20000 else -(-(n // 8) // per)  # persistent blocks
        assert grid % 4 == 0 and grid <= 2 * sms if split else grid == other
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    assert y.cpu().numpy().tobytes() == ol.matmul_w4(blocks, n, k, x).tobytes()
    del graph
    w.free()
