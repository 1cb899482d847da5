"""The work this library is used for, as cases that can be timed and compared.

Every case goes through the public entry points that a program calls: b2w4_matmul on the
weights of a stack of layers, lists of decode GEMVs (Chain), the routed mixture-of-experts
operator, and whole decoders (DenseDecoder: prefill of a prompt, one replayed decode step).
Shapes are those of the benchmark configurations (a 4B dense decoder's projections, a
30B-A3B mixture of experts' layer) and generic ones around them; values are synthetic with the
distributions of the benchmark: uniform int4 codes, group scales |N(0, 0.02)| rounded to fp16,
N(0, 1) activations.

listed() / draw(rng) -> cases, prepare(case, seed) -> state, run(state) -> outputs,
work(case) -> the bytes and operations one pass cannot do without, tolerance(case).
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
capi = pkg.capi

BLOCK_BYTES = 544  # canonical BG128 block: 8 fp32 row scales, 8 x 128 nibbles


# --------------------------------------------------------------------------------- cases

def listed():
    dec = dict(layers=8, hidden=2560, heads=32, kv_heads=8, head_dim=128, inter=9728,
               vocab=151936)
    moe = dict(experts=128, top_k=8, hidden=2048, inter=768)
    return [
        # the smallest call: one row through one small projection, where the call itself counts
        dict(name="gemv_call", kind="matmul", m=1, n=1024, k=1024, copies=1, rule=128,
             act=0, fp32_scales=False, head=0),
        # decode without the list kernel: the same projection of sixteen layers, one call each
        # (206 MB, so that every weight comes from HBM as in a decode step), and the lm_head
        # with the greedy token picked on the device
        dict(name="gemv_stack", kind="matmul", m=1, n=9728, k=2560, copies=16, rule=128,
             act=0, fp32_scales=False, head=151936),
        # batched decode, sixteen sequences, the reference's rule for several rows
        dict(name="rows_16", kind="matmul", m=16, n=9728, k=2560, copies=16, rule=32,
             act=0, fp32_scales=False, head=0),
        # a long ragged prompt through a down projection with a fused activation: rows and
        # columns that fill no tile, scales that fp16 cannot hold
        dict(name="rows_1000", kind="matmul", m=1000, n=4100, k=9728, copies=3, rule=32,
             act=1, fp32_scales=True, head=0),
        # a list of GEMVs on one vector in one launch (the benchmark's headline workload)
        dict(name="list_shared", kind="list", shared=True, ops=32, n=9728, k=2560),
        # a token's matmuls as one list, each consuming what an earlier one produced
        dict(name="list_walk", kind="list", shared=False, ops=16, hidden=2560, q_dim=4096,
             kv_dim=1024, inter=9728),
        # one decode step of a dense decoder behind a short and behind a long context
        dict(name="decode_300", kind="decode", past=300, capacity=512, **dec),
        dict(name="decode_6000", kind="decode", past=6000, capacity=7000, **dec),
        # a prompt of the benchmark's length and one of several pages
        dict(name="prompt_256", kind="prompt", tokens=256, capacity=512, **dec),
        dict(name="prompt_1500", kind="prompt", tokens=1500, capacity=2048, **dec),
        # one layer's routed experts: a decode token, the benchmark's prompt
        dict(name="moe_token", kind="moe", tokens=1, **moe),
        dict(name="moe_prompt", kind="moe", tokens=256, **moe),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["matmul"] * 4 + ["list"] + ["decode"] * 2 + ["prompt"] * 2 + ["moe"] * 2)
    if kind == "matmul":
        m = 1 if rng.random() < 0.25 else _log_int(rng, 2, 1000)
        n, k = _log_int(rng, 500, 20000), _log_int(rng, 512, 9728, 128)
        copies = max(1, min(16, (160 << 20) // (n * k // 2)))
        head = _log_int(rng, 5000, 151936) if m <= 8 and k <= 2560 and rng.random() < 0.5 else 0
        return dict(kind=kind, m=m, n=n, k=k, copies=copies,
                    rule=128 if m == 1 else rng.choice([32, 32, 128]),
                    act=rng.choice([0, 0, 1]), fp32_scales=rng.random() < 0.25, head=head)
    if kind == "list":
        if rng.random() < 0.5:
            return dict(kind=kind, shared=False, ops=4 * rng.randint(1, 4),
                        hidden=_log_int(rng, 1024, 2560, 128), q_dim=_log_int(rng, 1024, 4096, 128),
                        kv_dim=128 * rng.randint(1, 8), inter=_log_int(rng, 2048, 9728, 128))
        n, k = _log_int(rng, 1000, 20000), _log_int(rng, 1024, 9728, 128)
        return dict(kind=kind, shared=True, n=n, k=k,
                    ops=max(2, min(40, (400 << 20) // (n * k // 2))))
    if kind == "moe":
        top_k = rng.randint(2, 8)
        return dict(kind=kind, tokens=_log_int(rng, 1, 256), experts=8 * rng.randint(2, 16),
                    top_k=top_k, hidden=_log_int(rng, 1024, 4096, 128),
                    inter=128 * rng.randint(3, 12))
    head_dim = rng.choice([64, 128, 128])
    kv_heads = rng.choice([2, 4, 8])
    heads = kv_heads * rng.choice([2, 4]) * (2 if head_dim == 64 else 1)
    cfg = dict(layers=rng.randint(2, 8), hidden=_log_int(rng, 1024, 2560, 128), heads=heads,
               kv_heads=kv_heads, head_dim=head_dim, inter=_log_int(rng, 2048, 9728, 128),
               vocab=_log_int(rng, 20000, 151936))
    if kind == "decode":
        past = _log_int(rng, 10, 6000)
        return dict(kind=kind, past=past, capacity=past + rng.randint(1, 2048), **cfg)
    tokens = _log_int(rng, 2, 1500)
    return dict(kind=kind, tokens=tokens, capacity=tokens + rng.randint(1, 512), **cfg)


# -------------------------------------------------------------------------------- inputs

_context = None


def _ctx():
    """One context per GPU, as a program keeps it."""
    global _context
    if _context is None:
        _context = capi.Context(0)
    _context.set_stream(torch.cuda.current_stream().cuda_stream)
    return _context


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _blocks(g, n, k, fp32_scales=False):
    """Canonical BG128 blocks of an [n, k] weight in device memory.  Rows past n in the last
    8-row tile have scale 0 and zero codes, as the packers write them."""
    tiles, groups = (n + 7) // 8, k // 128
    b = torch.empty((tiles, groups, BLOCK_BYTES), dtype=torch.uint8, device="cuda")
    q = torch.randint(0, 256, (tiles, groups, 512), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.randn((tiles, groups, 8), device="cuda", generator=g).abs_().mul_(0.02)
    if not fp32_scales:
        s = s.half().float()
    if n % 8:
        s[-1, :, n % 8:] = 0.0
        q.view(tiles, groups, 4, 8, 16)[-1, :, :, n % 8:] = 0
    b[:, :, 32:] = q
    b[:, :, :32] = s.view(torch.uint8)
    return b.view(-1)


def _weight(ctx, g, n, k, fp32_scales=False):
    return ctx.weight_from_device(_blocks(g, n, k, fp32_scales), n, k)


class State:
    """What a program holds before the call; gives the device memory back when dropped."""

    def __init__(self, call, frees):
        self.call, self.frees = call, frees

    def __del__(self):
        for f in self.frees:
            f()
        self.frees = []


def _prepare_matmul(case, g):
    ctx = _ctx()
    m, n, k = case["m"], case["n"], case["k"]
    ws = [_weight(ctx, g, n, k, case["fp32_scales"]) for _ in range(case["copies"])]
    x = torch.randn((m, k), device="cuda", generator=g).half().float()
    ys = [torch.empty((m, n), device="cuda") for _ in ws]
    rule, act = case["rule"], case["act"]
    head = tokens = None
    if case["head"]:
        head = _weight(ctx, g, case["head"], k)
        tokens = torch.empty((m,), dtype=torch.int32, device="cuda")

    def call():
        for w, y in zip(ws, ys):
            ctx.matmul(w, x, y, rule=rule, act=act)
        if head is None:
            return ys
        ctx.matmul_argmax(head, x, tokens)
        return ys + [tokens]
    return State(call, [w.free for w in ws + ([head] if head else [])])


def _list_shapes(case):
    """(rows, columns) of every op: one projection many times, or a decoder's four in turn."""
    if case["shared"]:
        return [(case["n"], case["k"])] * case["ops"]
    h, q, i = case["hidden"], case["q_dim"], case["inter"]
    layer = [(q + 2 * case["kv_dim"], h), (h, q), (2 * i, h), (h, i)]
    return [layer[j % 4] for j in range(case["ops"])]


def _prepare_list(case, g):
    ctx = _ctx()
    shapes = _list_shapes(case)
    ws = [_weight(ctx, g, n, k) for n, k in shapes]
    x = torch.randn((shapes[0][1],), device="cuda", generator=g).half().float()
    ys = [torch.empty((n,), device="cuda") for n, _ in shapes]
    ops = [dict(w=w, y=y, x=x) if case["shared"] or i == 0 else dict(w=w, y=y, x_from=i - 1)
           for i, (w, y) in enumerate(zip(ws, ys))]
    chain = capi.Chain(ctx, ops)

    def call():
        chain.run()
        return ys
    return State(call, [chain.free] + [w.free for w in ws])


def _prepare_moe(case, g):
    ctx = _ctx()
    e, h, i = case["experts"], case["hidden"], case["inter"]
    gate_up, down = _weight(ctx, g, e * 2 * i, h), _weight(ctx, g, e * h, i)
    router = torch.randn((e, h), device="cuda", generator=g).mul_(0.02).half()
    x = torch.randn((case["tokens"], h), device="cuda", generator=g)
    out = torch.empty_like(x)

    def call():
        ctx.moe_forward(x, router, case["top_k"], i, gate_up, down, out)
        return out
    return State(call, [gate_up.free, down.free])


def _decoder(case, g):
    """A decoder on host weights as a package gives them (made on the GPU, where it is quick)."""
    cfg = pkg.decoder.DecoderConfig(case["layers"], case["hidden"], case["heads"],
                                    case["kv_heads"], case["head_dim"], case["inter"],
                                    case["vocab"])
    shapes = {"qkv": (cfg.q_dim + 2 * cfg.kv_dim, cfg.hidden), "o": (cfg.hidden, cfg.q_dim),
              "gate_up": (2 * cfg.intermediate, cfg.hidden),
              "down": (cfg.hidden, cfg.intermediate)}

    def norm(n):
        return torch.randn(n, device="cuda", generator=g).mul_(0.05).add_(1.0).cpu().numpy()

    def layer():
        w = {name: _blocks(g, n, k).cpu().numpy() for name, (n, k) in shapes.items()}
        w.update(ln1=norm(cfg.hidden), ln2=norm(cfg.hidden), q_norm=norm(cfg.head_dim),
                 k_norm=norm(cfg.head_dim))
        return w

    embed = torch.randn((cfg.vocab, cfg.hidden), device="cuda", dtype=torch.float16, generator=g)
    weights = {"shapes": shapes, "layers": (layer() for _ in range(cfg.layers)),
               "final_norm": norm(cfg.hidden), "embed": embed.mul_(0.02).cpu().numpy(),
               "lm_head": _blocks(g, cfg.vocab, cfg.hidden).cpu().numpy()}
    del embed
    return pkg.decoder.DenseDecoder(_ctx(), cfg, weights, case["capacity"])


def _decoder_outputs(dec, rows, past):
    """What a pass leaves behind: the final normalised hidden rows (the lm_head's input) and
    the cache rows it wrote.  The token is not among them: which of 150,000 flat logits is the
    largest can change as soon as they move by a part in a thousand (the tokens of
    matmul_argmax on given rows, which are exact, are compared in the matmul cases)."""
    out = [dec._b("h", rows, dec.cfg.hidden)]
    for layer in dec.layers:
        out += [layer["k_cache"][:, past:past + rows], layer["v_cache"][:, past:past + rows]]
    return out


def _prepare_decode(case, g):
    dec = _decoder(case, g)
    past = case["past"]
    for layer in dec.layers:  # the context: normalised keys, values of the projection's size
        layer["k_cache"][:, :past].normal_(generator=g)
        layer["v_cache"][:, :past].normal_(0.0, 4.0, generator=g)
    token = torch.randint(0, case["vocab"], (1,), dtype=torch.int32, device="cuda", generator=g)
    dec.past = past
    dec.capture_decode_step()
    outputs = _decoder_outputs(dec, 1, past)

    def call():
        dec.token.copy_(token)   # the token that goes in, and where
        dec.past_dev.fill_(past)
        dec.replay_decode_step()
        return outputs
    return State(call, [dec.free])


def _prepare_prompt(case, g):
    dec = _decoder(case, g)
    ids = torch.randint(0, case["vocab"], (case["tokens"],), device="cuda", generator=g)
    ids = ids.cpu().numpy().astype(np.int32)

    outputs = _decoder_outputs(dec, case["tokens"], 0)

    def call():
        dec.reset()
        dec.prefill(ids)
        return outputs
    return State(call, [dec.free])


def prepare(case, seed):
    make = {"matmul": _prepare_matmul, "list": _prepare_list, "moe": _prepare_moe,
            "decode": _prepare_decode, "prompt": _prepare_prompt}[case["kind"]]
    state = make(case, _gen(seed))
    torch.cuda.synchronize()
    return state


def run(state):
    return state.call()


# ------------------------------------------------------------------------- work, tolerance

def _weight_bytes(n, k, fp32_scales=False):
    return n * k // 2 + n * (k // 128) * (4 if fp32_scales else 2)


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        m, n, k, c = case["m"], case["n"], case["k"], case["copies"]
        return {"bytes": c * (_weight_bytes(n, k, case["fp32_scales"]) + 4 * m * n) + 4 * m * k +
                _weight_bytes(case["head"], k),
                "flops": 2 * m * k * (c * n + case["head"])}
    if kind == "list":
        shapes = _list_shapes(case)
        return {"bytes": sum(_weight_bytes(n, k) + 4 * n for n, k in shapes) + 4 * shapes[0][1],
                "flops": sum(2 * n * k for n, k in shapes)}
    if kind == "moe":
        t, e, h, i = case["tokens"], case["experts"], case["hidden"], case["inter"]
        used = e * (1.0 - (1.0 - case["top_k"] / e) ** t)  # experts that get a route
        return {"bytes": int(used * (_weight_bytes(2 * i, h) + _weight_bytes(h, i))) +
                2 * e * h + 8 * t * h,
                "flops": 2 * t * e * h + 6 * t * case["top_k"] * h * i}
    q, kv = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    h, i, layers = case["hidden"], case["inter"], case["layers"]
    t, past = (1, case["past"]) if kind == "decode" else (case["tokens"], 0)
    shapes = [(q + 2 * kv, h), (h, q), (2 * i, h), (h, i)]
    keys = t * past + t * (t + 1) // 2  # visible (query, key) pairs of a head
    return {"bytes": layers * (sum(_weight_bytes(n, k) for n, k in shapes) +
                               8 * kv * (past + t)) + _weight_bytes(case["vocab"], h) + 6 * t * h,
            "flops": layers * (sum(2 * t * n * k for n, k in shapes) +
                               4 * keys * q) + 2 * case["vocab"] * h}


def tolerance(case):
    # fp32 sums of the same int32 group sums and scales
    if case["kind"] in ("matmul", "moe") or case.get("shared"):
        return {"rel": 1e-5, "max": 1e-3}
    # results that went through several int8 quantisations: a last bit of an fp32 sum that
    # falls on the other side of a rounding boundary moves a code by one in 127
    return {"rel": 2e-2, "max": 0.8}
