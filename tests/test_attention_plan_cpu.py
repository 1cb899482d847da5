"""Which attention kernel a call takes (attn_plan in csrc/decoder_ops.cu), checked over the
sizes the entry point accepts: no device needed."""
import ctypes as C
import itertools

import pytest

from __graft_entry__ import load_package

pkg = load_package()
ROW, PLAIN, SPLIT, TILE = range(4)
SMS = 148


def plan(tokens, heads, kv_heads, dim, past=0, capacity=None, aligned=1, row=0, cluster=16):
    lib = C.CDLL(pkg.capi.LIB_PATH)
    out = (C.c_int * 4)()
    form = lib.b2w4_attention_plan(tokens, heads, kv_heads, dim, past,
                                   past + tokens if capacity is None else capacity, aligned, row,
                                   cluster, SMS, out)
    return form, dict(zip(("rows", "ctas", "one_range", "alone"), out))


HEADS = [(32, 8), (4, 2), (8, 8), (16, 4), (2, 1), (71, 1), (64, 2), (65, 1), (20, 20)]


@pytest.mark.parametrize("heads,kv_heads", HEADS)
def test_few_tokens(heads, kv_heads):
    """One to seven tokens on aligned rows of 64, 128 or 256 features: few visible keys stay
    with one block, more are split over a cluster whose blocks are all resident together (two to
    four per multiprocessor, by the kernel's registers) or as small as clusters get; other rows
    take the one-row kernel."""
    for tokens, dim, capacity in itertools.product(range(1, 8), (64, 128, 256),
                                                   (8, 300, 767, 768, 47000)):
        form, p = plan(tokens, heads, kv_heads, dim, capacity=capacity)
        assert form == SPLIT
        assert 96 <= p["one_range"] <= 4096 and p["ctas"] in (4, 8, 16)
        hr = (min(2, heads // kv_heads) if dim == 256 else
              4 if heads // kv_heads >= 3 else heads // kv_heads)
        groups = tokens * kv_heads * -(-(heads // kv_heads) // hr)
        resident = 4 if dim * hr <= 128 else 3 if dim * hr <= 256 else 2
        assert p["ctas"] == 4 or p["ctas"] * groups <= resident * SMS
        assert capacity >= 768 or p["ctas"] < 16
        # shared memory: the range's scores, the warps' sums and the small arrays
        for keys in {capacity, min(capacity, p["one_range"])}:
            n = max(-(-keys // p["ctas"]), min(keys, p["one_range"]))
            assert 4 * (n * hr + 9 * hr * dim + 1024) <= 227 * 1024
        assert plan(tokens, heads, kv_heads, dim, capacity=capacity, aligned=0)[0] == ROW
        assert plan(tokens, heads, kv_heads, dim, capacity=capacity, row=1)[0] == PLAIN
    for dim in (20, 32, 80, 96, 192):
        assert plan(3, heads, kv_heads, dim)[0] == ROW
        assert plan(300, heads, kv_heads, dim)[0] == ROW


def test_smaller_clusters():
    """A device or a switch that allows smaller clusters only."""
    for cluster in range(17):
        form, p = plan(1, 32, 8, 128, capacity=4096, cluster=cluster)
        assert form == SPLIT and p["ctas"] <= cluster
        assert p["ctas"] & (p["ctas"] - 1) == 0  # divides a block's share of the features
        assert p["one_range"] == 96


@pytest.mark.parametrize("heads,kv_heads", HEADS[:5] + HEADS[6:7] + HEADS[8:])
def test_runs_behind_a_context(heads, kv_heads):
    """Eight or more tokens on a cache of 384 rows or more: never tiles that leave most of the
    chip idle while they walk the keys one block after the other."""
    for tokens, dim, past in itertools.product((8, 9, 16, 33, 64, 100, 256, 600, 1400),
                                               (64, 128, 256), (0, 100, 1000, 6000, 40000)):
        capacity = max(384, past + tokens)
        form, p = plan(tokens, heads, kv_heads, dim, past, capacity)
        hr = (min(2, heads // kv_heads) if dim == 256 else
              4 if heads // kv_heads >= 3 else heads // kv_heads)
        groups = tokens * kv_heads * -(-(heads // kv_heads) // hr)
        assert form == (SPLIT if groups <= 10 * SMS else TILE)
        if form == TILE:
            rep = heads // kv_heads
            tiles = -(-tokens // (p["rows"] // rep)) * kv_heads
            assert p["rows"] in (32, 64) and rep <= p["rows"]
            assert tiles >= SMS // 4
            assert p["alone"] or tiles > SMS
        # a cache of 384 rows: the same form wherever the position is
        assert plan(tokens, heads, kv_heads, dim, 0, capacity)[0] == form
        if tokens < 300:
            assert plan(tokens, heads, kv_heads, dim, 0, 383)[0] == TILE
    assert plan(40, 71, 1, 128)[0] == ROW  # more query heads per kv head than a tile has rows
    assert plan(40, 64, 1, 128) == (TILE, dict(rows=64, ctas=0, one_range=0, alone=1))


def test_unaligned_runs():
    """Rows that are not 16-byte aligned: tiles too, unless one block per (token, head) is few
    blocks."""
    for tokens, (heads, kv_heads) in itertools.product((8, 23, 24, 100, 600), HEADS):
        for capacity in (tokens, 5000):
            form = plan(tokens, heads, kv_heads, 128, 0, capacity, aligned=0)[0]
            assert form == (ROW if heads // kv_heads > 64 or tokens * heads <= 5 * SMS else TILE)
