"""Which one-row calls go to the persistent kernel (gemv_stream_chunk in csrc/gemv_dp4a.cu), checked
over the sizes that the entry points take: no device needed."""
import ctypes as C

import pytest

from __graft_entry__ import load_package

pkg = load_package()
SMS = 148


def chunk(groups, fp16, ctas):
    return C.CDLL(pkg.capi.LIB_PATH).b2w4_gemv_stream_plan(groups, fp16, ctas, SMS)


@pytest.mark.parametrize("fp16", [0, 1])
def test_persistent_kernel_where_it_is_the_faster_one(fp16):
    """Chunks of three tiles and more from three and a half blocks per multiprocessor of the other
    kernel on, smaller ones from four and a half, chunks of one tile only where its groups fill
    five eighths of a round; a chunk fits half a multiprocessor's shared memory three times; and
    more blocks never turn a call back."""
    for groups in range(1, 310):
        sizes = {c: chunk(groups, fp16, c) for c in (1, 518 - 1, 518, 666 - 1, 666, 5000, 10 ** 6)}
        most = sizes[10 ** 6]
        assert sizes[1] == sizes[517] == 0
        assert sizes[518] == sizes[665] == (most if most >= 3 else 0)
        assert sizes[666] == sizes[5000] == most
        if most:
            assert 3 * most * groups * (512 + (16 if fp16 else 32)) <= 112 * 1024
        if most == 1:
            assert groups >= 40
        if groups <= 20:
            assert most >= 3
    for groups, tiles in ((20, 3), (22, 2), (28, 2), (34, 0), (36, 0), (38, 0), (40, 1), (60, 1)):
        assert chunk(groups, fp16, 10 ** 6) == tiles
    assert chunk(32, fp16, 10 ** 6) == (2 if fp16 else 0)
