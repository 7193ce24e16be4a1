"""CPU: the way a packed decode takes (csrc/tq_decode_mma.cu), asked of the library's own rules."""
from __future__ import annotations

import ctypes

import pytest

from anna_b200 import _lib

CUDA_CORES, ONE_LAUNCH, EVEN_SHARES, CHUNKS = range(4)


def schedule(*, q=0x1000, strides=None, batch=4, heads=32, kv_heads=8, dim=128, blocks=256, page=16, window=128, group=32,
             dtype=_lib.DTYPE_BF16, one_launch_ctas=444, share_ctas=592):
    """(way, tokens of a chunk)"""
    sb, sh = strides or (heads * dim, dim)
    way, tokens = ctypes.c_int(-1), ctypes.c_int(-1)
    _lib.check(_lib.lib().anna_kv_selftest_tq_schedule(q, sb, sh, batch, heads, kv_heads, dim, blocks, page, window, group, dtype,
                                                       one_launch_ctas, share_ctas, ctypes.byref(way), ctypes.byref(tokens)),
               "schedule")
    return way.value, tokens.value


# CTAs of the single launch and of the even-share kernel that 148 SMs hold at once, by head_dim
RESIDENT = {128: (148 * 3, 148 * 4), 256: (148 * 2, 148 * 3)}


def way_of(lengths, *, heads, kv_heads, dim, page=16, window=128):
    """(way, tokens of a chunk) of a batch whose table is as wide as its longest row"""
    blocks = max(-(-max(0, n - window) // page) for n in lengths)
    return schedule(batch=len(lengths), heads=heads, kv_heads=kv_heads, dim=dim, blocks=blocks, page=page, window=window,
                    one_launch_ctas=RESIDENT[dim][0], share_ctas=RESIDENT[dim][1])


def test_small_calls_take_one_launch_in_the_shortest_chunks_that_fit():
    one = dict(heads=32, kv_heads=8, dim=128)
    assert way_of([300], **one) == (ONE_LAUNCH, 64)
    assert way_of([128 + 53 * 64], **one) == (ONE_LAUNCH, 128)                # 53 + 2 chunks of 8 heads fit, but 53 > 40 partials
    assert way_of([128 + 40 * 64], **one) == (ONE_LAUNCH, 64)
    assert way_of([128 + 40 * 128], **one) == (ONE_LAUNCH, 128)
    assert way_of([128 + 40 * 128 + 1], **one) == (ONE_LAUNCH, 256)
    assert way_of([128 + 40 * 256], **one) == (ONE_LAUNCH, 256)
    assert way_of([128 + 40 * 256 + 1], **one)[0] == EVEN_SHARES
    wide = dict(heads=16, kv_heads=2, dim=256)                                # four column rounds in the merge: 24 / 4 partials
    assert way_of([128 + 6 * 256], **wide) == (ONE_LAUNCH, 256)
    assert way_of([128 + 6 * 256 + 1], **wide)[0] == EVEN_SHARES


def test_what_is_resident_at_once_bounds_the_single_launch():
    """8 KV heads, one window chunk and up to two packed ones: 18 rows of three CTAs a head, 27 of two, of 444."""
    for rows, want in ((18, (ONE_LAUNCH, 64)), (19, (ONE_LAUNCH, 128)), (27, (ONE_LAUNCH, 128)), (28, (CHUNKS, 64)),
                       (29, (CHUNKS, 64)), (30, (EVEN_SHARES, 64))):
        assert way_of([32 + 128] * rows, heads=8, kv_heads=8, dim=128, window=32) == want, rows


def test_long_streams_take_chunks_in_six_waves_or_of_two():
    heads = dict(heads=32, kv_heads=8, dim=128)
    assert way_of([32768] * 64, **heads) == (CHUNKS, 4096)                    # 4096 chunks, 592 CTAs at once
    assert way_of([24576] * 64, **heads) == (EVEN_SHARES, 4096)
    assert way_of([28672] * 64, **heads) == (CHUNKS, 4096)                    # 3584 of the 3552 that six waves are
    assert way_of([8192] * 75, **heads) == (CHUNKS, 4096)                     # two chunks a row
    assert way_of([8192 + 129] * 75, **heads) == (EVEN_SHARES, 4096)


@pytest.mark.parametrize("batch,blocks", [(1, 30), (4, 256), (64, 2048)])
def test_misaligned_queries_take_the_cuda_core_kernel(batch, blocks):
    """The tensor-core kernels read query rows as 32-bit pairs: a row at an odd element must not reach them."""
    base = dict(batch=batch, blocks=blocks)
    assert schedule(**base)[0] != CUDA_CORES
    assert schedule(**base, q=0x1004)[0] != CUDA_CORES and schedule(**base, strides=(8192, 130))[0] != CUDA_CORES
    for q in (0x1001, 0x1002, 0x1003):
        assert schedule(**base, q=q)[0] == CUDA_CORES
    assert schedule(**base, strides=(4097, 128))[0] == (CUDA_CORES if batch > 1 else schedule(**base)[0])  # no second row
    assert schedule(**base, strides=(8192, 129))[0] == CUDA_CORES
    assert schedule(**base, heads=1, kv_heads=1, strides=(128, 129))[0] != CUDA_CORES                       # no second head
    for other in (dict(dtype=_lib.DTYPE_F32), dict(dim=64), dict(page=24), dict(group=16)):
        assert schedule(**base, **other)[0] == CUDA_CORES
