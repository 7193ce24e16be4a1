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
