"""CPU: the kernel that a chunk's attention takes (csrc/gqa_prefill_umma.cu), asked of the library's own rules."""
from __future__ import annotations

import ctypes

from anna_b200 import _lib

MMA_SYNC, ONE_CTA = 0, 1
# CTAs in clusters of n that the GPU holds at once: any SMs together, or those of eight groups of 18
ANY, GROUPS = ((ctypes.c_int * 17)(0, 148, *[ctas(n) for n in range(2, 17)]) for ctas in (lambda n: 148 // n * n, lambda n: 8 * (18 // n) * n))


def choice(batch, heads, kv_heads, q_len, key_len, dim, dtype=_lib.DTYPE_BF16, ctas=ANY):
    splits = ctypes.c_int(-1)
    _lib.check(_lib.lib().anna_kv_selftest_prefill_choice(batch, heads, kv_heads, q_len, key_len, dim, dtype, ctas, ctypes.byref(splits)),
               "anna_kv_selftest_prefill_choice")
    return splits.value


def test_a_few_positions_over_a_few_keys_stay_with_mma_sync():
    assert choice(1, 8, 2, 8, 64, 128) == MMA_SYNC and choice(1, 8, 2, 8, 65, 128) == ONE_CTA
    assert choice(2, 16, 2, 5, 32, 256) == MMA_SYNC and choice(2, 16, 2, 5, 33, 256) == ONE_CTA
    assert choice(2, 4, 4, 33, 96, 64) == MMA_SYNC
    assert choice(1, 8, 2, 16, 48, 128, _lib.DTYPE_F32) == MMA_SYNC and choice(1, 8, 2, 64, 64, 80) == MMA_SYNC
    for dim in (64, 128, 256):
        assert choice(1, 8, 2, 64, 64, dim) == ONE_CTA                        # half of a CTA's rows


def test_keys_are_shared_where_query_tiles_leave_sms_empty():
    for ctas in (ANY, GROUPS):
        for dim, two, three, four, sixteen in (
                (64, (3, 9, 3, 279, 792), (3, 9, 3, 48, 324), (2, 1, 1, 141, 475), (1, 2, 2, 8, 1926)),
                (128, (4, 9, 3, 278, 936), (1, 2, 2, 6, 265), (1, 4, 4, 5, 507), (1, 2, 1, 10, 1976)),
                (256, (3, 9, 3, 144, 1359), (3, 12, 4, 15, 572), (1, 1, 1, 149, 969), (2, 1, 1, 5, 1994))):
            assert [choice(*shape, dim, ctas=ctas) for shape in (two, three, four, sixteen)] == [2, 3, 4, 16]
        assert choice(8, 16, 4, 2048, 10240, 128, ctas=ctas) == ONE_CTA       # many waves
        assert choice(1, 16, 2, 953, 3001, 256, ctas=ctas) == ONE_CTA         # 120 query tiles
        assert choice(1, 32, 8, 512, 128, 128, ctas=ctas) == ONE_CTA          # one key tile


def test_no_more_ctas_share_than_there_are_key_tiles():
    for tiles in range(1, 17):
        assert choice(1, 4, 4, 64, 128 * tiles, 128) <= tiles and choice(1, 4, 4, 64, 64 * tiles, 256) <= tiles


def test_sizes_that_the_gpu_has_no_clusters_of_are_not_chosen():
    for most in range(1, 17):
        ctas = (ctypes.c_int * 17)(0, 148, *[148 // n * n if n <= most else 0 for n in range(2, 17)])
        assert choice(1, 2, 1, 10, 1976, 128, ctas=ctas) <= most
        if 16 % most == 0:                                                     # sixteen key tiles
            assert choice(1, 2, 1, 10, 1976, 128, ctas=ctas) == most
