"""GPU: packed decode where the choice of its launches turns: one launch for window and packed chunks while all of them are
resident at once, two beyond that; even shares of long streams of three chunks or more, chunks of shorter ones."""
from __future__ import annotations

import pytest
import torch

from tests.test_gpu_tq_decode_schedules import WINDOW, assert_close, dense_attention, ragged_cache
from tests.test_tq_schedule import CHUNKS, CUDA_CORES, EVEN_SHARES, ONE_LAUNCH, way_of

pytestmark = pytest.mark.gpu


def check(device, lengths, *, heads, kv_heads, dim, bits, way, page=16, dtype=torch.bfloat16, gated=False):
    assert way_of(lengths, heads=heads, kv_heads=kv_heads, dim=dim, page=page, window=WINDOW)[0] == way
    cache, gen = ragged_cache(device, lengths, kv_heads=kv_heads, dim=dim, bits=bits, page=page, dtype=dtype)
    shape = (len(lengths), heads, 1, dim)
    query = torch.randn(shape, generator=gen, device=device).to(dtype)
    gate = torch.randn(shape, generator=gen, device=device).to(dtype) if gated else None
    out = cache.turboquant_single_token_decode_attention(0, query, scaling=dim ** -0.5, num_key_value_groups=heads // kv_heads,
                                                         gate=gate)
    again = cache.turboquant_single_token_decode_attention(0, query, scaling=dim ** -0.5,
                                                           num_key_value_groups=heads // kv_heads, gate=gate)
    assert torch.equal(out, again)  # the counters of the merge are zero again
    assert_close(out, dense_attention(cache, query, lengths, dim ** -0.5, gate), dtype)


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("dim", [128, 256])
@pytest.mark.parametrize("group", [1, 4, 8, 11])
def test_window_and_packed_chunks_in_one_launch(cuda_device, bits, dim, group):
    for lengths in ([1], [WINDOW], [WINDOW + 1], [WINDOW + 64], [WINDOW + 65, 3, WINDOW, 700], [900, 40, 1, 333, 95]):
        check(cuda_device, lengths, way=ONE_LAUNCH, heads=2 * group, kv_heads=2, dim=dim, bits=bits, page=32 if len(lengths) > 1 else 16,
              dtype=torch.float16 if group == 4 else torch.bfloat16, gated=group == 8)


@pytest.mark.parametrize("rows,way", [(18, ONE_LAUNCH), (27, ONE_LAUNCH), (28, CHUNKS), (40, EVEN_SHARES)])
def test_around_what_is_resident_at_once(cuda_device, rows, way):
    """8 KV heads, one window chunk and up to two packed ones."""
    check(cuda_device, [WINDOW + 1 + (37 * i) % 128 for i in range(rows)], way=way, heads=8, kv_heads=8, dim=128, bits=4)


@pytest.mark.parametrize("longest,way", [(8100, CHUNKS), (9100, EVEN_SHARES)])
def test_long_streams_of_two_and_of_three_chunks(cuda_device, longest, way):
    rows = 75 if longest < 8192 else 50
    check(cuda_device, [longest if i % 7 == 0 else 200 + (911 * i) % longest for i in range(rows)], way=way, heads=8,
          kv_heads=8, dim=128, bits=3)


@pytest.mark.parametrize("lengths", [[WINDOW + 3520], [WINDOW + 3521], [WINDOW + 128 * 55 + 1], [8100], [1500, 1377, 40, 1501],
                                     [2500, 200, 1100, 1999, 640, 2048, 311, 900]])
@pytest.mark.parametrize("dim,bits", [(128, 3), (256, 4)])
def test_longer_chunks_in_one_launch(cuda_device, lengths, dim, bits):
    """Chunks of 128 and 256 tokens where 64 give more CTAs than are resident, and lengths beyond those."""
    check(cuda_device, lengths, way=ONE_LAUNCH if len(lengths) < 8 else EVEN_SHARES, heads=16, kv_heads=8, dim=dim, bits=bits,
          page=32 if dim == 256 else 16)


@pytest.mark.parametrize("dim,kv_heads,rows", [(128, 8, 9), (256, 4, 13)])
@pytest.mark.parametrize("group", [1, 3, 4])
@pytest.mark.parametrize("longest", [1800, 3000, 6500])
def test_short_and_long_shares_of_4_bit_pairs(cuda_device, dim, kv_heads, rows, group, longest):
    """Shares of up to 512 tokens take an instance of their own: 303104 tokens of 592 CTAs at head_dim 128, 227328 of 444 at 256."""
    check(cuda_device, [longest if i % 4 == 0 else 1 + (977 * i) % longest for i in range(rows)], way=EVEN_SHARES, heads=group * kv_heads,
          kv_heads=kv_heads, dim=dim, bits=4, dtype=torch.float16 if group == 3 else torch.bfloat16, gated=group == 3)


@pytest.mark.parametrize("dim,bits,heads", [(128, 4, 8), (128, 3, 2), (256, 2, 22)])
@pytest.mark.parametrize("lengths", [[700], [WINDOW + 5, 1, 2300, 90]])
def test_query_rows_at_odd_elements(cuda_device, dim, bits, heads, lengths):
    """Views of a wider projection: an odd offset, an odd head stride, an odd row stride; with and without peers."""
    cache, gen = ragged_cache(cuda_device, lengths, kv_heads=2, dim=dim, bits=bits, page=16, dtype=torch.bfloat16)
    batch = len(lengths)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device=cuda_device).to(torch.bfloat16)

    for query in (randn(batch * heads * dim + 1)[1:].view(batch, heads, 1, dim), randn(batch, heads, 1, dim + 1)[..., :dim],
                  randn(batch, heads * dim + 1)[:, :-1].unflatten(1, (heads, 1, dim)),
                  randn(batch, heads * dim + 2)[:, 1:-1].unflatten(1, (heads, 1, dim))):
        assert query.stride(3) == 1
        assert batch == 1 or query.data_ptr() % 4 or query.stride(0) % 2 or query.stride(1) % 2
        args = dict(scaling=dim ** -0.5, num_key_value_groups=heads // 2)
        out = cache.turboquant_single_token_decode_attention(0, query, **args)
        assert_close(out, dense_attention(cache, query, lengths, dim ** -0.5), torch.bfloat16)
        local, peer = torch.empty_like(out), torch.empty_like(out)
        cache.turboquant_single_token_decode_attention(0, query, **args, output=local, peer_outputs=(peer.data_ptr(),))
        assert_close(local, dense_attention(cache, query, lengths, dim ** -0.5), torch.bfloat16)
        assert torch.equal(local, peer)


@pytest.mark.parametrize("dim,heads,bits", [(128, 16, 3), (128, 10, 2), (256, 8, 3), (256, 6, 4), (256, 10, 2), (256, 16, 4)])
def test_merges_of_groups_that_fill_the_threads_or_not(cuda_device, dim, heads, bits):
    """The last CTA's threads have one, two or four columns of four dims of the group, read side by side where an instance has
    the registers; 2 KV heads, so that one long row leaves many partials to merge."""
    check(cuda_device, [12000, 11000], way=EVEN_SHARES, heads=heads, kv_heads=2, dim=dim, bits=bits)


@pytest.mark.parametrize("page", [8, 24])
@pytest.mark.parametrize("dim,bits", [(128, 2), (128, 3), (256, 4)])
def test_single_heads_on_pages_that_are_no_multiple_of_16(cuda_device, page, dim, bits):
    """The CUDA-core kernel looks page and place in the page up a round ahead: rounds that end inside a page, at its end and past
    the last token."""
    for lengths in ([WINDOW + 1], [WINDOW + page], [WINDOW + 2 * page + 1, 3, WINDOW, 700], [900, 40, 1, 333, 95]):
        check(cuda_device, lengths, way=CUDA_CORES, heads=4, kv_heads=4, dim=dim, bits=bits, page=page, gated=bits == 3)
