"""GPU: decode over packed pages at the sizes where its schedules and fragment layouts can go wrong.

Contexts that end inside a 16-token tile, inside a pair of tiles or inside the window, ragged batches, head groups that
fill, half fill or overflow the eight columns of a product, every code width, both tensor-core head sizes, one-run and
six-run pages; each against 64-bit attention over the dense view of the same cache (which has parity tests of its own)."""
from __future__ import annotations

import dataclasses

import pytest
import torch

from anna_b200 import KVCacheConfig, Qwen3DynamicCache, Qwen3PageAllocator, _lib
from tests.helpers import TQ_ATOL

pytestmark = pytest.mark.gpu
WINDOW = 32


def ragged_cache(device, lengths, *, kv_heads, dim, bits, page, dtype, seed=0):
    config = KVCacheConfig(num_hidden_layers=1, cache_block_size=page)
    allocator = Qwen3PageAllocator(config)
    gen = torch.Generator(device=device).manual_seed(seed)
    rows = []
    for n in lengths:
        cache = Qwen3DynamicCache(config, allocator=allocator, batch_size=1, kv_cache_quantization="turboquant",
                                  kv_cache_quant_bits=bits, kv_cache_residual_len=WINDOW)
        k, v = (torch.randn((1, kv_heads, n, dim), generator=gen, device=device).to(dtype) for _ in range(2))
        cache.update(k, v, 0, require_dense_cache=False)
        rows.append(cache)
    return Qwen3DynamicCache.stack(rows, config, clone_turboquant_rows=False), gen


def dense_attention(cache, query, lengths, scaling, gate=None):
    keys, values, _ = cache._gather_layer_cache(0)
    batch, heads, _, dim = query.shape
    kv_heads = keys.shape[1]
    q = query.double().view(batch, kv_heads, heads // kv_heads, dim)
    scores = torch.einsum("bhgd,bhld->bhgl", q, keys.double()) * scaling
    hidden = torch.arange(keys.shape[2], device=query.device)[None] >= torch.tensor(lengths, device=query.device)[:, None]
    scores = scores.masked_fill(hidden[:, None, None], float("-inf"))
    out = torch.einsum("bhgl,bhld->bhgd", scores.softmax(-1), values.double()).reshape(batch, heads, 1, dim)
    return out if gate is None else out * torch.sigmoid(gate.double())


# 2-norm of the difference over that of the result: the keys and values of the 64-bit attention are the dense view's, rounded
# to the cache dtype (2^-9 of bf16), like the output and, inside, the probabilities and values (2^-11): up to 3.2e-3 together.
# In fp32 it is sums in another order: up to 8e-7.
REL = {torch.bfloat16: 1e-2, torch.float16: 1e-2, torch.float32: 5e-6}


def assert_close(out, want, dtype):
    tol = TQ_ATOL[dtype]  # what the quantized decode is allowed against the reference everywhere in these tests
    torch.testing.assert_close(out.double(), want, atol=tol, rtol=tol)
    # an average over a long context is far below that: a lost part of it shows in the relative error, row by row
    error = (out.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert float(error.max()) < REL[dtype], f"relative error of the rows up to {float(error.max()):.2e}"


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("dim,kv_heads,group,page", [(128, 2, 4, 16), (128, 1, 1, 32), (128, 3, 5, 16), (128, 2, 12, 16),
                                                     (256, 2, 8, 16), (256, 1, 3, 32)])
def test_edges_of_tiles_pairs_and_groups(bits, dim, kv_heads, group, page):
    device, dtype = torch.device("cuda"), torch.float16
    lengths = [1, WINDOW, WINDOW + 1, WINDOW + 15, WINDOW + 16, WINDOW + 17, WINDOW + 32, WINDOW + 33, 1000, 2111]
    cache, gen = ragged_cache(device, lengths, kv_heads=kv_heads, dim=dim, bits=bits, page=page, dtype=dtype)
    shape = (len(lengths), kv_heads * group, 1, dim)
    query, gate = (torch.randn(shape, generator=gen, device=device).to(dtype) for _ in range(2))
    scaling = dim ** -0.5
    for g in (None, gate):
        out = cache.turboquant_single_token_decode_attention(0, query, scaling=scaling, num_key_value_groups=group, gate=g)
        assert_close(out, dense_attention(cache, query, lengths, scaling, g), dtype)


@pytest.mark.parametrize("batch,length", [(1, 40000), (2, 9000), (300, 70), (300, 700), (1100, 50)])
def test_long_rows_and_large_batches(batch, length):
    """One row and two over the whole chip; a tile or two per row, which is a small call's chunks, and more, which are shares;
    more rows than the even-share schedule takes."""
    device, dtype = torch.device("cuda"), torch.bfloat16
    config = KVCacheConfig(num_hidden_layers=1, cache_block_size=16)
    gen = torch.Generator(device=device).manual_seed(3)
    cache = Qwen3DynamicCache(config, batch_size=batch, kv_cache_quantization="turboquant", kv_cache_quant_bits=3,
                              kv_cache_residual_len=WINDOW)
    k, v = (torch.randn((batch, 1, length, 128), generator=gen, device=device).to(dtype) for _ in range(2))
    cache.update(k, v, 0, require_dense_cache=False)
    query = torch.randn((batch, 4, 1, 128), generator=gen, device=device).to(dtype)
    for _ in range(2):  # the merge counters are back at zero after a call
        out = cache.turboquant_single_token_decode_attention(0, query, scaling=0.1, num_key_value_groups=4)
        assert_close(out, dense_attention(cache, query, [length] * batch, 0.1), dtype)


class Arguments:
    """The library with two arguments of the packed decode replaced: the chunk length and the merge counters."""

    def __init__(self, library, chunk_tokens: int, counters: bool) -> None:
        self._library, self._chunk_tokens, self._counters = library, chunk_tokens, counters

    def __getattr__(self, name):
        return getattr(self._library, name)

    def anna_tq_paged_decode(self, *args):
        args = list(args)
        assert args[20] >= 2 + -(-2111 // max(self._chunk_tokens, 64))  # the scratch was planned for 64-token chunks
        args[21] = self._chunk_tokens
        args[22] = args[22] if self._counters else None
        return self._library.anna_tq_paged_decode(*args)


@pytest.mark.parametrize("counters", [True, False])
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("dim,group", [(128, 3), (128, 8), (128, 12), (256, 3), (256, 8), (256, 12)])
def test_chunks_of_a_given_length(monkeypatch, bits, dim, group, counters):
    """The chunk length is the caller's: fixed chunks, whatever the batch, with the merge in the kernel or behind it."""
    device, dtype, kv_heads = torch.device("cuda"), torch.bfloat16, 2
    lengths = [1, WINDOW, WINDOW + 1, WINDOW + 127, WINDOW + 128, WINDOW + 145, 700, 2111]
    cache, gen = ragged_cache(device, lengths, kv_heads=kv_heads, dim=dim, bits=bits, page=16, dtype=dtype)
    query = torch.randn((len(lengths), kv_heads * group, 1, dim), generator=gen, device=device).to(dtype)
    want = dense_attention(cache, query, lengths, dim ** -0.5)
    library = _lib.lib()
    for chunk_tokens in (128, 1024):
        monkeypatch.setattr(_lib, "lib", lambda: Arguments(library, chunk_tokens, counters))
        for _ in range(2):  # the merge counters are back at zero after a call
            out = cache.turboquant_single_token_decode_attention(0, query, scaling=dim ** -0.5, num_key_value_groups=group)
            assert_close(out, want, dtype)


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("group", [1, 4, 5, 8])
def test_fp32_merges_in_one_or_two_kernels(dim, group):
    """Many 64-token chunks per head: up to 4 heads, or 64 dims, the split kernel merges them, else a second one does."""
    device, dtype = torch.device("cuda"), torch.float32
    lengths = [WINDOW, 65 + WINDOW, 3001]
    cache, gen = ragged_cache(device, lengths, kv_heads=2, dim=dim, bits=4, page=16, dtype=dtype)
    query = torch.randn((3, 2 * group, 1, dim), generator=gen, device=device)
    for _ in range(2):
        out = cache.turboquant_single_token_decode_attention(0, query, scaling=dim ** -0.5, num_key_value_groups=group)
        assert_close(out, dense_attention(cache, query, lengths, dim ** -0.5), dtype)


@pytest.mark.parametrize("group", [4, 8])
def test_codebook_without_symmetry(group):
    """Centroids are the caller's: the 3-bit path may not rely on +-c0, +-c1 beyond what it detects."""
    device, dtype = torch.device("cuda"), torch.float16
    lengths = [200, 77]
    cache, gen = ragged_cache(device, lengths, kv_heads=2, dim=128, bits=3, page=16, dtype=dtype)
    pool = cache.allocator.turboquant_layers[0]
    skewed = pool.tables.centroids + torch.tensor([0.0, 0.3, 0.1, -0.2], device=device)
    pool._tables = dataclasses.replace(pool.tables, centroids=skewed)
    query = torch.randn((2, 2 * group, 1, 128), generator=gen, device=device).to(dtype)
    out = cache.turboquant_single_token_decode_attention(0, query, scaling=0.2, num_key_value_groups=group)
    assert_close(out, dense_attention(cache, query, lengths, 0.2), dtype)


@pytest.mark.parametrize("bits", [2, 3, 4])
def test_nan_and_infinite_queries_stay_in_their_head(bits):
    device, dtype = torch.device("cuda"), torch.bfloat16
    lengths = [300]
    cache, gen = ragged_cache(device, lengths, kv_heads=1, dim=128, bits=bits, page=16, dtype=dtype)
    query = torch.randn((1, 4, 1, 128), generator=gen, device=device).to(dtype)
    clean = cache.turboquant_single_token_decode_attention(0, query, scaling=0.1, num_key_value_groups=4)
    query[0, 1, 0, 7] = float("nan")
    query[0, 2, 0, 9] = float("inf")
    out = cache.turboquant_single_token_decode_attention(0, query, scaling=0.1, num_key_value_groups=4)
    assert bool(out[0, 1].isnan().all()) and bool(out[0, 2].isnan().all())
    assert torch.equal(out[0, [0, 3]], clean[0, [0, 3]])
