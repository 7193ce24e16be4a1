"""Bit-exact parity of the fused TurboQuant append (codes, metadata, block tables, window ring) with the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from anna_b200 import KVCacheConfig, Qwen3DynamicCache
from anna_b200.turboquant import launch_tq_append
from tests.helpers import TqPair, outlier_kv, packed_row_fields

pytestmark = pytest.mark.gpu


def _run_schedule(pair: TqPair, schedule, seed: int) -> None:
    gen = torch.Generator().manual_seed(seed)
    for tokens in schedule:
        shape = (pair.batch, pair.kv_heads, tokens, pair.head_dim)
        keys = outlier_kv(gen, shape, pair.dtype)
        values = outlier_kv(gen, shape, pair.dtype)
        pair.append(keys, values)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("head_dim", [64, 128, 256])
def test_append_is_bit_exact_small_window(cuda_device, dtype, bits, head_dim):
    pair = TqPair(device=cuda_device, batch=2, kv_heads=2, head_dim=head_dim, bits=bits, residual_len=8,
                  block_size=16, dtype=dtype)
    # prefill below the window, cross it, single-token steps, a chunk larger than the window, more single steps
    _run_schedule(pair, [5, 1, 1, 1, 7, 1, 30, 1, 1, 1], seed=100 + bits)
    pair.assert_bit_exact()


def test_append_config1_prefill_and_decode_steps(cuda_device):
    """Benchmark configuration 1: fp32, 8q/2kv heads, D=128, S=16, 4-bit, R=128; prefill 512 then 64 single-token appends."""
    pair = TqPair(device=cuda_device, batch=2, kv_heads=2, head_dim=128, bits=4, residual_len=128, block_size=16,
                  dtype=torch.float32)
    _run_schedule(pair, [512] + [1] * 64, seed=1)
    pair.assert_bit_exact()
    assert pair.cache.turboquant_rows[0][0].quantized_length == 512 + 64 - 128


def test_append_edge_lengths_around_window_and_block(cuda_device):
    """L in {R-1, R, R+1} and quantized lengths in {S-1, S, S+1} (window 4, block 4)."""
    pair = TqPair(device=cuda_device, batch=1, kv_heads=2, head_dim=64, bits=4, residual_len=4, block_size=4,
                  dtype=torch.bfloat16)
    gen = torch.Generator().manual_seed(9)
    for _ in range(14):
        shape = (1, 2, 1, 64)
        pair.append(outlier_kv(gen, shape, torch.bfloat16), outlier_kv(gen, shape, torch.bfloat16))
        pair.assert_bit_exact()


def test_append_constant_and_zero_vectors(cuda_device):
    """Zero keys (norm 0) and constant values (max == min -> scale clamps to 1e-8) must not produce NaN codes."""
    pair = TqPair(device=cuda_device, batch=1, kv_heads=2, head_dim=128, bits=4, residual_len=2, block_size=16,
                  dtype=torch.bfloat16)
    keys = torch.zeros(1, 2, 6, 128, dtype=torch.bfloat16)
    values = torch.full((1, 2, 6, 128), 0.75, dtype=torch.bfloat16)
    keys[:, :, 1] = 1.0
    pair.append(keys, values)
    pair.assert_bit_exact()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("head_dim", [64, 128, 256])
def test_append_of_chunks_is_bit_exact(cuda_device, dtype, bits, head_dim):
    """Calls with many tokens hold several of them per warp: chunks that leave warps and the last page partly filled, that read
    ring slots and rewrite them in the same call, on pages that are no power of two long; then single steps."""
    pair = TqPair(device=cuda_device, batch=2, kv_heads=3, head_dim=head_dim, bits=bits, residual_len=40, block_size=24,
                  dtype=dtype)
    _run_schedule(pair, [333, 1, 171, 1], seed=200 + bits)
    pair.assert_bit_exact()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_append_of_chunks_with_special_values(cuda_device, dtype):
    """Zero and constant vectors, groups of equal values, zeros of both signs and ranges below the smallest scale."""
    pair = TqPair(device=cuda_device, batch=1, kv_heads=4, head_dim=128, bits=4, residual_len=8, block_size=16, dtype=dtype)
    gen = torch.Generator().manual_seed(5)
    keys, values = (outlier_kv(gen, (1, 4, 300, 128), dtype) for _ in range(2))
    keys[:, :, 0] = 0.0
    values[:, :, 1] = 0.75
    values[:, :, 2, 32:64] = -0.0
    values[:, :, 3, ::2] = 0.0
    values[:, :, 4] *= 1e-7
    pair.append(keys, values)
    pair.assert_bit_exact()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("head_dim", [64, 128, 256])
def test_append_of_infinities_and_nans(cuda_device, dtype, bits, head_dim):
    """One call, which holds several tokens per warp, against calls too small for that (a warp per token): the same bits of
    every page and window, with NaNs and infinities of both signs in single coordinates, groups and whole vectors."""
    gen = torch.Generator().manual_seed(head_dim + bits)
    tokens, heads = 340, 4
    keys, values = (outlier_kv(gen, (1, heads, tokens, head_dim), torch.float32) for _ in range(2))
    for x in (keys, values):
        kind = torch.randint(0, 10, (1, heads, tokens, 1), generator=gen)
        some = torch.rand(x.shape, generator=gen) < 0.03
        for at, value in ((0, float("nan")), (1, float("inf")), (2, float("-inf"))):
            x.masked_fill_((kind == at) & some, value)
        x.masked_fill_(kind == 3, float("nan"))
        x[:, :, ::17, 16:32] = float("inf")
        x.mul_(torch.where(kind == 4, 1e30, 1.0)).mul_(torch.where(kind == 5, 1e-30, 1.0))
    keys, values = keys.to(dtype).to(cuda_device), values.to(dtype).to(cuda_device)
    bulk, small = (Qwen3DynamicCache(KVCacheConfig(num_hidden_layers=1, cache_block_size=24), batch_size=1,
                                     kv_cache_quantization="turboquant", kv_cache_quant_bits=bits, kv_cache_residual_len=40)
                   for _ in range(2))
    bulk.update(keys, values, 0, require_dense_cache=False)
    for at in range(0, tokens, 85):                          # 4 heads x 85 tokens: below the 1024 of the other kernel
        small.update(keys[:, :, at:at + 85], values[:, :, at:at + 85], 0, require_dense_cache=False)
    (pool_a, row_a), (pool_b, row_b) = ((cache.allocator.turboquant_layers[0], cache.turboquant_rows[0][0]) for cache in (bulk, small))
    ours, theirs = packed_row_fields(pool_a, row_a), packed_row_fields(pool_b, row_b)
    assert ours["kcodes"].shape[1] == tokens - 40
    for name, field in ours.items():
        np.testing.assert_array_equal(field.view(np.uint8), theirs[name].view(np.uint8), err_msg=name)
    assert torch.equal(pool_a.window[row_a.slot].view(torch.uint8), pool_b.window[row_b.slot].view(torch.uint8))


def test_append_of_a_chunk_leaves_shared_blocks_alone(cuda_device):
    """Blocks of the mask keep their pages' bytes in a call that holds several tokens per warp; the others get theirs."""
    dtype, bits, dim, tokens = torch.bfloat16, 4, 128, 600
    gen = torch.Generator().manual_seed(12)
    keys, values = (outlier_kv(gen, (2, 4, tokens, dim), dtype).to(cuda_device) for _ in range(2))
    cache = Qwen3DynamicCache(KVCacheConfig(num_hidden_layers=1, cache_block_size=16), batch_size=2, kv_cache_quantization="turboquant",
                              kv_cache_quant_bits=bits, kv_cache_residual_len=24)
    cache.update(keys, values, 0, require_dense_cache=False)
    pool, rows = cache.allocator.turboquant_layers[0], cache.turboquant_rows[0]
    slots = [row.slot for row in rows]
    want, window = pool.packed_pages.clone(), pool.window[slots]
    pool.packed_pages.fill_(0xA5)
    table = torch.tensor([row.block_table for row in rows], dtype=torch.int32, device=cuda_device)
    shared = [{0, 1, 31, 32, 35}, {2, 30}]                    # 36 blocks of 16 tokens each
    mask = torch.zeros(2, 2, dtype=torch.int32)
    for b, blocks in enumerate(shared):
        for block in blocks:
            mask[b, block // 32] |= torch.tensor((1 << (block % 32)) - (1 << 32 if block % 32 == 31 else 0), dtype=torch.int32)
    launch_tq_append(pool, keys, values, table, slots, [0, 0], shared_blocks=mask.to(cuda_device))
    assert torch.equal(pool.window[slots], window) and int(pool.status.item()) == 0
    for b, row in enumerate(rows):
        for block, page in enumerate(row.block_table):
            got = pool.packed_pages[page]
            if block in shared[b]:
                assert bool((got == 0xA5).all())
            else:                                            # the padding of a chunk is never written
                assert torch.equal(torch.where(got == 0xA5, want[page], got), want[page]) and not bool((got == 0xA5).all())
