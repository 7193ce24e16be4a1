"""The dense view of packed rows (csrc/tq_materialize.cu) against the oracle's de-quantization of the same codes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from anna_b200.turboquant import launch_tq_gather_dense, launch_tq_materialize
from tests.helpers import DTYPE_CODE, TqPair, outlier_kv, to_np

pytestmark = pytest.mark.gpu
DTYPES, BITS, DIMS = [torch.float32, torch.bfloat16, torch.float16], [2, 3, 4], [64, 128, 256]


def _pair(device, dtype, bits, dim, *, batch, tokens, block, residual, seed=0):
    pair = TqPair(device=device, batch=batch, kv_heads=3, head_dim=dim, bits=bits, residual_len=residual, block_size=block, dtype=dtype)
    gen = torch.Generator().manual_seed(seed + bits)
    pair.append(*(outlier_kv(gen, (batch, 3, tokens, dim), dtype) for _ in range(2)))
    return pair


def _table(pair):
    rows = [row.block_table for row in pair.cache.turboquant_rows[0]]
    return torch.tensor(rows, dtype=torch.int32, device=pair.device)


def _dequantized(pair, row, tokens):
    """Keys and values of a row's first packed tokens, in fp32 before and after rounding to the cache dtype; norms of the keys."""
    orc, pool = pair.rows[row], pair.pool
    keys = oracle.dequantize_keys(orc.idx[:, :tokens], orc.sign[:, :tokens], orc.norms[:, :tokens], orc.rnorms[:, :tokens], pool.bits)
    values = oracle.dequantize_values(orc.vdata[:, :tokens], orc.vscales[:, :tokens], orc.vzeros[:, :tokens], pool.bits, pool.value_group)
    return keys, oracle.round_dtype(values, DTYPE_CODE[pair.dtype]), orc.norms[:, :tokens]


def _check_keys(got, want, norms, dtype, dim):
    """The kernel's fp32 sums contract differently: each of the two transforms' log2(D) levels and the few products around them
    rounds to 2^-24 of the token's norm at most, on both sides; then the kernel's are rounded to the cache dtype."""
    arithmetic = 2 * (2 * np.log2(dim) + 6) * 2.0 ** -24 * norms[..., None]
    spacing = {torch.float32: 0.0, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    tiny = 2.0 ** -25 if dtype == torch.float16 else 0.0   # half of its denormals' spacing is not relative
    half = spacing / 2 * np.abs(want) + tiny
    assert (np.abs(got - want) <= half + arithmetic * (1 + spacing)).all(), float((np.abs(got - want) - half).max())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bits", BITS)
@pytest.mark.parametrize("dim", DIMS)
@pytest.mark.parametrize("block,residual", [(24, 40), (16, 7)])
def test_dense_view_of_a_ragged_batch(cuda_device, dtype, bits, dim, block, residual):
    """Lengths below and at the window's, one packed token, the edges of a page and of a warp's tokens, all of it; a hole in a
    table reads as zeros, and so does what lies behind a row's length."""
    total = 333
    lengths = [3, residual, residual + 1, residual + block, residual + block + 1, 200, total]
    pair = _pair(cuda_device, dtype, bits, dim, batch=len(lengths), tokens=total, block=block, residual=residual)
    table = _table(pair)
    hole = 2
    table[-1, hole] = -1
    table[-2, hole] = pair.pool.capacity()
    max_len = total + 37
    slots = [row.slot for row in pair.cache.turboquant_rows[0]]
    keys, values, lengths_dev = launch_tq_gather_dense(pair.pool, table, slots, lengths, max_len)
    assert keys.shape == values.shape == (len(lengths), 3, max_len, dim) and lengths_dev.tolist() == lengths
    for b, length in enumerate(lengths):
        packed = max(0, length - residual)
        got_k, got_v = to_np(keys[b]), to_np(values[b])
        want_k, want_v, norms = _dequantized(pair, b, packed)
        if b >= len(lengths) - 2:
            for want in (want_k, want_v):
                want[:, hole * block:(hole + 1) * block] = 0.0
            assert not got_k[:, hole * block:(hole + 1) * block].any()
        np.testing.assert_array_equal(got_v[:, :packed], want_v)
        _check_keys(got_k[:, :packed], want_k, norms, dtype, dim)
        ring = torch.arange(packed, length, device=cuda_device) % residual
        for got, which in ((keys, 0), (values, 1)):
            assert torch.equal(got[b, :, packed:length], pair.pool.window[slots[b], which].index_select(1, ring))
            assert not got[b, :, length:].any()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bits", BITS)
@pytest.mark.parametrize("dim", DIMS)
def test_packed_prefix_into_strided_rows(cuda_device, dtype, bits, dim):
    """The packed prefix alone, into views of wider tensors, which keep what they hold behind a row's prefix and in holes.  Rows
    that are aligned for 16-byte stores take the kernel of several tokens per warp, others that of one: the same bits."""
    pair = _pair(cuda_device, dtype, bits, dim, batch=2, tokens=190, block=16, residual=13, seed=7)
    packed = [177, 60]
    table = _table(pair)
    table[0, 5] = -1
    access = min(16, dim // 32 * dtype.itemsize)             # what a lane of the second kernel stores at once
    results = []
    for shift in (0, access // dtype.itemsize if access < 16 else None):
        if shift is None:
            continue
        flat = [torch.full((2 * 3 * 180 * (dim + 16) + 16,), 7.0, dtype=dtype, device=cuda_device) for _ in range(2)]
        key_out, value_out = (x[shift:shift + 2 * 3 * 180 * (dim + 16)].view(2, 3, 180, dim + 16)[..., :dim] for x in flat)
        assert (key_out.data_ptr() % 16 == 0) == (shift == 0)
        launch_tq_materialize(pair.pool, table, packed, key_out, value_out)
        results.append((key_out, value_out))
        for b, n in enumerate(packed):
            want_k, want_v, norms = _dequantized(pair, b, n)
            for got in (key_out[b], value_out[b]):
                assert bool((got[:, n:] == 7.0).all()) and (b == 1 or bool((got[:, 80:96] == 7.0).all()))
            keep = [t for t in range(n) if b == 1 or not 80 <= t < 96]
            np.testing.assert_array_equal(to_np(value_out[b])[:, keep], want_v[:, keep])
            _check_keys(to_np(key_out[b])[:, keep], want_k[:, keep], norms[:, keep], dtype, dim)
        assert all(bool((x.view(-1)[:shift] == 7.0).all()) for x in flat)
    if len(results) == 2:
        assert all(torch.equal(a, b) for a, b in zip(*results, strict=True))


def test_outputs_at_misaligned_addresses_are_refused(cuda_device):
    pair = _pair(cuda_device, torch.bfloat16, 4, 256, batch=1, tokens=50, block=16, residual=8)
    wide = torch.zeros(1, 3, 48, 260, dtype=torch.bfloat16, device=cuda_device)
    for out in (wide[..., 4:], wide[..., :256]):             # an address, a stride of 8 bytes too many for 16-byte stores
        with pytest.raises(RuntimeError, match="aligned"):
            launch_tq_materialize(pair.pool, _table(pair), [42], out, out)
