"""GPU: the merge of split-K partials and the division of the work, at the sizes where they can go wrong.

Un-quantized paged decode against 64-bit attention: numbers of partials around the loads a thread keeps in flight, head groups
whose columns fill a part of the CTA, all of it or several rounds, and batches around the 32 rows that a warp lines up by
itself, with rows that have no key."""
from __future__ import annotations

import pytest
import torch

from anna_b200 import fused_ops

pytestmark = pytest.mark.gpu

# 2-norm of the difference over that of the result, row by row: 16-bit probabilities (2^-9 of bf16, 2^-12 of fp16) and the
# output's own rounding, each at most half a unit; in fp32 sums in another order (up to 8e-7).
REL = {torch.bfloat16: 6e-3, torch.float16: 1e-3, torch.float32: 5e-6}


def check(device, dtype, lengths, *, heads, kv_heads, dim, page=16, seed=0):
    gen = torch.Generator(device=device).manual_seed(seed)
    batch, blocks = len(lengths), [(n + page - 1) // page for n in lengths]
    pages = sum(blocks) + 3
    keys, values = (torch.randn((pages, kv_heads, page, dim), generator=gen, device=device).to(dtype) for _ in range(2))
    order = torch.randperm(pages, generator=gen, device=device).to(torch.int32)
    table = torch.full((batch, max(blocks)), -1, dtype=torch.int32, device=device)
    at = 0
    for row, n in enumerate(blocks):
        table[row, :n] = order[at:at + n]
        at += n
    query = torch.randn((batch, heads, 1, dim), generator=gen, device=device).to(dtype)
    visible = torch.tensor(lengths, dtype=torch.long, device=device)
    out = fused_ops.run_paged_gqa_decode_fused(query=query, key_pages=keys, value_pages=values, page_table=table,
                                               visible_lengths=visible, scaling=dim ** -0.5)
    for row, n in enumerate(lengths):
        if n == 0:
            assert not out[row].any()
            continue
        ids = table[row, :blocks[row]].long()
        k, v = (x[ids].transpose(0, 1).flatten(1, 2)[:, :n].double() for x in (keys, values))
        q = query[row, :, 0].double().view(kv_heads, heads // kv_heads, dim)
        want = ((q @ k.transpose(1, 2)) * dim ** -0.5).softmax(-1) @ v
        error = (out[row, :, 0].double() - want.flatten(0, 1)).norm() / want.norm()
        assert float(error) < REL[dtype], f"row {row} of {n} keys: {float(error):.2e}"


@pytest.mark.parametrize("dtype,dim", [(torch.bfloat16, 64), (torch.float16, 128), (torch.bfloat16, 256), (torch.float32, 64),
                                       (torch.float32, 128)])
@pytest.mark.parametrize("group", [1, 3, 4, 5, 8, 11])
def test_merge_of_any_number_of_partials(cuda_device, dtype, dim, group):
    for length in (1, 16, 17, 960, 1040, 2111, 5000):
        check(cuda_device, dtype, [length], heads=2 * group, kv_heads=2, dim=dim, seed=length)


@pytest.mark.parametrize("rows", [1, 2, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("kv_heads", [1, 4])
def test_rows_around_a_warp(cuda_device, rows, kv_heads):
    lengths = [0 if i % 5 == 3 else 1 + (997 * i) % 700 for i in range(rows)]
    check(cuda_device, torch.bfloat16, lengths, heads=4 * kv_heads, kv_heads=kv_heads, dim=128, page=32, seed=rows)
    check(cuda_device, torch.float16, [0] * (rows - 1) + [333], heads=kv_heads, kv_heads=kv_heads, dim=64, seed=rows)
