"""The work a serving engine has the KV cache do, as cases that can be prepared, run and timed one by one.

A case is a dict of plain values; ``kind`` says which call it is:

* ``tq_decode``    one decode step's attention over a TurboQuant cache
                   (``Qwen3DynamicCache.turboquant_single_token_decode_attention``)
* ``paged_decode`` one decode step's attention over un-quantized pages (``run_paged_gqa_decode_fused``)
* ``prefill``      causal attention of a chunk of prompt tokens over dense keys (``grouped_query_attention``)
* ``admit``        new sequences are quantize-appended into the page pool and leave it again
                   (``Qwen3DynamicCache.update`` / ``release``)
* ``prompt``       one layer's whole prompt over a TurboQuant cache in chunks: append, dense view, attention
* ``generate``     one layer's whole request: prompt, then decode steps of one token (append + attention), then release

Shapes follow the benchmark's configurations (32 query / 8 KV heads, 16 / 4 and 16 / 2, head_dim 128 and 256, windows of
128 tokens, pages of 16 tokens, the cache's default of 32, 2- to 4-bit codes, contexts from a few hundred to 32768).
"""
from __future__ import annotations

import json
import math
import random
import struct
from pathlib import Path

import torch

import anna_b200

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEM = {"bf16": 2, "fp16": 2, "fp32": 4}
KEYS_AT_ONCE = 1 << 18  # token-heads of one exact() piece


def listed() -> list[dict]:
    return [
        # one chat user, a few thousand tokens of history: nothing but launches and latency
        dict(name="tq4_one_chat", kind="tq_decode", dtype="bf16", bits=4, batch=1, q_heads=32, kv_heads=8, dim=128,
             low=4000, high=4000, page=16, window=128, gate=False, dist="normal"),
        # the CPU-runnable layer: fp32, two rows, outlier channels
        dict(name="tq4_fp32_pair", kind="tq_decode", dtype="fp32", bits=4, batch=2, q_heads=8, kv_heads=2, dim=128,
             low=576, high=576, page=16, window=128, gate=False, dist="outlier"),
        # a mid-size batch of short conversations with gated attention, on the cache's default page size
        dict(name="tq4_d256_gated", kind="tq_decode", dtype="fp16", bits=4, batch=16, q_heads=16, kv_heads=2, dim=256,
             low=400, high=4100, page=32, window=128, gate=True, dist="normal"),
        # whole-box decode: one GPU's eighth of 512 sequences x 32768 tokens
        dict(name="tq4_batch_long", kind="tq_decode", dtype="bf16", bits=4, batch=64, q_heads=32, kv_heads=8, dim=128,
             low=32768, high=32768, page=16, window=128, gate=False, dist="normal"),
        # 2-bit codes, head_dim 256, ragged contexts, channels of very different scale
        dict(name="tq2_d256_ragged", kind="tq_decode", dtype="bf16", bits=2, batch=64, q_heads=16, kv_heads=2, dim=256,
             low=4096, high=32768, page=16, window=128, gate=False, dist="lognormal"),
        # the decode rows of a continuously batched step, 3-bit codes
        dict(name="tq3_ragged", kind="tq_decode", dtype="bf16", bits=3, batch=128, q_heads=16, kv_heads=4, dim=128,
             low=512, high=16384, page=16, window=128, gate=False, dist="normal"),
        # un-quantized serving: ragged batch, pages in random order
        dict(name="paged_ragged", kind="paged_decode", dtype="bf16", batch=32, q_heads=32, kv_heads=8, dim=128, low=1024,
             high=8192, page=16, gate=False),
        # a handful of short un-quantized rows with gated attention
        dict(name="paged_small", kind="paged_decode", dtype="fp16", batch=4, q_heads=16, kv_heads=4, dim=128, low=60,
             high=900, page=32, gate=True),
        # the prefill side of a continuously batched step: 2048-token chunks over 8192 cached tokens
        dict(name="prefill_chunks", kind="prefill", dtype="bf16", batch=8, q_heads=16, kv_heads=4, dim=128, chunk=2048,
             past=8192, ragged=False),
        # the append of the same step: eight 2048-token chunks of new sequences into the 3-bit pool
        dict(name="admit_3bit", kind="admit", dtype="bf16", bits=3, batch=8, kv_heads=4, dim=128, tokens=2048, page=16,
             window=128, dist="normal"),
        # one long prompt of odd length, chunked, over a 2-bit cache of head_dim 256
        dict(name="prompt_d256", kind="prompt", dtype="bf16", bits=2, batch=1, q_heads=16, kv_heads=2, dim=256,
             tokens=3001, chunk=2048, page=16, window=128, dist="lognormal"),
        # a few short requests from admission to release
        dict(name="generate_short", kind="generate", dtype="bf16", bits=4, batch=4, q_heads=32, kv_heads=8, dim=128,
             tokens=300, steps=32, page=16, window=128, dist="normal"),
    ]


def _log_int(rng: random.Random, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["tq_decode"] * 5 + ["paged_decode"] * 2 + ["prefill"] * 2 + ["admit", "prompt", "generate"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    dim = rng.choice([128, 128, 128, 256, 256, 64])
    kv_heads = rng.choice([2, 4, 8]) if dim < 256 else rng.choice([2, 4])
    group = rng.choice([4, 8, rng.choice([1, 2, 3, 6, 12])])
    case = dict(kind=kind, dtype=dtype, kv_heads=kv_heads, dim=dim)
    if kind != "admit":
        case["q_heads"] = kv_heads * group
    if kind == "paged_decode":
        batch = _log_int(rng, 1, 64)
        high = _log_int(rng, 50, min(16384, 262144 // batch))
        return dict(case, batch=batch, low=max(1, high // rng.randint(1, 8)), high=high, page=rng.choice([16, 32]),
                    gate=rng.random() < 0.3)
    if kind == "prefill":
        batch, chunk = rng.choice([1, 1, 2, 4, 8]), _log_int(rng, 5, 2048)
        return dict(case, batch=batch, chunk=chunk, past=rng.choice([0, _log_int(rng, 100, 8192)]),
                    ragged=rng.random() < 0.5)
    case.update(bits=rng.choice([2, 3, 4, 4]), page=rng.choice([16, 16, 32]), window=rng.choice([128, 128, 64]),
                dist=rng.choice(["normal", "normal", "outlier", "lognormal"]))
    if kind == "tq_decode":
        if rng.random() < 0.1:
            case["dtype"] = "fp32"
        most = 8192 if case["dtype"] == "fp32" or dim == 64 else 1 << 20
        batch = _log_int(rng, 1, 8 if most == 8192 else 128)
        high = _log_int(rng, 200, min(32768, max(400, most // batch)))
        return dict(case, batch=batch, low=max(1, high // rng.randint(1, 8)), high=high, gate=rng.random() < 0.3)
    if kind == "admit":
        return dict(case, batch=_log_int(rng, 1, 16), tokens=_log_int(rng, 130, 2048))
    if kind == "prompt":
        return dict(case, batch=rng.choice([1, 1, 2, 4]), tokens=_log_int(rng, 200, 4096), chunk=rng.choice([512, 2048]))
    return dict(case, batch=_log_int(rng, 1, 16), tokens=_log_int(rng, 20, 1000), steps=rng.randint(4, 32))


# ---------------------------------------------------------------------------------------------------------------
# inputs


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen: torch.Generator, shape, dtype: torch.dtype) -> torch.Tensor:
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def _channels(case: dict, gen: torch.Generator) -> torch.Tensor | None:
    """Per (K or V, head, channel) factors of the case's distribution."""
    heads, dim = case["kv_heads"], case["dim"]
    if case["dist"] == "lognormal":
        return torch.exp(0.5 * torch.randn((2, heads, 1, dim), generator=gen, device="cuda"))
    if case["dist"] == "outlier":
        order = torch.rand((2, heads, 1, dim), generator=gen, device="cuda").argsort(dim=-1)
        return torch.where(order < 4, 8.0, 1.0)
    return None


def _kv(case: dict, gen: torch.Generator, factors, rows: int, tokens: int) -> tuple[torch.Tensor, torch.Tensor]:
    shape = (rows, case["kv_heads"], tokens, case["dim"])
    pair = []
    for i in range(2):
        x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
        pair.append((x if factors is None else x.mul_(factors[i])).to(DTYPES[case["dtype"]]))
    return pair[0], pair[1]


def _lengths(case: dict) -> list[int]:
    """Context lengths of the rows: spread evenly over [low, high], in a fixed shuffled order."""
    n, low, high = case["batch"], case["low"], case["high"]
    if n == 1:
        return [high]
    lengths = [low + (high - low) * i // (n - 1) for i in range(n)]
    random.Random(n).shuffle(lengths)
    return lengths


def _pieces(case: dict):
    """(first row, rows, tokens) in the order in which the context of a tq_decode case is appended."""
    lengths = _lengths(case)
    if len(set(lengths)) == 1:
        step = max(64, (1 << 20) // max(1, case["batch"] * case["kv_heads"]))
        for start in range(0, lengths[0], step):
            yield 0, case["batch"], min(step, lengths[0] - start)
        return
    for start in range(0, max(lengths), 4096):  # the rows of a ragged batch grow side by side
        for row, length in enumerate(lengths):
            if start < length:
                yield row, 1, min(4096, length - start)


def _config(case: dict):
    return anna_b200.KVCacheConfig(num_hidden_layers=1, cache_block_size=case["page"])


def _new_cache(case: dict, batch: int, allocator=None):
    return anna_b200.Qwen3DynamicCache(_config(case), allocator=allocator, batch_size=batch,
                                       kv_cache_quantization="turboquant", kv_cache_quant_bits=case["bits"],
                                       kv_cache_residual_len=case["window"])


def _query(case: dict, gen: torch.Generator):
    shape = (case["batch"], case["q_heads"], 1, case["dim"])
    q = _randn(gen, shape, DTYPES[case["dtype"]])
    return q, _randn(gen, shape, DTYPES[case["dtype"]]) if case["gate"] else None


def _paged_inputs(case: dict, seed: int) -> dict:
    gen = _generator(seed)
    lengths, page = _lengths(case), case["page"]
    blocks = [(n + page - 1) // page for n in lengths]
    pool = sum(blocks) + 8
    shape = (pool, case["kv_heads"], page, case["dim"])
    keys, values = _randn(gen, shape, DTYPES[case["dtype"]]), _randn(gen, shape, DTYPES[case["dtype"]])
    order = torch.rand(pool, generator=gen, device="cuda").argsort().to(torch.int32)
    table = torch.full((case["batch"], max(blocks)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for row, n in enumerate(blocks):
        table[row, :n] = order[at:at + n]
        at += n
    q, gate = _query(case, gen)
    return dict(query=q, key_pages=keys, value_pages=values, page_table=table,
                visible_lengths=torch.tensor(lengths, dtype=torch.long, device="cuda"), gate=gate)


def _prefill_inputs(case: dict, seed: int) -> dict:
    gen, dtype = _generator(seed), DTYPES[case["dtype"]]
    batch, dim, total = case["batch"], case["dim"], case["past"] + case["chunk"]
    q = _randn(gen, (batch, case["q_heads"], case["chunk"], dim), dtype)
    k = _randn(gen, (batch, case["kv_heads"], total, dim), dtype)
    v = _randn(gen, (batch, case["kv_heads"], total, dim), dtype)
    lengths = [total - (case["past"] * row // (2 * batch) if case["ragged"] else 0) for row in range(batch)]
    return dict(q=q, k=k, v=v, lengths=torch.tensor(lengths, dtype=torch.long, device="cuda"))


def _request_inputs(case: dict, seed: int) -> dict:
    """Keys and values (and queries) of a prompt and, for ``generate``, of the tokens after it."""
    gen = _generator(seed)
    total = case["tokens"] + case.get("steps", 0)
    k, v = _kv(case, gen, _channels(case, gen), case["batch"], total)
    if case["kind"] == "admit":
        return dict(k=k, v=v)
    return dict(k=k, v=v, q=_randn(gen, (case["batch"], case["q_heads"], total, case["dim"]), DTYPES[case["dtype"]]))


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "paged_decode":
        return dict(case=case, **_paged_inputs(case, seed))
    if kind == "prefill":
        return dict(case=case, **_prefill_inputs(case, seed))
    if kind == "tq_decode":
        gen = _generator(seed)
        factors = _channels(case, gen)
        ragged = len(set(_lengths(case))) > 1
        allocator = anna_b200.Qwen3PageAllocator(_config(case))
        caches = ([_new_cache(case, 1, allocator) for _ in range(case["batch"])] if ragged
                  else [_new_cache(case, case["batch"], allocator)])
        for row, rows, tokens in _pieces(case):
            k, v = _kv(case, gen, factors, rows, tokens)
            caches[row].update(k, v, 0, require_dense_cache=False)
        cache = (anna_b200.Qwen3DynamicCache.stack(caches, _config(case), clone_turboquant_rows=False) if ragged
                 else caches[0])
        q, gate = _query(case, gen)
        return dict(case=case, cache=cache, q=q, gate=gate)
    # an engine's allocator outlives the requests: its pool has held such a request before, and is blank here
    allocator = anna_b200.Qwen3PageAllocator(_config(case))
    inputs = _request_inputs(case, seed)
    before = _new_cache(case, case["batch"], allocator)
    before.update(inputs["k"], inputs["v"], 0, require_dense_cache=False)
    before.release()
    pool = allocator.turboquant_layers[0]
    pool.window.zero_()
    if pool.packed_pages is not None:
        pool.packed_pages.zero_()
    return dict(case=case, allocator=allocator, **inputs)


# ---------------------------------------------------------------------------------------------------------------
# one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    scaling = case["dim"] ** -0.5
    if kind == "tq_decode":
        return state["cache"].turboquant_single_token_decode_attention(
            0, state["q"], scaling=scaling, num_key_value_groups=case["q_heads"] // case["kv_heads"],
            gate=state["gate"])
    if kind == "paged_decode":
        return anna_b200.run_paged_gqa_decode_fused(
            query=state["query"], key_pages=state["key_pages"], value_pages=state["value_pages"],
            page_table=state["page_table"], visible_lengths=state["visible_lengths"], scaling=scaling,
            gate=state["gate"])
    if kind == "prefill":
        return anna_b200.grouped_query_attention(state["q"], state["k"], state["v"], scaling=scaling,
                                                 key_lengths=state["lengths"], causal=True)
    k, v = state["k"], state["v"]
    cache = _new_cache(case, case["batch"], state["allocator"])
    if kind == "admit":
        cache.update(k, v, 0, require_dense_cache=False)
        cache.release()
        pool = state["allocator"].turboquant_layers[0]
        return pool.packed_pages, pool.window
    q, outputs = state["q"], []
    tokens = case["tokens"]
    chunk = case.get("chunk", tokens)
    for start in range(0, tokens, chunk):
        end = min(tokens, start + chunk)
        keys, values, _ = cache.update(k[:, :, start:end], v[:, :, start:end], 0, require_dense_cache=True)
        outputs.append(anna_b200.grouped_query_attention(q[:, :, start:end], keys, values, scaling=scaling, causal=True))
    for at in range(tokens, tokens + case.get("steps", 0)):
        cache.update(k[:, :, at:at + 1], v[:, :, at:at + 1], 0, require_dense_cache=False)
        outputs.append(cache.turboquant_single_token_decode_attention(
            0, q[:, :, at:at + 1], scaling=scaling, num_key_value_groups=case["q_heads"] // case["kv_heads"]))
    cache.release()
    return outputs


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without


def _packed_bytes(case: dict) -> int:
    """Bytes of one packed token of one KV head: key codes, two norms, value codes, scales and zeros."""
    dim, bits = case["dim"], case["bits"]
    return dim * bits // 8 + 8 + dim // (4 if bits == 2 else 2) + 2 * (dim // 32) * ELEM[case["dtype"]]


def _decode_work(case: dict, lengths: list[int]) -> dict:
    elem, dim = ELEM[case["dtype"]], case["dim"]
    vectors = 2 + bool(case.get("gate"))
    total = len(lengths) * case["q_heads"] * dim * elem * vectors
    for n in lengths:
        packed = max(0, n - case["window"]) if "bits" in case else 0
        total += case["kv_heads"] * (n - packed) * 2 * dim * elem
        if packed:
            total += case["kv_heads"] * packed * _packed_bytes(case)
    return dict(bytes=total, flops=4 * dim * case["q_heads"] * sum(lengths))


def _causal_pairs(chunk: int, length: int) -> int:
    return chunk * (length - chunk) + chunk * (chunk + 1) // 2


def work(case: dict) -> dict:
    kind, elem, dim = case["kind"], ELEM[case["dtype"]], case["dim"]
    if kind in ("tq_decode", "paged_decode"):
        return _decode_work(case, _lengths(case))
    batch, kv_heads = case["batch"], case["kv_heads"]
    if kind == "prefill":
        total = case["past"] + case["chunk"]
        lengths = [total - (case["past"] * row // (2 * batch) if case["ragged"] else 0) for row in range(batch)]
        return dict(bytes=2 * dim * elem * (kv_heads * sum(lengths) + batch * case["q_heads"] * case["chunk"]),
                    flops=4 * dim * case["q_heads"] * sum(_causal_pairs(case["chunk"], n) for n in lengths))
    tokens, window = case["tokens"], case["window"]
    append = batch * kv_heads * (tokens * 2 * dim * elem + max(0, tokens - window) * _packed_bytes(case)
                                 + min(tokens, window) * 2 * dim * elem)
    transforms = batch * kv_heads * tokens * 2 * dim * int(math.log2(dim))
    if kind == "admit":
        return dict(bytes=append, flops=transforms)
    total, flops = append, transforms
    chunk = case.get("chunk", tokens)
    for start in range(0, tokens, chunk):
        end = min(tokens, start + chunk)
        packed = max(0, end - window)
        total += batch * kv_heads * (packed * _packed_bytes(case) + (end - packed) * 2 * dim * elem)
        total += 2 * batch * case["q_heads"] * (end - start) * dim * elem
        flops += 4 * dim * batch * case["q_heads"] * _causal_pairs(end - start, end)
    for at in range(tokens, tokens + case.get("steps", 0)):
        one = _decode_work(case, [at + 1] * batch)
        total += one["bytes"] + batch * kv_heads * (4 * dim * elem + (_packed_bytes(case) if at >= window else 0))
        flops += one["flops"] + batch * kv_heads * 2 * dim * int(math.log2(dim))
    return dict(bytes=total, flops=flops)


def tolerance(case: dict):
    """Codes and copies are the same bytes.  16-bit outputs carry their own rounding (2^-9 relative in bf16, 2^-12 in fp16)
    and that of 16-bit probabilities and values inside; scores of quantized keys add the rounding of rotated queries and
    centroids to a few bytes, dense views of them one more rounding to 16 bits.  Measured against 64 bits: up to 3.2e-3
    (bf16), 2.4e-3 (fp16, quantized), 2.5e-4 (fp16), 8e-7 (fp32)."""
    if case["kind"] == "admit":
        return "exact"
    if case["dtype"] == "fp32":
        rel = 5e-6
    elif case["dtype"] == "bf16" or "bits" in case:
        rel = 1e-2
    else:
        rel = 1.5e-3
    return {"rel": rel, "max": 20 * rel}


# ---------------------------------------------------------------------------------------------------------------
# the same in 64 bits


def _signs(dim: int, stream: int) -> torch.Tensor:
    mask = (1 << 64) - 1
    x = (42 ^ ((0xD1B54A32D192ED03 * (stream + 1)) & mask) ^ ((dim * 0x9E3779B97F4A7C15) & mask)) & mask
    out = []
    for _ in range(dim):
        x = (x + 0x9E3779B97F4A7C15) & mask
        z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        out.append(-1.0 if ((z ^ (z >> 31)) >> 63) else 1.0)
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _codebook(dim: int, index_bits: int) -> tuple[torch.Tensor, torch.Tensor]:
    tables = json.loads(Path("anna_b200/data/tq_codebooks.json").read_text())["tables"][f"d{dim}_m{index_bits}"]
    return tuple(torch.tensor([struct.unpack(">f", bytes.fromhex(h))[0] for h in tables[name]], dtype=torch.float64,
                              device="cuda") for name in ("centroids", "boundaries"))


def _fwht(x: torch.Tensor) -> torch.Tensor:
    dim = x.shape[-1]
    shape, step = x.shape, 1
    while step < dim:
        x = x.reshape(*shape[:-1], dim // (2 * step), 2, step)
        x = torch.stack((x[..., 0, :] + x[..., 1, :], x[..., 0, :] - x[..., 1, :]), dim=-2).reshape(shape)
        step *= 2
    return x


def _exact_keys(x: torch.Tensor, bits: int) -> torch.Tensor:
    """Keys [..., D] as the quantizer represents them: Lloyd-Max indices of the rotated unit vector plus the signs and
    the norm of the projected residual."""
    dim = x.shape[-1]
    s1, s2 = _signs(dim, 0), _signs(dim, 1)
    centroids, boundaries = _codebook(dim, bits - 1)
    x = x.double()
    norm = x.norm(dim=-1, keepdim=True)
    w = _fwht(s1 * x) / norm.clamp(min=1e-20)
    c = centroids[torch.bucketize(w, boundaries)]
    e = w - c
    rnorm = e.norm(dim=-1, keepdim=True) / math.sqrt(dim)
    sign = torch.where(_fwht(s2 * e) >= 0, 1.0, -1.0).double()
    return norm / dim * s1 * _fwht(c + math.sqrt(math.pi / 2 / dim) * rnorm * s2 * _fwht(sign))


def _exact_values(x: torch.Tensor, bits: int) -> torch.Tensor:
    """Values [..., D] as the quantizer represents them: groups of 32, scale and zero point held in the cache's type."""
    groups = x.unflatten(-1, (-1, 32))
    low = groups.amin(dim=-1, keepdim=True)
    span = (groups.amax(dim=-1, keepdim=True).float() - low.float()) / (2 ** bits - 1)
    scale = span.clamp(min=1e-8).to(x.dtype).double()
    code = ((groups.double() - low.double()) / scale).round().clamp(0, 2 ** bits - 1)
    return (code * scale + low.double()).flatten(-2)


def _quantized(case: dict, k: torch.Tensor, v: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """[B, H, T, D] keys and values after quantization, in pieces that bound the memory taken."""
    rows = max(1, KEYS_AT_ONCE // max(1, k.shape[1] * k.shape[2]))
    k_hat = torch.cat([_exact_keys(x, case["bits"]) for x in k.split(rows)])
    v_hat = torch.cat([_exact_values(x, case["bits"]) for x in v.split(rows)])
    return k_hat, v_hat


def _attend(q, k, v, scaling: float, gate=None, allowed=None):
    """q [Hq, T, D], k / v [Hkv, L, D] in 64 bits; allowed [T, L]."""
    heads, kv_heads = q.shape[0], k.shape[0]
    q = q.double().unflatten(0, (kv_heads, heads // kv_heads))
    scores = torch.einsum("hgtd,hld->hgtl", q, k.double()) * scaling
    if allowed is not None:
        scores = scores.masked_fill(~allowed, -math.inf)
    out = torch.einsum("hgtl,hld->hgtd", scores.softmax(dim=-1), v.double()).flatten(0, 1)
    return out if gate is None else out * torch.sigmoid(gate.double())


def _causal(length: int, chunk: int) -> torch.Tensor:
    return (torch.arange(length, device="cuda")[None, :]
            <= torch.arange(length - chunk, length, device="cuda")[:, None])


def _exact_tq_decode(case: dict, seed: int):
    gen = _generator(seed)
    factors = _channels(case, gen)
    lengths = _lengths(case)
    # Only running sums are kept while the context streams by, so the queries, which come last from the generator, are
    # drawn first from a copy of it that has seen the whole context.
    ahead = _generator(seed)
    _channels(case, ahead)
    for _, rows, tokens in _pieces(case):
        _kv(case, ahead, factors, rows, tokens)
    q, gate = _query(case, ahead)
    batch, kv_heads, dim = case["batch"], case["kv_heads"], case["dim"]
    qd = q[:, :, 0].double().unflatten(1, (kv_heads, -1)) * dim ** -0.5  # [B, Hkv, G, D]
    best = torch.full(qd.shape[:3], -math.inf, dtype=torch.float64, device="cuda")
    total = torch.zeros_like(best)
    out = torch.zeros_like(qd)
    seen = [0] * batch
    for row, rows, tokens in _pieces(case):
        k, v = _kv(case, gen, factors, rows, tokens)
        packed = max(0, min(tokens, lengths[row] - case["window"] - seen[row]))
        for r in range(rows):
            one_k, one_v = k[r].double(), v[r].double()
            if packed:
                one_k[:, :packed] = _exact_keys(k[r, :, :packed], case["bits"])
                one_v[:, :packed] = _exact_values(v[r, :, :packed], case["bits"])
            at = row + r
            scores = qd[at] @ one_k.transpose(1, 2)
            top = torch.maximum(best[at], scores.amax(dim=-1))
            p = torch.exp(scores - top[..., None])
            keep = torch.exp(best[at] - top)
            total[at] = total[at] * keep + p.sum(dim=-1)
            out[at] = out[at] * keep[..., None] + p @ one_v
            best[at] = top
            seen[at] += tokens
    out = (out / total[..., None]).flatten(1, 2)[:, :, None]
    return out if gate is None else out * torch.sigmoid(gate.double())


def _exact_request(case: dict, seed: int):
    inputs = _request_inputs(case, seed)
    k, v, q = inputs["k"], inputs["v"], inputs["q"]
    k_hat, v_hat = _quantized(case, k, v)
    scaling, window, tokens = case["dim"] ** -0.5, case["window"], case["tokens"]
    chunk = case.get("chunk", tokens)
    spans = [(start, min(tokens, start + chunk)) for start in range(0, tokens, chunk)]
    spans += [(at, at + 1) for at in range(tokens, tokens + case.get("steps", 0))]
    outputs = []
    for start, end in spans:
        packed = max(0, end - window)
        allowed = _causal(end, end - start)
        outputs.append(torch.stack([
            _attend(q[b, :, start:end], torch.cat((k_hat[b, :, :packed], k[b, :, packed:end].double()), dim=1),
                    torch.cat((v_hat[b, :, :packed], v[b, :, packed:end].double()), dim=1), scaling, allowed=allowed)
            for b in range(case["batch"])]))
    return outputs


def exact(case: dict, seed: int):
    kind, scaling = case["kind"], case["dim"] ** -0.5
    if kind == "admit":
        return None
    if kind == "tq_decode":
        return _exact_tq_decode(case, seed)
    if kind == "paged_decode":
        x = _paged_inputs(case, seed)
        rows = []
        for b, n in enumerate(_lengths(case)):
            pages = x["page_table"][b, :(n + case["page"] - 1) // case["page"]].long()
            k, v = (x[name][pages].transpose(0, 1).flatten(1, 2)[:, :n] for name in ("key_pages", "value_pages"))
            rows.append(_attend(x["query"][b], k, v, scaling, None if x["gate"] is None else x["gate"][b]))
        return torch.stack(rows)
    if kind == "prefill":
        x = _prefill_inputs(case, seed)
        chunk, piece = case["chunk"], 256
        rows = []
        for b, n in enumerate(x["lengths"].tolist()):
            allowed = _causal(n, chunk)
            rows.append(torch.cat([_attend(x["q"][b, :, t:t + piece], x["k"][b, :, :n], x["v"][b, :, :n], scaling,
                                           allowed=allowed[t:t + piece]) for t in range(0, chunk, piece)], dim=1))
        return torch.stack(rows)
    return _exact_request(case, seed)
