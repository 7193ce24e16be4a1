"""GPU: decode steps that go on from the previous one, with the rows changed in every other way in between.

A quantized layer keeps the device table, lengths and ring slots of its last step; whatever happens to its rows or pages
outside that sequence has to be seen by the next append and decode."""
from __future__ import annotations

import pytest
import torch

from anna_b200 import KVCacheConfig, Qwen3DynamicCache
from tests.helpers import TQ_ATOL
from tests.test_gpu_tq_decode_schedules import dense_attention

pytestmark = pytest.mark.gpu
HEADS, DIM, WINDOW, PAGE = 2, 128, 16, 16


class Steps:
    def __init__(self, batch: int) -> None:
        self.device, self.dtype = torch.device("cuda", torch.cuda.current_device()), torch.bfloat16
        self.gen = torch.Generator(device=self.device).manual_seed(7)
        self.config = KVCacheConfig(num_hidden_layers=1, cache_block_size=PAGE)
        self.cache = Qwen3DynamicCache(self.config, batch_size=batch, kv_cache_quantization="turboquant",
                                       kv_cache_quant_bits=4, kv_cache_residual_len=WINDOW)

    def kv(self, batch: int, tokens: int):
        shape = (batch, HEADS, tokens, DIM)
        return [torch.randn(shape, generator=self.gen, device=self.device).to(self.dtype) for _ in range(2)]

    def append(self, cache, tokens: int) -> None:
        before = list(cache.layer_lengths[0])
        _, _, past = cache.update(*self.kv(cache.get_batch_size(), tokens), 0, require_dense_cache=False)
        assert past.tolist() == before

    def check(self, cache) -> None:
        lengths = [row.length for row in cache.turboquant_rows[0]]
        query = torch.randn((len(lengths), 4 * HEADS, 1, DIM), generator=self.gen, device=self.device).to(self.dtype)
        for _ in range(2):
            out = cache.turboquant_single_token_decode_attention(0, query, scaling=0.1, num_key_value_groups=4)
            cache.layer_lengths[0][:] = lengths  # the dense view goes by these
            torch.testing.assert_close(out.double(), dense_attention(cache, query, lengths, 0.1),
                                       atol=TQ_ATOL[self.dtype], rtol=TQ_ATOL[self.dtype])


def test_steps_across_pages_and_multi_token_appends():
    s = Steps(3)
    for tokens in (5, 1, 1, 30, 1, 17, 1, 1) + (1,) * 20:
        s.append(s.cache, tokens)
        s.check(s.cache)


def test_clone_row_append_and_restack_between_steps():
    s = Steps(2)
    s.append(s.cache, 70)
    s.append(s.cache, 1)
    s.check(s.cache)
    clone = s.cache.clone()                      # shares pages: the next appends copy the partly filled ones
    for _ in range(3):
        s.append(s.cache, 1)
        s.append(clone, 1)
        s.check(s.cache)
        s.check(clone)
    k, v = s.kv(1, 1)
    s.cache.turboquant_rows[0][1].append(k[0], v[0])   # one row grows behind the cache's back
    s.check(s.cache)
    clone.release()
    s.check(s.cache)
    parts = s.cache.split_batch(clone_turboquant_rows=False)
    s.append(parts[0], 1)                        # the same row objects through another cache
    s.check(s.cache)
    stacked = Qwen3DynamicCache.stack(parts, s.config, clone_turboquant_rows=False)
    for _ in range(PAGE + 2):
        s.append(stacked, 1)
        s.check(stacked)


def test_graph_of_a_decode_outlives_the_step_it_was_captured_from():
    """A re-stacked batch has no lengths on the device yet; a capture reads those that an earlier decode uploaded, on
    whichever stream, and they stay alive when the cache's step moves on."""
    s = Steps(3)
    s.append(s.cache, 70)
    stacked = Qwen3DynamicCache.stack(s.cache.split_batch(clone_turboquant_rows=False), s.config, clone_turboquant_rows=False)
    query = torch.randn((3, 4 * HEADS, 1, DIM), generator=s.gen, device=s.device).to(s.dtype)

    def decode():
        return stacked.turboquant_single_token_decode_attention(0, query, scaling=0.1, num_key_value_groups=4)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        decode()                                 # this stream's scratch exists before the capture
    torch.cuda.synchronize()
    want = decode()                              # the step is the default stream's now
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = decode()
    stacked.turboquant_rows[0][0]._length = 70   # counts as a change: the next decode uploads anew and the old step goes
    again = decode()
    junk = [torch.zeros(64, dtype=torch.int64, device=s.device) for _ in range(64)]  # would take freed memory
    captured.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, want) and torch.equal(again, want) and len(junk) == 64
