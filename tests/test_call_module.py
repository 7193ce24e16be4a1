"""The call module (csrc/launch_module.cpp): which calls it takes and which it declines, and that those it takes give what the
general path gives."""
from __future__ import annotations

import sys
import threading
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from anna_b200 import KVCacheConfig, Qwen3DynamicCache, _lib, attention, fused_ops, turboquant


class Declining:
    """The module with its calls declined, so that the general path runs."""

    def __getattr__(self, name):
        return lambda *args: None


def install(monkeypatch, module):
    monkeypatch.setattr(fused_ops, "_LAUNCH", module)
    for caller in (attention, turboquant):
        monkeypatch.setattr(caller, "launch_module", lambda: module)


def general(monkeypatch):
    install(monkeypatch, Declining())


def rows_contiguous(*tensors):
    return all(t is None or t.stride(-1) == 1 for t in tensors)


# what the module takes of the calls in these tests, by the layouts of their arguments
SERVED = {
    "paged_decode": lambda query, keys, values, table, lengths, scaling, gate: rows_contiguous(query, table, lengths, gate),
    "prefill": lambda query, keys, values, lengths, scaling, causal: (
        rows_contiguous(query, keys, values) and keys.stride() == values.stride()
        and all(stride % 8 == 0 for t in (query, keys) for stride in t.stride()[:3])),
    "tq_append": lambda keys, values, *rest: rows_contiguous(keys) and keys.stride() == values.stride(),
    "tq_decode": lambda query, gate, *rest: rows_contiguous(query, gate),
}


class Watched:
    """The module; notes of every call whether it was taken, and that this is what SERVED says."""

    def __init__(self):
        self.module, self.taken = _lib.launch(), {name: [] for name in SERVED}

    def __getattr__(self, name):
        call = getattr(self.module, name)
        if name not in SERVED:
            return call

        def watched(*args):
            result = call(*args)
            assert (result is not None) == SERVED[name](*args), name
            self.taken[name].append(result is not None)
            return result

        return watched


@pytest.fixture
def watched(monkeypatch):
    fused_ops.launch_module()
    module = Watched()
    install(monkeypatch, module)
    return module


def test_cpu_tensors_and_other_objects_are_declined():
    module = _lib.launch()
    x = torch.zeros(1, 2, 1, 64)
    pages, table, one = torch.zeros(1, 2, 16, 64), torch.zeros(1, 1, dtype=torch.int32), torch.ones(1, dtype=torch.long)
    assert module.paged_decode(x, pages, pages, table, one, 1.0, None) is None
    assert module.paged_decode(x, pages, pages, table, [1], 1.0, None) is None
    assert module.prefill(x, pages, pages, None, 1.0, True) is None
    assert module.prefill("q", pages, pages, None, 1.0, True) is None
    window = torch.zeros(1, 2, 2, 8, 64)
    assert module.tq_decode(x, None, None, None, window, one, one, x, x, x, 1.0, 2, 16, 8, 4, 32, 0) is None
    assert module.tq_append(x, x, None, None, window, one, one, None, x, x, x, x, None, 16, 8, 4, 32, 0) is None
    with pytest.raises(TypeError):
        module.tq_decode(x)
    with pytest.raises(TypeError):
        module.paged_decode(x, pages, pages, table, one, "scale", None)


@pytest.mark.parametrize("changed", ["torch", "python"])
def test_module_of_other_versions_is_rebuilt_and_not_loaded(monkeypatch, changed):
    """The module reads tensors and objects by the layout of the headers that it was compiled with."""
    from anna_b200 import build

    compiled = []
    monkeypatch.setattr(build.subprocess, "run",
                        lambda cmd, **kw: compiled.append(cmd) or SimpleNamespace(returncode=1, stderr="", stdout=""))
    _lib.launch()
    build.build_module()
    assert not compiled
    if changed == "torch":
        monkeypatch.setattr(torch, "__version__", "2.99.0")
    else:
        monkeypatch.setattr(sys.implementation, "cache_tag", "cpython-399")
    with pytest.raises(RuntimeError, match="launch_module.cpp failed"):
        build.build_module()
    assert len(compiled) == 1
    monkeypatch.setattr(_lib, "_LAUNCH", None)
    with pytest.raises(RuntimeError, match="was built for"):
        _lib.launch()


def strided(shape, dtype, device, gen, order):
    """A tensor of `shape` whose dims lie in memory in `order` (outermost first)."""
    x = torch.randn([shape[d] for d in order], generator=gen, device=device).to(dtype)
    return x.permute([order.index(d) for d in range(len(shape))])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("gate", [None, "4d", "4d_strided", "3d", "3d_strided"])
def test_paged_decode_equals_general_path(cuda_device, watched, dtype, gate):
    gen = torch.Generator(device=cuda_device).manual_seed(1)
    batch, heads, kv_heads, dim, page = 3, 8, 2, 128, 16
    for order in ((0, 1, 2, 3), (1, 0, 2, 3), (2, 0, 1, 3), (0, 1, 3, 2), (3, 0, 1, 2)):
        query = strided((batch, heads, 1, dim), dtype, cuda_device, gen, order)
        keys, values = (torch.randn(40, kv_heads, page, dim, generator=gen, device=cuda_device).to(dtype) for _ in range(2))
        table = torch.randperm(36, generator=gen, device=cuda_device).to(torch.int32).view(3, 12)
        lengths = torch.tensor([5, 170, 100], device=cuda_device)
        g = None
        if gate is not None:
            g = strided((batch, heads, 1, dim), dtype, cuda_device, gen, order if "strided" in gate else (0, 1, 2, 3))
            if gate.startswith("3d"):
                g = strided((batch, 1, heads * dim), dtype, cuda_device, gen, (2, 1, 0) if "strided" in gate else (0, 1, 2))
        for tab, visible in ((table, lengths), (table.t().contiguous().t(), lengths.repeat_interleave(2)[::2]),
                             (table[:, :11], lengths)):
            args = dict(query=query, key_pages=keys, value_pages=values, page_table=tab, visible_lengths=visible,
                        scaling=0.1, gate=g)
            out = fused_ops.run_paged_gqa_decode_fused(**args)
            with pytest.MonkeyPatch.context() as patch:
                general(patch)
                assert torch.equal(out, fused_ops.run_paged_gqa_decode_fused(**args))
            assert out.is_contiguous() and out.shape == query.shape and out.dtype == dtype
    taken = watched.taken["paged_decode"]
    assert len(taken) == 15 and taken.count(True) == (0 if gate == "3d_strided" else 8)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,query_len,key_len", [(64, 70, 200), (128, 5, 133), (256, 96, 96)])
def test_prefill_equals_general_path(cuda_device, watched, dim, query_len, key_len):
    gen = torch.Generator(device=cuda_device).manual_seed(2)
    for order in ((0, 1, 2, 3), (0, 2, 1, 3), (2, 0, 1, 3), (0, 1, 3, 2)):
        query = strided((2, 4, query_len, dim), torch.bfloat16, cuda_device, gen, order)
        keys = strided((2, 2, key_len, dim), torch.bfloat16, cuda_device, gen, order)
        for values in (strided((2, 2, key_len, dim), torch.bfloat16, cuda_device, gen, order),
                       strided((2, 2, key_len, dim), torch.bfloat16, cuda_device, gen, (1, 0, 2, 3))):
            for lengths in (None, torch.tensor([key_len, key_len - 3], device=cuda_device)):
                for causal in (None, True):
                    args = dict(scaling=0.1, key_lengths=lengths, causal=causal)
                    out = attention.grouped_query_attention(query, keys, values, **args)
                    with pytest.MonkeyPatch.context() as patch:
                        general(patch)
                        assert torch.equal(out, attention.grouped_query_attention(query, keys, values, **args))
    taken = watched.taken["prefill"]
    assert len(taken) == 32 and taken.count(True) == 12


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,dim", [(torch.bfloat16, 128), (torch.float16, 64), (torch.float32, 128)])
@pytest.mark.parametrize("gated", [False, True])
def test_cache_steps_equal_general_path(cuda_device, watched, dtype, dim, gated):
    """Prompt and decode steps over pages that run out, on two streams, with every layout of queries, keys and values."""

    def steps():
        gen = torch.Generator(device=cuda_device).manual_seed(3)
        cache = Qwen3DynamicCache(KVCacheConfig(num_hidden_layers=1, cache_block_size=16), batch_size=3,
                                  kv_cache_quantization="turboquant", kv_cache_quant_bits=3, kv_cache_residual_len=16)
        outputs = []
        for i, tokens in enumerate((40, 1, 1, 17, 1, 1, 1, 1)):
            # (the append rejects token strides that break 16-byte alignment, as those of a transposed single token do)
            order = ((0, 1, 2, 3), (0, 2, 1, 3), (2, 0, 1, 3), (0, 1, 3, 2) if tokens > 1 else (1, 0, 2, 3))[i % 4]
            k = strided((3, 2, tokens, dim), dtype, cuda_device, gen, order)
            v = strided((3, 2, tokens, dim), dtype, cuda_device, gen, order if i % 3 else (0, 1, 2, 3))
            cache.update(k, v, 0, require_dense_cache=False)
            q = strided((3, 6, 1, dim), dtype, cuda_device, gen, order)
            gate = strided((3, 6, 1, dim), dtype, cuda_device, gen, order) if gated else None
            stream = torch.cuda.Stream(cuda_device) if i == 5 else torch.cuda.current_stream(cuda_device)
            stream.wait_stream(torch.cuda.current_stream(cuda_device))
            with torch.cuda.stream(stream):
                outputs.append(cache.turboquant_single_token_decode_attention(0, q, scaling=0.1, num_key_value_groups=3,
                                                                              gate=gate))
            torch.cuda.current_stream(cuda_device).wait_stream(stream)
        return [*outputs, *cache._gather_layer_cache(0)[:2]]

    ours = steps()
    assert watched.taken["tq_decode"].count(True) >= 5 and watched.taken["tq_append"].count(True) >= 3
    with pytest.MonkeyPatch.context() as patch:
        general(patch)
        theirs = steps()
    assert all(torch.equal(a, b) for a, b in zip(ours, theirs, strict=True))


def test_uploads_of_other_rows_run_no_code_of_theirs():
    """The module reads the rows in place, so an entry whose __index__ takes rows or entries away must not run meanwhile."""
    module, ran = _lib.launch(), []

    class Shortens:
        def __init__(self, what):
            self.what = what

        def __index__(self):
            ran.append(self.what)
            self.what.clear()
            return 1

    rows = [[1, 2], [3, 4], [5, 6]]
    rows[0][1] = Shortens(rows)
    row = [1, 2, 3]
    row[0] = Shortens(row)
    for other in (rows, [row, [4, 5, 6]], [row], [[1, 2], [3]], [], [[]] * 2 + [[1]], [np.arange(3)], iter([[1]]), [[1 << 63]], [[1.0]], 7):
        assert module.upload(0, other) is None
    assert not ran and len(rows) == 3 and len(row) == 3


def test_uploads_without_the_module(monkeypatch):
    """Un-quantized pages are written by the library alone, and their lengths and tables go up without the call module."""
    def missing():
        raise RuntimeError("not built")

    monkeypatch.setattr(_lib, "launch", missing)
    uploader = fused_ops.MetadataUploader(torch.device("cpu"))
    rows = uploader.upload([[1, 2, 3], [1 << 40, 5, 6]])
    assert rows.dtype == torch.int64 and rows.tolist() == [[1, 2, 3], [1 << 40, 5, 6]]
    words = uploader.upload_i32(np.arange(6)[::2])
    assert words.dtype == torch.int32 and words.tolist() == [0, 2, 4]


@pytest.mark.gpu
def test_pages_are_written_without_the_module(cuda_device, monkeypatch):
    def missing():
        raise RuntimeError("not built")

    monkeypatch.setattr(_lib, "launch", missing)
    monkeypatch.setattr(fused_ops.MetadataUploader, "_instances", {})
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    keys, values = (torch.randn(2, 2, 41, 64, generator=gen, device=cuda_device, dtype=torch.bfloat16) for _ in range(2))
    cache = Qwen3DynamicCache(KVCacheConfig(num_hidden_layers=1, cache_block_size=16), batch_size=2)
    for at in range(0, 41, 20):
        dense = cache.update(keys[:, :, at:at + 20], values[:, :, at:at + 20], 0)
    assert torch.equal(dense[0][:, :, :41], keys) and torch.equal(dense[1][:, :, :41], values)


@pytest.mark.gpu
def test_uploads(cuda_device):
    """More uploads than the ring has buffers, behind work that keeps the copies waiting; growing ones; other integers."""
    uploader = fused_ops.MetadataUploader.for_device(torch.device(cuda_device))
    busy = torch.randn(4096, 4096, device=cuda_device)
    for _ in range(4):
        busy = busy @ busy * 1e-3
    got, want = [], []
    for i in range(40):
        rows = [[i * 7 + j for j in range(1 + i * 60)], [-(2 ** 40) - i] * (1 + i * 60)]
        got.append(uploader.upload(rows))
        want.append(torch.tensor(rows))
        words = np.arange(i * 50, i * 50 + 3000, dtype=np.int32)
        got.append(uploader.upload_i32(words))
        want.append(torch.from_numpy(words))
    # whatever numpy makes int64 of
    others = [([[np.int64(3), True]], [[3, 1]]), ([(4,)], [[4]]), (([5, 6], np.array([7, 8])), [[5, 6], [7, 8]]),
              ([[1.5, -2.5], (3, 4.0)], [[1, -2], [3, 4]]), ([[1, 2], [3]], [[1, 2], [3, 3]]), (np.arange(6).reshape(2, 3), [[0, 1, 2], [3, 4, 5]])]
    got += [uploader.upload([[]]), *(uploader.upload(rows) for rows, _ in others)]
    want += [torch.empty(1, 0, dtype=torch.int64), *(torch.tensor(rows) for _, rows in others)]
    for ours, theirs in zip(got, want, strict=True):
        assert ours.dtype == theirs.dtype and torch.equal(ours.cpu(), theirs)
    for rows in ([], [[1], [2, 3]], [["a"]], [[1 << 63]], 7):
        with pytest.raises((IndexError, ValueError, OverflowError, TypeError)):
            uploader.upload(rows)
    for values in (np.arange(5), np.arange(10, dtype=np.int32)[::2], np.array([1.5, -2.5]), np.array([True, False]), np.zeros(0, dtype=np.int64)):
        ours = uploader.upload_i32(values)
        assert ours.dtype == torch.int32 and ours.cpu().tolist() == values.astype(np.int32).tolist()
    assert _lib.launch().upload_i32(0, np.zeros(3, dtype=np.float32)) is None


@pytest.mark.gpu
def test_scratch_follows_its_buffers(cuda_device):
    """The module keeps the scratch of a problem and stream until a buffer behind it is replaced by a larger one."""
    gen = torch.Generator(device=cuda_device).manual_seed(4)
    query = torch.randn(1, 8, 1, 128, generator=gen, device=cuda_device, dtype=torch.float16)
    keys, values = (torch.randn(19, 8, 16, 128, generator=gen, device=cuda_device, dtype=torch.float16) for _ in range(2))
    args = dict(query=query, key_pages=keys, value_pages=values, scaling=0.1,
                page_table=torch.arange(19, dtype=torch.int32, device=cuda_device)[None],
                visible_lengths=torch.tensor([300], device=cuda_device))
    asked = []

    def source(*problem):
        asked.append(problem)
        return fused_ops._scratch_source(*problem)

    device, scratch = torch.device(cuda_device), fused_ops._SCRATCH
    module = fused_ops.launch_module()
    module.set_scratch_source(source)
    try:
        fused_ops._forget_scratch()
        want = fused_ops.run_paged_gqa_decode_fused(**args)
        assert len(asked) == 1
        for replace, buffers in ((scratch.get, scratch._buffers), (scratch.counters, scratch._counters),
                                 (scratch.bytes, scratch._byte_buffers)):
            assert torch.equal(fused_ops.run_paged_gqa_decode_fused(**args), want) and len(asked) == 1
            replace(device, 2 * max((buf.numel() for buf in buffers.values()), default=1 << 20) + 1)
            assert torch.equal(fused_ops.run_paged_gqa_decode_fused(**args), want) and len(asked) == 2
            assert asked.pop() == asked[0]
        stream = torch.cuda.Stream(device)
        stream.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(stream):
            out = fused_ops.run_paged_gqa_decode_fused(**args)
        torch.cuda.current_stream(device).wait_stream(stream)
        assert torch.equal(out, want) and len(asked) == 2  # its own scratch
    finally:
        module.set_scratch_source(fused_ops._scratch_source)
        fused_ops._forget_scratch()


@pytest.mark.gpu
def test_two_threads_on_one_stream(cuda_device):
    """The module gives up the interpreter lock while it launches.  Calls of two threads on one stream share its scratch: the
    launches of a call that hand it partials must not mix with the other's."""
    problems = []
    for seed, dtype in ((5, torch.bfloat16), (6, torch.bfloat16)):
        gen = torch.Generator(device=cuda_device).manual_seed(seed)
        cache = Qwen3DynamicCache(KVCacheConfig(num_hidden_layers=1, cache_block_size=16), batch_size=24,
                                  kv_cache_quantization="turboquant", kv_cache_quant_bits=4, kv_cache_residual_len=128)
        k, v = (torch.randn(24, 8, 700, 128, generator=gen, device=cuda_device).to(dtype) for _ in range(2))
        cache.update(k, v, 0, require_dense_cache=False)
        q = torch.randn(24, 32, 1, 128, generator=gen, device=cuda_device).to(dtype)

        def call(cache=cache, q=q):
            return cache.turboquant_single_token_decode_attention(0, q, scaling=0.1, num_key_value_groups=4)

        problems.append((call, call()))
    torch.cuda.synchronize(cuda_device)
    wrong = [torch.zeros((), dtype=torch.int64, device=cuda_device) for _ in problems]
    start = threading.Barrier(len(problems))
    errors = []

    def work(i):
        try:
            call, want = problems[i]
            start.wait()
            for _ in range(60):
                outputs = [call() for _ in range(20)]
                for out in outputs:
                    wrong[i].add_((out != want).any())
        except Exception as exc:  # a thread's exception is the test's
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(problems))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not errors, errors
    assert [int(count) for count in wrong] == [0, 0]


@pytest.mark.gpu
def test_uploads_under_a_capture(cuda_device):
    """A captured upload has a host copy of its own, which replays read for as long as the graph lives; the ring goes on
    without it, in sizes that it had and in larger ones."""
    uploader = fused_ops.MetadataUploader.for_device(torch.device(cuda_device))

    def capture(first, sizes):
        rows = [[list(range(first + n, first + 2 * n))] for n in sizes]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = [uploader.upload(row) for row in rows] + [uploader.upload_i32(np.array(row[0])) for row in rows]
        return graph, captured, [torch.tensor(row) for row in rows] + [torch.tensor(row[0], dtype=torch.int32) for row in rows]

    def replayed(graph, captured, want):
        for out in captured:
            out.fill_(-7)
        graph.replay()
        return all(torch.equal(out.cpu(), row) for out, row in zip(captured, want, strict=True))

    uploader.upload([[1]])
    first = capture(0, [1, 700, 5000, 20000])
    assert replayed(*first)
    for i in range(40):                                              # the ring goes round, and grows
        rows = [[i] * (1 + 900 * i)]
        assert uploader.upload(rows).cpu().tolist() == rows
    second = capture(1000, [3, 30000])
    assert replayed(*second) and replayed(*first)
    del first
    torch.cuda.synchronize()
    third = capture(5000, [1, 700, 5000, 20000])                     # may have the host copies of the first
    for i in range(20):
        assert uploader.upload([[i, -i]]).cpu().tolist() == [[i, -i]]
    assert replayed(*third) and replayed(*second)
