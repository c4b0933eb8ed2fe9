"""Recorded calls keep the workspace that they were recorded with when a larger call has it replaced: the replay gives what the call gave, and
memory that is handed out in between stays as it is.  (Run with the library only as it is: a replay into freed memory would be a fault.)"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tests.util import KIND_Q4_K, KIND_Q6_K, random_blocks

pytestmark = pytest.mark.gpu


def _context(torch):
    from marmot_b200 import Context

    ctx = Context(0, use_torch_stream=False)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    return ctx, stream


def _canaries(torch, ctx, sizes):
    """Allocations of the sizes that a freed workspace would leave room for, filled with a pattern."""
    kept = []
    for size in sizes:
        p = C.c_void_p()
        ctx._check(ctx.lib.mcu_malloc(ctx.handle, C.c_size_t(size), C.byref(p)))
        pattern = np.full(size, 0xA5, dtype=np.uint8)
        ctx._check(ctx.lib.mcu_memcpy_to_device(ctx.handle, p, C.c_void_p(pattern.ctypes.data), C.c_size_t(size)))
        kept.append((p, pattern))
    return kept


def _untouched(ctx, kept):
    for p, pattern in kept:
        back = np.empty_like(pattern)
        ctx._check(ctx.lib.mcu_memcpy_to_host(ctx.handle, C.c_void_p(back.ctypes.data), p, C.c_size_t(back.size)))
        ctx._check(ctx.lib.mcu_free(ctx.handle, p))
        if not np.array_equal(back, pattern):
            return False
    return True


# recorded: (kind, T, K, F); larger: the call that replaces the buffer.  The integer kernel behind a call of four tokens, the mma.sync one, the
# fp16 one, a call without a kernel that streams (packed activations).
@pytest.mark.parametrize("capture", ["library", "torch"])
@pytest.mark.parametrize("recorded,larger", [((KIND_Q4_K, 8, 2048, 2048), (KIND_Q6_K, 4, 14336, 4096)), ((KIND_Q4_K, 9, 1024, 8192), (KIND_Q4_K, 16, 8192, 256)),
                                             ((KIND_Q4_K, 64, 1024, 256), (KIND_Q4_K, 512, 4096, 256)), ((KIND_Q6_K, 2, 1280, 300), (KIND_Q4_K, 16, 8192, 256))])
def test_replay_behind_a_larger_call(recorded, larger, capture):
    import torch

    kind, T, K, F = recorded
    rng = np.random.default_rng(T + K)
    ctx, stream = _context(torch)
    x = torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda()
    w = ctx.upload(random_blocks(kind, F, K, rng))
    x2 = torch.from_numpy(rng.normal(0, 1, (larger[1], larger[2])).astype(np.float32)).cuda()
    w2 = ctx.upload(random_blocks(larger[0], larger[3], larger[2], rng))
    out = torch.zeros((T, F), device="cuda")
    torch.cuda.synchronize()
    ctx.linear(kind, x, w, F, out=out)
    ctx.synchronize()
    first = out.cpu().numpy()
    if capture == "library":
        ctx.graph_capture_begin()
        ctx.linear(kind, x, w, F, out=out)
        graph = ctx.graph_capture_end()
        replay = graph.launch
    else:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.linear(kind, x, w, F, out=out)
        replay = lambda: _on(torch, stream, graph)
    ctx.linear(larger[0], x2, w2, larger[3])
    ctx.synchronize()
    kept = _canaries(torch, ctx, [256 << s for s in range(12)] * 2)
    out.zero_()
    torch.cuda.synchronize()
    replay()
    ctx.synchronize()
    again = out.cpu().numpy()
    assert _untouched(ctx, kept)
    assert np.array_equal(again, first)
    if capture == "library":
        graph.close()
    del replay, graph
    ctx.close()


def _on(torch, stream, graph):
    with torch.cuda.stream(stream):
        graph.replay()


def test_outgrown_workspace_is_given_back_behind_its_graph():
    import torch

    ctx, _ = _context(torch)
    rng = np.random.default_rng(1)
    K, F = 14336, 64
    w = ctx.upload(random_blocks(KIND_Q4_K, F, K, rng))
    x = torch.zeros((3072, K), device="cuda")
    out = torch.zeros((3072, F), device="cuda")
    torch.cuda.synchronize()

    def call(T):
        ctx.linear(KIND_Q4_K, x[:T], w, F, out=out[:T])
        ctx.synchronize()

    used = lambda: -torch.cuda.mem_get_info()[0]
    call(1024)
    before = used()
    ctx.graph_capture_begin()
    ctx.linear(KIND_Q4_K, x[:1024], w, F, out=out[:1024])
    graph = ctx.graph_capture_end()
    call(2048)
    assert used() - before >= 2 * 2048 * K - (4 << 20)  # the first rows are still there
    graph.launch()
    ctx.synchronize()
    graph.close()
    call(3072)
    assert used() - before <= 2 * 2048 * K + (24 << 20)  # 3072 rows in the place of 1024, and nothing else
    ctx.close()
