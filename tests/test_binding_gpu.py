"""Context.linear through the native binding gives what the ctypes call gives: results, given outputs, row strides, bias, errors."""
from __future__ import annotations

import numpy as np
import pytest

from tests.util import KIND_Q4_K, KIND_Q8_0, random_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,T,K,F", [(KIND_Q4_K, 1, 2048, 256), (KIND_Q4_K, 3, 300, 1), (KIND_Q8_0, 9, 96, 70)])
def test_native_call_equals_ctypes(kind, T, K, F):
    import torch
    from marmot_b200 import Context, MarmotCudaError
    from marmot_b200.runtime import load_binding

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert load_binding()
    ctx, plain = Context(0), Context(0)
    plain._linear = None
    rng = np.random.default_rng(K)
    w = ctx.upload(random_blocks(kind, F, K, rng))
    x = torch.from_numpy(rng.normal(0, 1, (T, K + 4)).astype(np.float32)).cuda()[:, :K]
    bias = torch.from_numpy(rng.normal(0, 1, F).astype(np.float32)).cuda()
    want = plain.linear(kind, x, w, F, bias=bias)
    got = ctx.linear(kind, x, w, F, bias=bias)
    assert got.dtype == torch.float32 and torch.equal(got, want)
    wide = torch.zeros((T, F + 3), device="cuda")
    assert ctx.linear(kind, x, w, F, bias=bias, out=wide[:, :F]).data_ptr() == wide.data_ptr()
    assert torch.equal(wide[:, :F], want) and not wide[:, F:].any()
    for c in (ctx, plain):
        with pytest.raises(AssertionError):
            c.linear(kind, x, w, F + 1)  # more rows than the matrix has
        with pytest.raises(MarmotCudaError):
            c.linear(kind, x, w, F, out=torch.zeros((T, F), device="cuda").expand(T, F)[:, :0])  # rows shorter than F
        c.synchronize()
        c.close()
        with pytest.raises(MarmotCudaError):
            c.linear(kind, x, w, F)


def test_errors_are_those_of_the_ctypes_call():
    """Out of memory and sizes beyond the library's limits come as the same exceptions."""
    import torch
    from marmot_b200 import Context

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx, plain = Context(0), Context(0)
    plain._linear = None
    rows = 1 << 20
    w, x = torch.zeros(rows * 34, dtype=torch.uint8, device="cuda"), torch.zeros((rows, 32), device="cuda")
    for c in (ctx, plain):
        with pytest.raises(torch.OutOfMemoryError):
            c.linear(KIND_Q8_0, x, w, rows)  # a result of four terabytes
        with pytest.raises(AssertionError):
            c.linear(KIND_Q8_0, x[:1], w, 1 << 62, out=torch.zeros((1, 4), device="cuda"))  # rows x bytes overflows 64 bits
        c.close()
