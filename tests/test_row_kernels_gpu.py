"""The row kernels at the edges of their batches: RMSNorm with 1, 4, 8 and 16 elements per thread and turn, and SwiGLU on both sides of the
size from which a thread takes four values."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from marmot_b200 import Context

    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 256, 257, 1024, 1025, 2048, 2049, 4096, 4097, 9000])
def test_norms(ctx, n):
    import torch

    rng = np.random.default_rng(n)
    dev = lambda *s: torch.from_numpy(rng.normal(0, 1, s).astype(np.float32)).cuda()
    x, d, w = dev(5, n), dev(5, n), dev(n)
    want = lambda v: v.double() / torch.sqrt((v.double() ** 2).mean(1, keepdim=True) + 1e-5) * (w.double() + 0.5)
    # 32-bit sums of n squares, a root, a quotient and two products: a few ulp
    close = lambda got, ref: float((got.double() - ref).abs().max()) <= 2e-6 * max(1.0, float(ref.abs().max()))
    assert close(ctx.rmsnorm(x, w, 1e-5, weight_offset=0.5), want(x))
    assert close(ctx.rmsnorm(x, w, 1e-5, residual=d, weight_offset=0.5), want(x + d))
    x_out, h = torch.empty_like(x), torch.empty_like(x)
    ctx.add_rmsnorm(x, d, w, 1e-5, x_out, h, weight_offset=0.5)
    assert torch.equal(x_out, x + d) and close(h, want(x + d))
    inplace = x.clone()
    ctx.add_rmsnorm(inplace, d, w, 1e-5, inplace, h, weight_offset=0.5)
    assert torch.equal(inplace, x_out) and close(h, want(x_out))
    ctx.synchronize()


@pytest.mark.parametrize("n", [1, 196604, 196607, 196608, 196609, 196612])
@pytest.mark.parametrize("offset", [0, 1])
def test_swiglu(ctx, n, offset):
    import torch

    rng = np.random.default_rng(n)
    g, u = (torch.from_numpy(rng.normal(0, 2, n + offset).astype(np.float32)).cuda()[offset:].view(1, n) for _ in range(2))
    out = torch.zeros(n + offset + 8, device="cuda")[offset:offset + n].view(1, n)
    ctx.swiglu(g, u, out=out)
    ctx.synchronize()
    want = g.double() / (1 + torch.exp(-g.double())) * u.double()
    assert float((out.double() - want).abs().max()) <= 1e-6 * float(want.abs().max())
    assert not out._base[offset + n:].any()
