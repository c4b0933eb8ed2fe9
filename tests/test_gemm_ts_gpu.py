"""The tcgen05 matmul with weights in tensor memory, at the edges of its tiles: token counts around the 64- / 128- / 256-column
tiles, row counts around the 128-row tile, one slab of K up to several split over a cluster or over ranges, rows that are not
16-byte multiples (fetched as every eighth row, the last ones with plain loads), several matrices in one launch."""
from __future__ import annotations

import numpy as np
import pytest

from tests.util import KIND_Q4_K, KIND_Q6_K, KIND_Q8_0, KINDS, TOL_MMA, max_rel_err, random_blocks

pytestmark = pytest.mark.gpu

SHAPES = [  # T, K, F
    (1, 256, 1), (16, 256, 128), (17, 512, 127), (63, 2048, 129), (64, 2304, 257), (65, 256, 1003), (128, 1280, 96),
    (129, 2048, 130), (256, 512, 384), (257, 768, 72), (300, 2816, 1001), (33, 4096, 2048),
]


@pytest.fixture(scope="module")
def ctx():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from marmot_b200 import Context
    from marmot_b200.runtime import REGIME_GEMM

    c = Context(0)
    c.set_regime(REGIME_GEMM)
    yield c
    c.close()


def run(ctx, oracle, kind, T, K, F, bias=False):
    import torch

    rng = np.random.default_rng(T * 7 + K * 3 + F)
    W = random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    b = rng.normal(0, 1, F).astype(np.float32) if bias else None
    bd = torch.from_numpy(b).cuda() if bias else None
    got = ctx.linear(kind, torch.from_numpy(x).cuda(), ctx.upload(W), F, bias=bd).cpu().numpy()
    ctx.synchronize()
    ref = oracle.linear(kind, x, W, F)
    assert max_rel_err(got, ref + b if bias else ref) <= TOL_MMA


@pytest.mark.parametrize("name", sorted(KINDS))
@pytest.mark.parametrize("T,K,F", SHAPES)
def test_tile_edges(ctx, oracle, name, T, K, F):
    run(ctx, oracle, KINDS[name], T, K, F, bias=F % 2 == 1)


@pytest.mark.parametrize("T,K,F", [(20, 32, 40), (70, 1056, 135), (200, 288, 67)])
def test_q8_0_partial_slabs_and_unaligned_rows(ctx, oracle, T, K, F):
    run(ctx, oracle, KIND_Q8_0, T, K, F)


@pytest.mark.parametrize("T", [24, 140])
def test_jobs_of_two_kinds_equal_single_calls(ctx, T):
    import torch

    rng = np.random.default_rng(T)
    K, sizes = 1280, [(KIND_Q4_K, 200), (KIND_Q6_K, 72), (KIND_Q4_K, 131)]
    x = torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda()
    ws = [ctx.upload(random_blocks(k, F, K, rng)) for k, F in sizes]
    outs = [torch.zeros((T, F), device="cuda") for _, F in sizes]
    ctx.linear_multi(x, [(k, w, F, o) for (k, F), w, o in zip(sizes, ws, outs)])
    for (k, F), w, o in zip(sizes, ws, outs):
        assert max_rel_err(o.cpu().numpy(), ctx.linear(k, x, w, F).cpu().numpy()) <= 1e-5
    ctx.synchronize()


@pytest.mark.parametrize("name,T", [("q4_k", 3073), ("q8_0", 3120), ("q6_k", 4161)])
def test_many_tokens_equal_calls_on_slices(ctx, name, T):
    """Token counts at which tiles widened to 16 columns are fewer than the plan asked for.  The sums' order differs: 32-bit rounding."""
    import torch

    K, F, kind = 1536, 4700, KINDS[name]
    rng = np.random.default_rng(T)
    w = ctx.upload(random_blocks(kind, F, K, rng))
    x = torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda()
    got = ctx.linear(kind, x, w, F)
    ref = torch.cat([ctx.linear(kind, part, w, F) for part in x.split(500)])
    ctx.synchronize()
    assert max_rel_err(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("T,K,F", [(20, 1024, 130), (70, 3072, 64), (150, 5632, 200)])
def test_q6_k_rows_off_16_bytes_round_their_weights_once(ctx, T, K, F):
    """Integer activations with a largest value of 127 are exact operands, so the result is that of the weights rounded to fp16, up to the
    order of 32-bit sums.  (Rounded twice, by way of the scale, it is 2e-4 off.)"""
    import torch
    from marmot_b200.synthetic import normal_blocks

    gen = torch.Generator(device="cuda")
    gen.manual_seed(K)
    w = normal_blocks(torch, KIND_Q6_K, F, K, torch.device("cuda"), gen).reshape(-1)
    x = torch.randint(-126, 127, (T, K), device="cuda", generator=gen).float()
    x[:, ::256] = 127.0
    got = ctx.linear(KIND_Q6_K, x, w, F)
    want = x.double() @ ctx.dequantize(KIND_Q6_K, w, F * K).view(F, K).half().double().T
    ctx.synchronize()
    assert max_rel_err(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5
