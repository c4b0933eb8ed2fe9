"""The integer tensor-core matmul for a handful of tokens, at the edges of its tiles (16 tokens, 128 rows, one slab of K up to
several split over a cluster or over ranges, Q6_K rows of any alignment), and the few-route MoE that is built on it."""
from __future__ import annotations

import numpy as np
import pytest

from tests.util import KIND_Q4_K, KIND_Q6_K, TOL_FP32, TOL_MOE, max_rel_err, random_blocks

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


@pytest.mark.parametrize("kind", [KIND_Q4_K, KIND_Q6_K])
@pytest.mark.parametrize("T,K,F", [(2, 256, 1), (7, 512, 129), (8, 2048, 130), (9, 4096, 1000), (15, 2304, 257), (16, 768, 20000),
                                   (17, 1280, 135), (33, 256, 128), (64, 2816, 96)])
def test_tile_edges(ctx, oracle, kind, T, K, F):
    import torch
    from marmot_b200.runtime import REGIME_AUTO, REGIME_I8MMA

    rng = np.random.default_rng(T * 7 + K * 3 + F)
    W = random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    bias = rng.normal(0, 1, F).astype(np.float32)
    ctx.set_regime(REGIME_I8MMA)
    got = ctx.linear(kind, torch.from_numpy(x).cuda(), ctx.upload(W), F, bias=torch.from_numpy(bias).cuda()).cpu().numpy()
    ctx.set_regime(REGIME_AUTO)
    ctx.synchronize()
    assert max_rel_err(got, oracle.linear(kind, x, W, F) + bias) <= TOL_FP32


@pytest.mark.parametrize("T,K,F", [(3, 3072, 125), (8, 1280, 61), (4, 768, 1)])
def test_rows_that_cannot_be_streamed(ctx, oracle, T, K, F):
    import torch

    rng = np.random.default_rng(T + K)
    W = random_blocks(KIND_Q6_K, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    got = ctx.linear(KIND_Q6_K, torch.from_numpy(x).cuda(), ctx.upload(W), F).cpu().numpy()
    ctx.synchronize()
    assert max_rel_err(got, oracle.linear(KIND_Q6_K, x, W, F)) <= TOL_FP32


# Sizes just beyond the lines, and just short of them
BEYOND = [(KIND_Q4_K, 2, 1024, 12289), (KIND_Q4_K, 2, 16384, 3100), (KIND_Q4_K, 3, 1536, 8200), (KIND_Q4_K, 3, 14336, 1030), (KIND_Q4_K, 4, 768, 8200),
          (KIND_Q6_K, 3, 2048, 12300), (KIND_Q6_K, 3, 10240, 4928), (KIND_Q6_K, 4, 1024, 8200), (KIND_Q6_K, 4, 14336, 1030), (KIND_Q6_K, 4, 4096, 8200)]
SHORT = [(KIND_Q4_K, 2, 1024, 12280), (KIND_Q4_K, 2, 16384, 3070), (KIND_Q4_K, 3, 1536, 8184), (KIND_Q4_K, 3, 14336, 1020), (KIND_Q4_K, 4, 768, 8184),
         (KIND_Q6_K, 3, 2048, 12280), (KIND_Q6_K, 3, 10240, 4912), (KIND_Q6_K, 3, 8448, 8000), (KIND_Q6_K, 4, 1024, 8184), (KIND_Q6_K, 4, 14336, 1020),
         (KIND_Q6_K, 4, 4096, 8184), (KIND_Q6_K, 4, 4096, 9600), (KIND_Q6_K, 4, 3584, 10752)]


@pytest.mark.parametrize("kind,T,K,F,beyond", [(*s, True) for s in BEYOND] + [(*s, False) for s in SHORT])
def test_lines_of_two_to_four_tokens(ctx, oracle, kind, T, K, F, beyond):
    """Beyond the lines a call is two launches, short of them one, and one where it is being recorded: the dp4a kernel, whose graph holds no address
    of the workspace that a later, larger call moves.  The results are the dp4a kernel's but for the order of the f32 terms."""
    import torch
    from marmot_b200 import Context
    from marmot_b200.runtime import REGIME_AUTO, REGIME_GEMV

    rng = np.random.default_rng(T + K + F)
    W = random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    xd, wd = torch.from_numpy(x).cuda(), ctx.upload(W)
    before = ctx.launch_count()
    got = ctx.linear(kind, xd, wd, F).cpu().numpy()
    assert ctx.launch_count() - before == (2 if beyond else 1)
    ctx.set_regime(REGIME_GEMV)
    ref = ctx.linear(kind, xd, wd, F).cpu().numpy()
    ctx.set_regime(REGIME_AUTO)
    ctx.synchronize()
    assert max_rel_err(got, ref) <= 1e-5
    if not beyond:
        assert np.array_equal(got, ref)
        return
    assert max_rel_err(got, oracle.linear(kind, x, W, F)) <= TOL_FP32
    fresh = Context(0, use_torch_stream=False)
    stream = torch.cuda.Stream()
    fresh.set_stream(stream.cuda_stream)
    out = torch.zeros((T, F), device="cuda")
    more = torch.from_numpy(rng.normal(0, 1, (16, K)).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    fresh.linear(kind, xd, wd, F, out=out)
    fresh.synchronize()
    fresh.graph_capture_begin()
    before = fresh.launch_count()
    fresh.linear(kind, xd, wd, F, out=out)
    assert fresh.launch_count() - before == 1
    graph = fresh.graph_capture_end()
    fresh.linear(kind, more, wd, F)
    out.zero_()
    torch.cuda.synchronize()
    graph.launch()
    fresh.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
    graph.close()
    fresh.close()


def test_few_tokens_without_memory_for_workspace():
    """A call that the dp4a kernel can have does not fail for want of the integer matmul's workspace; a larger one does, and works again later."""
    import torch
    from marmot_b200 import Context, MarmotCudaError
    from marmot_b200.runtime import REGIME_AUTO, REGIME_GEMV

    T, K, F = 4, 768, 16384
    rng = np.random.default_rng(4)
    ctx = Context(0)
    x, w = torch.from_numpy(rng.normal(0, 1, (16, K)).astype(np.float32)).cuda(), ctx.upload(random_blocks(KIND_Q4_K, F, K, rng))
    ctx.set_regime(REGIME_GEMV)
    ref = ctx.linear(KIND_Q4_K, x[:T], w, F).cpu().numpy()
    ctx.set_regime(REGIME_AUTO)
    ctx._check(ctx.lib.mcu_test_device_full(ctx.handle, 1))
    assert np.array_equal(ctx.linear(KIND_Q4_K, x[:T], w, F).cpu().numpy(), ref)
    with pytest.raises(MarmotCudaError, match="no device memory"):
        ctx.linear(KIND_Q4_K, x, w, F)
    ctx._check(ctx.lib.mcu_test_device_full(ctx.handle, 0))
    before = ctx.launch_count()
    assert max_rel_err(ctx.linear(KIND_Q4_K, x[:T], w, F).cpu().numpy(), ref) <= 1e-5
    assert ctx.launch_count() - before == 2
    ctx.close()


def test_two_tokens_on_rows_too_long_to_stream():
    """The call and its recording are the same kernels: the one finds the workspace that the other has reserved."""
    import torch
    from marmot_b200 import Context

    T, K, F = 2, 131072, 400
    rng = np.random.default_rng(3)
    ctx = Context(0, use_torch_stream=False)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    x, w = torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda(), ctx.upload(random_blocks(KIND_Q4_K, F, K, rng))
    out = torch.zeros((T, F), device="cuda")
    torch.cuda.synchronize()
    ctx.linear(KIND_Q4_K, x, w, F, out=out)
    ctx.synchronize()
    first = out.cpu().numpy()
    ctx.graph_capture_begin()
    ctx.linear(KIND_Q4_K, x, w, F, out=out)
    graph = ctx.graph_capture_end()
    out.zero_()
    torch.cuda.synchronize()
    graph.launch()
    ctx.synchronize()
    assert np.array_equal(out.cpu().numpy(), first)
    graph.close()
    ctx.close()


@pytest.mark.parametrize("T,K,F", [(4, 768, 16384), (8, 4096, 4096)])
def test_diagnostic_switch(T, K, F):
    """MARMOT_CUDA_NO_I8MMA leaves a call of few tokens to the dp4a kernel, which is one launch (the integer matmul: two)."""
    import os
    import subprocess
    import sys

    program = f"""
import torch
from marmot_b200 import Context
from marmot_b200.runtime import KIND_Q4_K
ctx = Context(0)
x, w = torch.zeros(({T}, {K}), device="cuda"), torch.zeros({F} * {K} // 256 * 144, dtype=torch.uint8, device="cuda")
before = ctx.launch_count()
ctx.linear(KIND_Q4_K, x, w, {F})
ctx.synchronize()
print("launches", ctx.launch_count() - before)
"""
    for switch, launches in ((None, 2), ("1", 1)):
        env = {k: v for k, v in os.environ.items() if k != "MARMOT_CUDA_NO_I8MMA"}
        if switch:
            env["MARMOT_CUDA_NO_I8MMA"] = switch
        r = subprocess.run([sys.executable, "-c", program], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        assert f"launches {launches}" in r.stdout.splitlines(), (switch, r.stdout)


@pytest.mark.parametrize("T,K,F", [(3, 4096, 5632), (4, 4096, 4096), (5, 2048, 2056), (8, 4096, 1030), (16, 512, 40)])
def test_two_matrices_of_each_kind_with_prologues(ctx, oracle, T, K, F):
    """The sizes at which linear_multi leaves the dp4a kernel: every result equals the one of the plain regime, and x' is exact."""
    import torch
    from marmot_b200.runtime import REGIME_AUTO, REGIME_GEMV_PLAIN

    rng = np.random.default_rng(T + K + F)
    dev = lambda a: torch.from_numpy(a.astype(np.float32)).cuda()
    x, aux, w = dev(rng.normal(0, 1, (T, K))), dev(rng.normal(0, 1, (T, K))), dev(rng.normal(1, 0.2, K))
    kinds = (KIND_Q4_K, KIND_Q4_K) if T < 5 else (KIND_Q4_K, KIND_Q6_K, KIND_Q4_K, KIND_Q6_K)
    ws = [ctx.upload(random_blocks(k, F, K, rng)) for k in kinds]

    def run(prologue, x_out=None):
        outs = [torch.zeros((T, F), device="cuda") for _ in kinds]
        ctx.linear_multi(x, [(k, m, F, o) for k, m, o in zip(kinds, ws, outs)], prologue(x_out) if prologue else None)
        ctx.synchronize()
        return outs

    for prologue in (None, lambda xo: ("swiglu", aux), lambda xo: ("add_rmsnorm", aux, w, 1e-5, 0.0, xo)):
        x_out = torch.zeros((T, K), device="cuda")
        got = run(prologue, x_out)
        if prologue is not None and x_out.abs().max() > 0:
            assert torch.equal(x_out, x + aux)
        ctx.set_regime(REGIME_GEMV_PLAIN)
        ref = run(prologue, torch.zeros((T, K), device="cuda"))
        ctx.set_regime(REGIME_AUTO)
        for a, b in zip(got, ref):  # a last bit of the prologue may move an int8 quant by one
            assert max_rel_err(a.cpu().numpy(), b.cpu().numpy()) <= 2e-3


@pytest.mark.parametrize("kinds", [(KIND_Q4_K, KIND_Q4_K, KIND_Q6_K), (KIND_Q6_K, KIND_Q6_K, KIND_Q4_K)])
@pytest.mark.parametrize("T,E,k", [(1, 4, 1), (17, 6, 2), (40, 3, 3), (127, 300, 2)])
def test_few_route_moe(ctx, oracle, kinds, T, E, k):
    import torch
    from marmot_b200 import MarmotCudaError

    H, FF = 512, 256
    rng = np.random.default_rng(T + E + k)
    hid = rng.normal(0, 1, (T, H)).astype(np.float32)
    rows = ((E * FF, H), (E * FF, H), (E * H, FF))
    gate, up, down = (random_blocks(kd, F, K, rng, d_sigma=0.0005) for kd, (F, K) in zip(kinds, rows))
    p = rng.random((T, E)).astype(np.float32)
    p[:, E - 1] = 0.0  # the last expert is hardly chosen
    vals, ids = oracle.topk(p, k)
    ref = oracle.moe_experts(kinds, hid, gate, up, down, ids, vals, FF, E)
    hd, vd = torch.from_numpy(hid).cuda(), torch.from_numpy(np.ascontiguousarray(vals)).cuda()
    idd = torch.from_numpy(np.ascontiguousarray(ids)).cuda()
    gd, ud, dd = ctx.upload(gate), ctx.upload(up), ctx.upload(down)
    got = ctx.moe_experts(kinds, hd, gd, ud, dd, idd, vd, FF, E)
    ctx.synchronize()
    assert max_rel_err(got.cpu().numpy(), ref) <= TOL_MOE
    bad = ids.copy()
    bad[T - 1, k - 1] = E
    with pytest.raises(MarmotCudaError):
        ctx.moe_experts(kinds, hd, gd, ud, dd, torch.from_numpy(np.ascontiguousarray(bad)).cuda(), vd, FF, E)
        ctx.synchronize()
    again = ctx.moe_experts(kinds, hd, gd, ud, dd, idd, vd, FF, E)
    ctx.synchronize()
    assert torch.equal(again, got)


@pytest.mark.parametrize("T", [9, 64])  # the integer and the fp16 kernel, both with tiles cut between CTAs
def test_calls_after_a_wait_that_ran_out(ctx, T):
    """The tickets of cut tiles that a kernel left drawn do not reach the next call (a host-side hook sets the state; nothing times out)."""
    import torch
    from marmot_b200 import MarmotCudaError

    K, F = 2048, 20000
    rng = np.random.default_rng(T)
    w = ctx.upload(random_blocks(KIND_Q4_K, F, K, rng))
    x, before = (torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda() for _ in range(2))
    want = ctx.linear(KIND_Q4_K, x, w, F)
    ctx.linear(KIND_Q4_K, before, w, F)  # its shares are what a ticket drawn too early would add up
    ctx.synchronize()
    assert ctx.lib.mcu_test_matmul_gave_up(ctx.handle) == 0
    with pytest.raises(MarmotCudaError, match="timed out"):
        ctx.synchronize()
    assert torch.equal(ctx.linear(KIND_Q4_K, x, w, F), want)
    ctx.synchronize()


@pytest.mark.parametrize("T", [17, 130])  # few routes on the integer kernel, 260 on the fp16 one
def test_recorded_moe_follows_its_routes(ctx, T):
    """Replays whose routes were written just ahead of them equal eager calls: the matmuls read the groups' sizes of this replay."""
    import torch

    H, FF, E, k = 512, 256, 8, 2
    rng = np.random.default_rng(T)
    kinds = (KIND_Q4_K,) * 3
    gate, up, down = (ctx.upload(random_blocks(KIND_Q4_K, F, K, rng, d_sigma=0.0005)) for F, K in ((E * FF, H), (E * FF, H), (E * H, FF)))
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.stream(stream):
            hid = torch.randn((T, H), device="cuda")
            weights = torch.full((T, k), 0.5, device="cuda")
            routes = [torch.from_numpy(np.stack([rng.permutation(e)[:k] for _ in range(T)]).astype(np.int32)).cuda() for e in (2, 8, 3, 5) * 4]
            ids = routes[0].clone()
            call = lambda i: ctx.moe_experts(kinds, hid, gate, up, down, i, weights, FF, E)
            want = [call(r) for r in routes]
            ctx.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                out = call(ids)
            got = []
            for r in routes:
                ids.copy_(r)
                g.replay()
                got.append(out.clone())
            ctx.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
            del g
    finally:
        ctx.synchronize()
        ctx.set_stream(0)


def test_a_rank_without_routes_between_others(ctx):
    """Grouped launches that find no work do not let the kernels behind them run ahead: calls for empty expert ranges in between."""
    import torch

    T, H, FF, E, k = 200, 512, 256, 8, 2
    rng = np.random.default_rng(5)
    kinds = (KIND_Q4_K,) * 3
    blocks = lambda F, K: ctx.upload(random_blocks(KIND_Q4_K, F, K, rng, d_sigma=0.0005))
    gate, up, down = blocks(4 * FF, H), blocks(4 * FF, H), blocks(4 * H, FF)
    hid, weights = torch.randn((T, H), device="cuda"), torch.full((T, k), 0.5, device="cuda")
    ids = torch.from_numpy(np.stack([rng.permutation(4)[:k] for _ in range(T)]).astype(np.int32)).cuda()
    local = lambda lo: ctx.moe_experts_local(kinds, hid, gate, up, down, ids, weights, FF, E, lo, 4)
    want = local(0)
    ctx.synchronize()
    for _ in range(5):
        none, some = local(4), local(0)
        ctx.synchronize()
        assert not none.any() and torch.equal(some, want)


@pytest.mark.parametrize("kind", [KIND_Q4_K, KIND_Q6_K])
@pytest.mark.parametrize("K", [256 * 33, 256 * 65, 256 * 130])
def test_staging_of_long_rows(ctx, oracle, kind, K):
    """Rows whose sub-blocks take less than a turn of the staging's threads, or a turn and a little."""
    import torch

    T, F = 9, 130
    rng = np.random.default_rng(K)
    W = random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    got = ctx.linear(kind, torch.from_numpy(x).cuda(), ctx.upload(W), F).cpu().numpy()
    ctx.synchronize()
    assert max_rel_err(got, oracle.linear(kind, x, W, F)) <= TOL_FP32


def test_few_route_moe_leaves_the_glu_in_its_buffer(ctx):
    """The down staging writes act(gate) * up over the gate rows that it reads: rows of more blocks than a CTA has warps."""
    T, k, E, H, FF = 20, 2, 2, 256, 256 * 40
    rng = np.random.default_rng(9)
    import torch

    kinds = (KIND_Q4_K,) * 3
    gate, up, down = (ctx.upload(random_blocks(KIND_Q4_K, F, K, rng, d_sigma=0.0005)) for F, K in ((E * FF, H), (E * FF, H), (E * H, FF)))
    hid = torch.from_numpy(rng.normal(0, 1, (T, H)).astype(np.float32)).cuda()
    ids = torch.from_numpy(np.tile(np.arange(E, dtype=np.int32), (T, 1))).cuda()  # every token to both experts
    ctx.moe_experts(kinds, hid, gate, up, down, ids, torch.full((T, k), 0.5, device="cuda"), FF, E)
    b = ctx.moe_last_buffers(T, k, H, FF)
    assert not b["grouped"]
    half = gate.numel() // 2
    for e in range(E):  # sorted routes: expert by expert, tokens in order
        # (the calls below do not use the MoE buffers; slices of sixteen tokens take the same kernel)
        g, u = (torch.cat([ctx.linear(KIND_Q4_K, p, w[e * half:(e + 1) * half], FF) for p in (hid[:10], hid[10:])]) for w in (gate, up))
        want = g / (1 + torch.exp(-g)) * u
        assert max_rel_err(b["gate_out"][e * T:(e + 1) * T].cpu().numpy(), want.cpu().numpy()) <= 1e-4
    ctx.synchronize()


@pytest.mark.parametrize("T", [9, 16])
@pytest.mark.parametrize("prologue", [False, True])
def test_q8_0_among_k_quants_leaves_them_exact(ctx, oracle, T, prologue):
    """Nine to sixteen tokens: the K-quant matrices of a call keep their integer dots (32-bit rounding) beside a Q8_0 matrix."""
    import torch
    from tests.util import KIND_Q8_0, TOL_MMA

    K, F = 2048, 300
    rng = np.random.default_rng(T)
    kinds = (KIND_Q8_0, KIND_Q4_K, KIND_Q6_K, KIND_Q4_K)
    ws = [random_blocks(k, F, K, rng) for k in kinds]
    x, aux, w = (rng.normal(0, 1, s).astype(np.float32) for s in ((T, K), (T, K), (K,)))
    xd, ad, wd = (torch.from_numpy(a).cuda() for a in (x, aux, w))
    outs, x_out = [torch.zeros((T, F), device="cuda") for _ in kinds], torch.zeros((T, K), device="cuda")
    ctx.linear_multi(xd, [(k, ctx.upload(m), F, o) for k, m, o in zip(kinds, ws, outs)],
                     ("add_rmsnorm", ad, wd, 1e-5, 0.0, x_out) if prologue else None)
    ctx.synchronize()
    if prologue:
        assert torch.equal(x_out, xd + ad)
        h = torch.empty_like(xd)
        ctx.add_rmsnorm(xd, ad, wd, 1e-5, torch.empty_like(xd), h)  # the same operations in the same order
        x = h.cpu().numpy()
    for k, m, o in zip(kinds, ws, outs):
        assert max_rel_err(o.cpu().numpy(), oracle.linear(k, x, m, F)) <= (TOL_MMA if k == KIND_Q8_0 else 2e-5)


@pytest.mark.parametrize("kind,T,K", [(KIND_Q4_K, 9, 53248), (KIND_Q6_K, 12, 50176), (KIND_Q4_K, 10, 131072)])
def test_rows_longer_than_the_static_shared_memory(ctx, oracle, kind, T, K):
    """More than 48,000 values to a row: still integer dots, so 32-bit rounding."""
    import torch

    F = 40
    rng = np.random.default_rng(K)
    W = random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    got = ctx.linear(kind, torch.from_numpy(x).cuda(), ctx.upload(W), F).cpu().numpy()
    ctx.synchronize()
    assert max_rel_err(got, oracle.linear(kind, x, W, F)) <= 5e-5


@pytest.mark.parametrize("kind,T,E,k", [(KIND_Q6_K, 40, 4, 4), (KIND_Q4_K, 1, 8, 1), (KIND_Q4_K, 1, 8, 2), (KIND_Q6_K, 9, 3, 2)])
def test_recorded_moe_after_an_eager_call(ctx, oracle, kind, T, E, k):
    """Few-route calls that go expert by expert when the counts can be read (many rows or next to none per expert) can still be recorded
    after one eager call, and give the same up to a re-quantised intermediate; an id out of range leaves the output alone."""
    import torch
    from marmot_b200 import Context, MarmotCudaError

    H, FF = 512, 256
    rng = np.random.default_rng(T + E)
    hid = rng.normal(0, 1, (T, H)).astype(np.float32)
    gate, up, down = (random_blocks(kind, F, K, rng, d_sigma=0.0005) for F, K in ((E * FF, H), (E * FF, H), (E * H, FF)))
    vals, ids = oracle.topk(rng.random((T, E)).astype(np.float32), k)
    ref = oracle.moe_experts((kind,) * 3, hid, gate, up, down, ids, vals, FF, E)
    c = Context(0, use_torch_stream=False)  # (a workspace of its own)
    stream = torch.cuda.Stream()
    c.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        hd, vd, idd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (hid, vals, ids))
        gd, ud, dd = (c.upload(w) for w in (gate, up, down))
        out = torch.empty((T, H), device="cuda")
        call = lambda i: c.moe_experts_local((kind,) * 3, hd, gd, ud, dd, i, vd, FF, E, 0, E, out=out)
        assert max_rel_err(call(idd).cpu().numpy(), ref) <= TOL_MOE
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            call(idd)
        out.zero_()
        g.replay()
        c.synchronize()
        assert max_rel_err(out.cpu().numpy(), ref) <= TOL_MOE
        out.fill_(7.0)
        bad = idd.clone()
        bad[0, 0] = E
        with pytest.raises(MarmotCudaError):
            call(bad)
        c.synchronize()
        assert (out == 7.0).all()
        del g
    c.close()


@pytest.mark.parametrize("kind,T,K,F", [(KIND_Q4_K, 8, 1024, 2000), (KIND_Q4_K, 9, 256, 70), (KIND_Q4_K, 16, 1000, 129), (KIND_Q6_K, 5, 2048, 4097),
                                        (KIND_Q6_K, 9, 4096, 2049), (KIND_Q6_K, 16, 14336, 513), (KIND_Q6_K, 8, 2048, 20003)])
def test_mma_sync_sizes(ctx, oracle, kind, T, K, F):
    """Sizes that stay with the mma.sync kernel: one stage per CTA, row groups cut between CTAs, ragged rows, one and two token tiles."""
    import torch

    rng = np.random.default_rng(T + K + F)
    W, W2 = random_blocks(kind, F, K, rng), random_blocks(kind, F, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    bias = rng.normal(0, 1, F).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    got = ctx.linear(kind, xd, ctx.upload(W), F, bias=torch.from_numpy(bias).cuda()).cpu().numpy()
    assert max_rel_err(got, oracle.linear(kind, x, W, F) + bias) <= 2e-5
    a, b = ctx.linear_dual(kind, xd, ctx.upload(W), ctx.upload(W2), F)
    ctx.synchronize()
    assert max_rel_err(a.cpu().numpy(), oracle.linear(kind, x, W, F)) <= 2e-5
    assert max_rel_err(b.cpu().numpy(), oracle.linear(kind, x, W2, F)) <= 2e-5


def test_recorded_mma_sync_call_keeps_its_workspace(ctx, oracle):
    """A recorded call replays after calls of more rows and of more tokens per tile: shares and tickets stay where they were."""
    import torch
    from marmot_b200 import Context

    T, K, F, more = 16, 2048, 20003, 40001
    rng = np.random.default_rng(F)
    W, W2 = random_blocks(KIND_Q6_K, F, K, rng), random_blocks(KIND_Q6_K, more, K, rng)
    x = rng.normal(0, 1, (T, K)).astype(np.float32)
    c = Context(0, use_torch_stream=False)  # (a workspace of its own)
    stream = torch.cuda.Stream()
    c.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        xd, wd, wd2 = torch.from_numpy(x).cuda(), c.upload(W), c.upload(W2)
        out = torch.empty((8, F), device="cuda")
        c.linear(KIND_Q6_K, xd, wd, F)  # (the staged activations of sixteen tokens are reserved)
        c.linear(KIND_Q6_K, xd[:8], wd, F, out=out)
        first = out.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            c.linear(KIND_Q6_K, xd[:8], wd, F, out=out)
        c.linear(KIND_Q6_K, xd, wd2, more)
        out.zero_()
        g.replay()
        c.synchronize()
        assert torch.equal(out, first)
        del g
    assert max_rel_err(first.cpu().numpy(), oracle.linear(KIND_Q6_K, x[:8], W, F)) <= 2e-5
    c.close()
