"""Attention over a paged f16 pool with several tokens per CTA: a token's result must not depend on the tokens that share its CTA.
Prompts of one and of several sequences (runs that start and end inside a block of tokens, that cross chunks of 128 positions, with
groups of one to eight query heads) against the same tokens one call at a time, bit for bit, and against plain attention."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,hd,bs", [(8, 1, 64, 16), (8, 2, 128, 16), (6, 2, 64, 64), (4, 4, 128, 256), (4, 2, 128, 1), (2, 2, 64, 2), (4, 1, 128, 8)])
@pytest.mark.parametrize("spans", [[(0, 40)], [(100, 60), (0, 5), (250, 17)], [(3, 1), (130, 1), (126, 4), (500, 33)], [(0, 300)]])
def test_blocks_equal_single_tokens(hq, hkv, hd, bs, spans):
    import torch
    from marmot_b200 import Context

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = Context(0)
    rng = np.random.default_rng(hq * hd + len(spans))
    max_blocks = max(a + n for a, n in spans) // bs + 1
    n_blocks = max_blocks * len(spans)
    table = rng.permutation(n_blocks).reshape(len(spans), max_blocks).astype(np.uint32)
    meta = np.array([(s, pos, int(table[s, pos // bs]) * bs + pos % bs, 0) for s, (a, n) in enumerate(spans) for pos in range(a, a + n)],
                    dtype=np.uint32)
    T = len(meta)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    randn = lambda *shape: torch.from_numpy(rng.normal(0, 1, shape).astype(np.float32)).cuda()
    pool_k, pool_v = randn(n_blocks, 1, hkv, bs, hd).half(), randn(n_blocks, 1, hkv, bs, hd).half()
    q, k, v = randn(T, hq * hd), randn(T, hkv * hd), randn(T, hkv * hd)
    tab = dev(table)
    k1, v1 = pool_k.clone(), pool_v.clone()
    got = ctx.paged_attention(dev(meta), q, k, v, k1, v1, tab, 0, hq, hkv, hd, bs, hd ** -0.5)
    k2, v2 = pool_k.clone(), pool_v.clone()
    one = [ctx.paged_attention(dev(meta[i:i + 1]), q[i:i + 1].clone(), k[i:i + 1].clone(), v[i:i + 1].clone(), k2, v2, tab, 0, hq, hkv, hd, bs,
                               hd ** -0.5) for i in range(T)]
    ctx.synchronize()
    assert torch.equal(k1, k2) and torch.equal(v1, v2)
    assert torch.equal(got, torch.cat(one))
    for i in (0, T // 2, T - 1):  # and plain attention in double precision
        s, pos = int(meta[i, 0]), int(meta[i, 1])
        rows = [(int(table[s, x // bs]), x % bs) for x in range(pos + 1)]
        keys = torch.stack([k1[b, 0, :, o] for b, o in rows]).double()
        vals = torch.stack([v1[b, 0, :, o] for b, o in rows]).double()
        qi = q[i].double().view(hkv, hq // hkv, hd)
        w = torch.softmax(torch.einsum("hgd,phd->hgp", qi, keys) * hd ** -0.5, dim=-1)
        want = torch.einsum("hgp,phd->hgd", w, vals).reshape(-1)
        assert float((got[i].double() - want).abs().max()) <= 2e-5
    ctx.close()


@pytest.mark.parametrize("n_seq,hd,bs", [(9, 128, 16), (40, 128, 2), (40, 64, 32), (260, 64, 16)])
def test_decode_blocks_equal_three_steps(n_seq, hd, bs):
    """The fused decode step with several sequences per CTA (contexts on both sides of a chunk, a sequence's first token)."""
    import torch
    from marmot_b200 import Context

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx, hq, hkv = Context(0), 16, 8
    rng = np.random.default_rng(n_seq)
    lens = rng.integers(0, 300, n_seq)
    lens[:4] = (0, 127, 128, 6000)
    max_blocks = int(lens.max()) // bs + 1
    used = [int(n) // bs + 1 for n in lens]
    n_blocks = sum(used)
    table = np.full((n_seq, max_blocks), 0xFFFFFFFF, dtype=np.uint32)
    order, at = rng.permutation(n_blocks), 0
    for s, n in enumerate(used):
        table[s, :n] = order[at:at + n]
        at += n
    meta = np.array([(s, n, int(table[s, n // bs]) * bs + n % bs, 0) for s, n in enumerate(lens)], dtype=np.uint32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    randn = lambda *shape: torch.from_numpy(rng.normal(0, 1, shape).astype(np.float32)).cuda()
    k1, v1 = randn(n_blocks, 1, hkv, bs, hd).half(), randn(n_blocks, 1, hkv, bs, hd).half()
    k2, v2 = k1.clone(), v1.clone()
    q, k, v, pos = randn(n_seq, hq * hd), randn(n_seq, hkv * hd), randn(n_seq, hkv * hd), dev(lens.astype(np.int32))
    got = ctx.paged_attention_decode(dev(meta), q.clone(), k.clone(), v, k1, v1, dev(table), 0, hq, hkv, hd, bs, hd ** -0.5, pos, 10000.0)
    ctx.rope_qk(q, k, pos, hq, hkv, hd, 10000.0)
    want = ctx.paged_attention(dev(meta), q, k, v, k2, v2, dev(table), 0, hq, hkv, hd, bs, hd ** -0.5)
    ctx.synchronize()
    assert torch.equal(k1, k2) and torch.equal(v1, v2) and torch.equal(got, want)
    ctx.close()


@pytest.mark.parametrize("hq,hkv,hd,bs", [(8, 2, 128, 16), (8, 8, 64, 16), (16, 2, 64, 32)])
@pytest.mark.parametrize("lengths", [(1,), (20,), (1, 7, 33, 2)])
def test_values_that_are_not_finite_stay_with_the_tokens_that_see_them(hq, hkv, hd, bs, lengths):
    """Many sequences, runs of the given lengths whose last V rows overflow f16 or are NaN: the tokens ahead of them, which share
    their CTAs, equal single-token calls bit for bit, as do the last ones."""
    import torch
    from marmot_b200 import Context

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = Context(0)
    rng = np.random.default_rng(hq + len(lengths))
    n_seq = 400 // sum(lengths) * len(lengths)
    spans = [(int(rng.integers(0, 300)), lengths[i % len(lengths)]) for i in range(n_seq)]
    max_blocks = max(a + n for a, n in spans) // bs + 1
    table = rng.permutation(max_blocks * n_seq).reshape(n_seq, max_blocks).astype(np.uint32)
    meta = np.array([(s, pos, int(table[s, pos // bs]) * bs + pos % bs, 0) for s, (a, n) in enumerate(spans) for pos in range(a, a + n)],
                    dtype=np.uint32)
    T = len(meta)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    randn = lambda *shape: torch.from_numpy(rng.normal(0, 1, shape).astype(np.float32)).cuda()
    pool_k, pool_v = randn(max_blocks * n_seq, 1, hkv, bs, hd).half(), randn(max_blocks * n_seq, 1, hkv, bs, hd).half()
    q, k, v = randn(T, hq * hd), randn(T, hkv * hd), randn(T, hkv * hd)
    last = np.cumsum([n for _, n in spans]) - 1
    v[last[::2], 5] = 1e6
    v[last[1::2], hkv * hd - 1] = float("nan")
    tab, m = dev(table), dev(meta)
    k1, v1, k2, v2 = pool_k.clone(), pool_v.clone(), pool_k.clone(), pool_v.clone()
    got = ctx.paged_attention(m, q, k, v, k1, v1, tab, 0, hq, hkv, hd, bs, hd ** -0.5)
    one = torch.cat([ctx.paged_attention(m[i:i + 1].clone(), q[i:i + 1].clone(), k[i:i + 1].clone(), v[i:i + 1].clone(), k2, v2, tab, 0, hq, hkv, hd,
                                         bs, hd ** -0.5) for i in range(T)])
    ctx.synchronize()
    others = torch.ones(T, dtype=torch.bool)
    others[last] = False
    assert torch.isfinite(got[others.cuda()]).all()
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), one.nan_to_num(7.0, 8.0, 9.0))
    ctx.close()
