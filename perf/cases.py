"""The work a user of marmot_b200 has it do, as cases that can be timed and compared.

Four kinds of pass, each through the public Python interface (`marmot_b200.runtime.Context`, `marmot_b200.decoder.Decoder`):

* "linear": y = x @ W.T on a block-quantised matrix, one call per matrix of `layers` distinct matrices.  Weights of a model
  are far larger than the 126 MB L2, so a pass goes over enough matrices that they come from HBM, except where one small call
  is the case.  "graph": the calls are recorded once and replayed, as a decode loop does; otherwise they are made one by one.
* "ffn_in": gate and up projection of a decoder layer with the residual add and RMSNorm in front, the form in which a decode
  step of a few sequences calls the matmuls (`linear_multi`).
* "moe": the expert FFN of a mixture-of-experts layer on routed tokens.
* "decode" / "prefill": `Decoder.step` on a slice of a model: embedding rows, the layers, the output projection, logits out.
  Slices have one or two layers: every matmul re-quantises its input to 8 bits, so a rounding-level difference grows to
  per cents over the depth of a whole model and could no longer be told from a mistake.  They have an eighth of the
  vocabulary, so that the output projection does not outweigh the layers.

Weights are N(0, 0.02) quantised into GGUF blocks, activations N(0, 1), router weights the softmax of N(0, 1) logits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from marmot_b200.decoder import LLAMA3_8B, TINYLLAMA_1B, Decoder, DecoderShape, weight_bytes
from marmot_b200.runtime import KIND_BY_NAME, KIND_Q4_K, Context, row_bytes
from marmot_b200.synthetic import normal_blocks

DEVICE = 0
MODELS = {"tinyllama_1b": TINYLLAMA_1B, "llama3_8b": LLAMA3_8B}
MOST_FLOPS = 6e11  # of a drawn case: the largest listed one has 1.4e12, on the fastest path


def listed():
    return [
        # The smallest matmul of a model: the key projection of a 1.1B decoder for one token, called on its own.
        {"name": "linear q4_k 1x2048x256", "op": "linear", "kind": "q4_k", "T": 1, "K": 2048, "F": 256, "layers": 1, "graph": False},
        # Batch-1 decode: the 4096 x 4096 GEMV the benchmark is quoted on, over 32 matrices in a replayed graph.
        {"name": "linear q4_k 1x4096x4096 graph", "op": "linear", "kind": "q4_k", "T": 1, "K": 4096, "F": 4096, "layers": 32, "graph": True},
        # The output projection of an 8B model for one token: the largest matrix there is.
        {"name": "linear q6_k 1x4096x128256", "op": "linear", "kind": "q6_k", "T": 1, "K": 4096, "F": 128256, "layers": 1, "graph": False},
        # A few sequences: FFN input of a decode step of eight.
        {"name": "ffn_in q4_k 8x4096x14336", "op": "ffn_in", "kind": "q4_k", "T": 8, "K": 4096, "F": 14336, "layers": 4},
        # Batched decode of 64 sequences: gate / up projection.
        {"name": "linear q4_k 64x4096x14336", "op": "linear", "kind": "q4_k", "T": 64, "K": 4096, "F": 14336, "layers": 8, "graph": False},
        # A ragged batch on the down projection, in the format the Q4_K_M mix gives it.
        {"name": "linear q6_k 37x14336x4096", "op": "linear", "kind": "q6_k", "T": 37, "K": 14336, "F": 4096, "layers": 6, "graph": False},
        # Prefill of 512 tokens on an 8-bit model.
        {"name": "linear q8_0 512x4096x14336", "op": "linear", "kind": "q8_0", "T": 512, "K": 4096, "F": 14336, "layers": 4, "graph": False},
        # Mixture of experts, 8 experts top-2: a prefill batch of 2048 tokens and a decode batch of 16.
        {"name": "moe q4_k 2048 tokens", "op": "moe", "kind": "q4_k", "down": "q4_k", "T": 2048, "H": 4096, "FF": 14336, "E": 8, "top_k": 2},
        {"name": "moe q4_k 16 tokens", "op": "moe", "kind": "q4_k", "down": "q4_k", "T": 16, "H": 4096, "FF": 14336, "E": 8, "top_k": 2},
        # One token of a single sequence, one token of 64 sequences with mixed contexts (both replayed graphs), and a prompt.
        {"name": "decode tinyllama_1b 1 seq", "op": "decode", "model": "tinyllama_1b", "layers": 2, "seqs": 1, "ctx_lo": 250, "ctx_hi": 250},
        {"name": "decode llama3_8b 64 seqs", "op": "decode", "model": "llama3_8b", "layers": 1, "seqs": 64, "ctx_lo": 256, "ctx_hi": 4096},
        {"name": "prefill llama3_8b 500 tokens", "op": "prefill", "model": "llama3_8b", "layers": 1, "seqs": 1, "tokens": 500, "start": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["linear", "linear", "linear", "ffn_in", "moe", "decode", "prefill"])
    if op == "linear":
        kind = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0"])
        T = _log_int(rng, 1, 2048)
        K = 256 * _log_int(rng, 4, 56)
        F = _log_int(rng, 64, 32768)
        if rng.random() < 0.7:  # matrix heights are mostly multiples of a head or a tile, vocabularies are not
            F = max(64, F // 64 * 64)
        F = min(F, max(64, int(MOST_FLOPS / (2.0 * T * K))))
        one = F * row_bytes(KIND_BY_NAME[kind], K)
        layers = max(1, min(16, (160 << 20) // one, int(MOST_FLOPS / (2.0 * T * K * F))))
        return {"op": op, "kind": kind, "T": T, "K": K, "F": F, "layers": layers, "graph": T <= 8 and rng.random() < 0.5}
    if op == "ffn_in":
        K = 256 * _log_int(rng, 4, 32)
        F = 256 * _log_int(rng, 4, 112)
        kind = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0"])
        one = 2 * F * row_bytes(KIND_BY_NAME[kind], K)
        return {"op": op, "kind": kind, "T": rng.randint(1, 64), "K": K, "F": F, "layers": max(1, min(8, (160 << 20) // one))}
    if op == "moe":
        E = rng.choice([4, 8, 16])
        H = 256 * _log_int(rng, 4, 16)
        FF = min(256 * _log_int(rng, 2, 56), 7 * 2**26 // (E * H) // 256 * 256)
        top_k = rng.choice([1, 2, 2, 4])
        return {"op": op, "kind": "q4_k", "down": rng.choice(["q4_k", "q4_k", "q6_k"]),
                "T": min(_log_int(rng, 1, 2048), int(MOST_FLOPS / (6.0 * top_k * H * FF))), "H": H, "FF": FF, "E": E, "top_k": top_k}
    model = rng.choice(sorted(MODELS))
    if op == "decode":
        seqs = _log_int(rng, 1, 64)
        lo = _log_int(rng, 16, 2048)
        return {"op": op, "model": model, "layers": 2 if seqs == 1 else 1, "seqs": seqs, "ctx_lo": lo, "ctx_hi": min(4096, lo * rng.randint(1, 4))}
    seqs = rng.choice([1, 1, 2, 4])
    return {"op": op, "model": model, "layers": 1, "seqs": seqs, "tokens": max(seqs, _log_int(rng, 9, 512) // seqs * seqs),
            "start": rng.choice([0, 0, rng.randint(1, 1500)])}


_kept = {}


def _context():
    """The context of a program that makes its calls one by one, on torch's stream."""
    if "ctx" not in _kept:
        _kept["ctx"] = Context(DEVICE)
    return _kept["ctx"]


def _decode_stream():
    """The stream that recorded sequences run on: one for all of them, since a step of decoding follows the one before."""
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream(torch.device("cuda", DEVICE))
    return _kept["stream"]


def _shape(case) -> DecoderShape:
    m = MODELS[case["model"]]
    return DecoderShape(case["layers"], m.d, m.ffn, m.n_heads, m.n_kv_heads, m.head_dim, m.vocab // 8, m.rope_theta, m.rms_eps)


def _contexts(case):
    """Cached positions of every sequence before the pass."""
    if case["op"] == "prefill":
        return np.full(case["seqs"], case["start"], dtype=np.int64)
    # spread evenly over the range: the same amount of work whatever the seed
    return np.linspace(case["ctx_lo"], case["ctx_hi"], case["seqs"]).astype(np.int64)


def prepare(case, seed):
    dev = torch.device("cuda", DEVICE)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    op = case["op"]
    randn = lambda *shape: torch.randn(shape, device=dev, generator=gen)
    if op in ("linear", "ffn_in"):
        kind, T, K, F = KIND_BY_NAME[case["kind"]], case["T"], case["K"], case["F"]
        blocks = lambda: normal_blocks(torch, kind, F, K, dev, gen)
        s = {"op": op, "kind": kind, "F": F, "x": randn(T, K)}
        if op == "ffn_in":
            s.update(ctx=_context(), delta=randn(T, K), norm=1.0 + 0.1 * randn(K), gate=[blocks() for _ in range(case["layers"])],
                     up=[blocks() for _ in range(case["layers"])])
            s["out"] = [(torch.empty((T, F), device=dev), torch.empty((T, F), device=dev), torch.empty((T, K), device=dev))
                        for _ in range(case["layers"])]
            return s
        s["w"] = [blocks() for _ in range(case["layers"])]
        if not case["graph"]:
            s["ctx"] = _context()
            return s
        s["ctx"] = ctx = Context(DEVICE, use_torch_stream=False)
        ctx.set_stream(_decode_stream().cuda_stream)
        s["out"] = [torch.empty((T, F), device=dev) for _ in s["w"]]
        torch.cuda.synchronize()
        for w, y in zip(s["w"], s["out"]):  # workspace does not grow while a sequence is recorded
            ctx.linear(kind, s["x"], w, F, out=y)
        ctx.synchronize()
        ctx.graph_capture_begin()
        for w, y in zip(s["w"], s["out"]):
            ctx.linear(kind, s["x"], w, F, out=y)
        s["replay"] = ctx.graph_capture_end()
        return s
    if op == "moe":
        kind, down = KIND_BY_NAME[case["kind"]], KIND_BY_NAME[case["down"]]
        T, H, FF, E = case["T"], case["H"], case["FF"], case["E"]
        weights, ids = torch.topk(torch.softmax(randn(T, E), dim=1), case["top_k"], dim=1)
        return {"op": op, "ctx": _context(), "kinds": (kind, kind, down), "FF": FF, "E": E, "hidden": randn(T, H),
                "ids": ids.to(torch.int32).contiguous(), "weights": weights.contiguous(),
                "gate": normal_blocks(torch, kind, E * FF, H, dev, gen), "up": normal_blocks(torch, kind, E * FF, H, dev, gen),
                "down": normal_blocks(torch, down, E * H, FF, dev, gen)}
    shape, cached = _shape(case), _contexts(case)
    new = case["tokens"] // case["seqs"] if op == "prefill" else 1
    graph = op == "decode"
    ctx = Context(DEVICE, use_torch_stream=False) if graph else _context()
    dec = Decoder(ctx, shape, max_seqs=case["seqs"], max_ctx=int(cached.max()) + new + 16, block_size=16, seed=seed)
    dec.kv_k.normal_(generator=gen)
    dec.kv_v.normal_(generator=gen)
    seq = np.repeat(np.arange(case["seqs"]), new)
    pos = (cached[:, None] + np.arange(new)[None, :]).reshape(-1)
    s = {"op": op, "ctx": ctx, "dec": dec, "ids": torch.randint(0, shape.vocab, (len(pos),), device=dev, generator=gen, dtype=torch.int32),
         "meta": torch.from_numpy(dec.token_meta(seq, pos)).to(dev), "pos": torch.from_numpy(pos.astype(np.int32)).to(dev)}
    if graph:
        s["logits"] = torch.empty((len(pos), shape.vocab), device=dev)
        stream = _decode_stream()
        ctx.set_stream(stream.cuda_stream)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(2):
                dec.step(s["ids"], s["meta"], s["pos"], logits_out=s["logits"], decode=True)
            torch.cuda.synchronize()
            s["replay"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["replay"], stream=stream):
                dec.step(s["ids"], s["meta"], s["pos"], logits_out=s["logits"], decode=True)
    return s


def run(s):
    op, ctx = s["op"], s["ctx"]
    if op == "linear":
        if "replay" in s:
            s["replay"].launch()
            return s["out"]
        return [ctx.linear(s["kind"], s["x"], w, s["F"]) for w in s["w"]]
    if op == "ffn_in":
        for g, u, (yg, yu, x_out) in zip(s["gate"], s["up"], s["out"]):
            ctx.linear_multi(s["x"], [(s["kind"], g, s["F"], yg), (s["kind"], u, s["F"], yu)],
                             ("add_rmsnorm", s["delta"], s["norm"], 1e-5, 0.0, x_out))
        return s["out"]
    if op == "moe":
        return ctx.moe_experts(s["kinds"], s["hidden"], s["gate"], s["up"], s["down"], s["ids"], s["weights"], s["FF"], s["E"])
    dec = s["dec"]
    if op == "decode":
        with torch.cuda.stream(_decode_stream()):
            s["replay"].replay()
        return s["logits"], dec.kv_k, dec.kv_v
    return dec.step(s["ids"], s["meta"], s["pos"]), dec.kv_k, dec.kv_v


def work(case):
    op = case["op"]
    if op in ("linear", "ffn_in"):
        kind, T, K, F, n = KIND_BY_NAME[case["kind"]], case["T"], case["K"], case["F"], case["layers"]
        mats = 2 if op == "ffn_in" else 1
        more = 4 * T * K * 2 + 4 * K if op == "ffn_in" else 0  # the residual's other half in, their sum out
        return {"bytes": n * (mats * F * (row_bytes(kind, K) + 4 * T) + more) + 4 * T * K, "flops": 2.0 * n * mats * T * K * F}
    if op == "moe":
        kind, down = KIND_BY_NAME[case["kind"]], KIND_BY_NAME[case["down"]]
        T, H, FF, E, k = case["T"], case["H"], case["FF"], case["E"], case["top_k"]
        used = E * (1.0 - (1.0 - k / E) ** T)  # experts with a token, on average
        expert = 2 * FF * row_bytes(kind, H) + H * row_bytes(down, FF)
        return {"bytes": used * expert + 8 * T * H + 8 * T * k, "flops": 6.0 * T * k * H * FF}
    s, cached = _shape(case), _contexts(case)
    new = case["tokens"] // case["seqs"] if op == "prefill" else 1
    T = new * case["seqs"]
    kv_row = 2 * s.n_kv_heads * s.head_dim * 2  # K and V, float16, one layer
    kv_d = s.n_kv_heads * s.head_dim
    matmul = s.layers * s.d * (2 * s.n_heads * s.head_dim + 2 * kv_d + 3 * s.ffn) + s.vocab * s.d
    pairs = float(sum(new * int(c) + new * (new + 1) // 2 for c in cached))
    return {"bytes": weight_bytes(s) + T * row_bytes(KIND_Q4_K, s.d) + s.layers * kv_row * (int(cached.sum()) + T) + 4 * T * s.vocab,
            "flops": 2.0 * T * matmul + 4.0 * s.layers * s.n_heads * s.head_dim * pairs}


def tolerance(case):
    """Matmuls of up to eight tokens are integer dots scaled and summed in 32 bits: only the order of sums may differ.  Larger
    ones multiply fp16 operands.  Where a matmul's output is quantised to 8 bits for the next one, an operand that lands on
    the other side of a rounding moves by a whole step of 1/127 of its block's largest value."""
    if case["op"] in ("linear", "ffn_in"):
        return {"rel": 1e-5} if case["T"] <= 8 and case["op"] == "linear" else {"rel": 3e-3, "max": 0.05}
    if case["op"] == "moe":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 3e-2, "max": 0.5}
