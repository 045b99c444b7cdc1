"""The work this package is asked to do, as measurable cases over its public entry points.

Four kinds of pass:

* ``call``    one fused decode GEMV through the functional interface (``decode_int2_linear`` / ``decode_int4_linear``)
* ``linear``  one forward of a packed Linear module: 1 - 4 rows (decode), 5 - 16 rows (a decode batch), more rows (a prompt)
* ``step``    one decode step of a whole mixed-bit decoder replayed from a CUDA graph, as a serving loop with its own
              sampler runs it: token ids and position in, logits and the appended key / value caches out
* ``pack``    quantising one weight matrix with activation statistics, what the per-layer planner does for every candidate

Weights are quantised from N(0, 0.02) with the package's own quantisers; activations are fp16 / bf16 N(0, 1), with lognormal
channel scales where outlier columns are kept.  Decoder shapes are the repository's (``model_tools.SHAPES``), with fewer
layers where the full depth would only repeat the same work.
"""
from __future__ import annotations

import math

import torch
from torch import nn

from ai_accel_studio_b200 import model_tools
from ai_accel_studio_b200.kernels.decode_int2 import decode_int2_linear
from ai_accel_studio_b200.kernels.groupwise_int2 import pack_groupwise_int2
from ai_accel_studio_b200.kernels.groupwise_int4 import decode_int4_linear, pack_groupwise_int4
from ai_accel_studio_b200.optimize import HybridInt2Linear, HybridInt4Linear
from ai_accel_studio_b200.optimize._hybrid_base import snap_outlier_count
from ai_accel_studio_b200.optimize.siblings import fuse_decoder_siblings
from ai_accel_studio_b200.runtime_v5 import StaticGraphDecoder

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _linear(name, bits, m, n, k, group=128, dtype="fp16", outliers=0, rank=0, bias=False, kind="linear"):
    return {"name": name, "kind": kind, "bits": bits, "m": m, "n": n, "k": k, "group": group, "dtype": dtype,
            "outliers": outliers, "rank": rank, "bias": bias}


def _step(name, shape, layers, batch, context, fused):
    return {"name": name, "kind": "step", "shape": shape, "layers": layers, "batch": batch, "context": context, "fused": fused}


def _pack(name, bits, n, k, group):
    return {"name": name, "kind": "pack", "bits": bits, "n": n, "k": k, "group": group}


def listed():
    return [
        # the key projection of a 0.5B decoder, one token: the smallest call a decode loop makes
        _linear("int4_m1_k_proj_small", 4, 1, 128, 896, outliers=8, rank=8, bias=True),
        # the kernel micro-benchmark: one token, square projection, no extra terms, functional interface
        _linear("int2_m1_4096_call", 2, 1, 4096, 4096, group=64, kind="call"),
        # the benchmark Linear: four tokens, outlier columns and low-rank residual
        _linear("int4_m4_11008", 4, 4, 11008, 4096, outliers=41, rank=8),
        # nothing aligned: odd rows, K padded to the group, odd rank, bf16, bias, three tokens
        _linear("int4_m3_ragged_bf16", 4, 3, 4999, 4300, group=64, dtype="bf16", outliers=16, rank=5, bias=True),
        # a decode batch of 16 through the gate projection of an 8B decoder
        _linear("int2_m16_gate", 2, 16, 14336, 4096, outliers=40, rank=8),
        # a decode batch of 8 through the down projection of a 70B decoder: the largest matrix read for few rows
        _linear("int4_m8_down_large", 4, 8, 8192, 28672, outliers=64, rank=8),
        # a 512-token prompt through the gate projection of an 8B decoder
        _linear("int4_m512_gate_bf16", 4, 512, 14336, 4096, dtype="bf16", outliers=40, rank=8),
        # a 1000-token prompt through the gate projection of a 70B decoder: the largest Linear
        _linear("int2_m1000_gate_large", 2, 1000, 28672, 8192, outliers=64, rank=8),
        # whole decode steps: 0.5B at full depth; 8B and 70B widths with fewer layers and fused siblings
        _step("step_0.5b_b1", "qwen2.5-0.5b", 24, 1, 160, False),
        _step("step_8b_b1", "llama-3-8b", 16, 1, 576, True),
        _step("step_70b_b4", "llama-3-70b", 6, 4, 1088, True),
        # quantising a square projection for the planner
        _pack("pack_int2_4096", 2, 4096, 4096, 128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, v, common):
    """Mostly a multiple of ``common``, sometimes of 8, sometimes anything."""
    u = rng.random()
    step = common if u < 0.6 else 8 if u < 0.85 else 1
    return max(step, v // step * step)


def draw(rng):
    kind = rng.choices(("linear", "call", "step", "pack"), (12, 4, 2, 2))[0]
    if kind == "step":
        shape = rng.choice(sorted(model_tools.SHAPES))
        most = {"qwen2.5-0.5b": 24, "llama-3-8b": 8, "llama-3-70b": 2}[shape]
        c = _step("", shape, rng.randint(1, most), rng.choice((1, 1, 2, 3, 4)), _log_int(rng, 16, 2048), rng.random() < 0.5)
    elif kind == "pack":
        c = _pack("", rng.choice((2, 4)), _log_int(rng, 512, 4096), _ragged(rng, _log_int(rng, 512, 4096), 128), rng.choice((64, 128)))
    else:
        bits = rng.choice((2, 4))
        if kind == "call":
            m = rng.randint(1, 4)
        else:
            m = rng.choice((rng.randint(1, 4), rng.randint(5, 16), _log_int(rng, 17, 1000)))
        n = _ragged(rng, _log_int(rng, 128, 28672), 64)
        k = _ragged(rng, _log_int(rng, 512, 28672), 128)
        while n * k > 28672 * 8192:
            n = max(128, n // 2)
        c = _linear("", bits, m, n, k, rng.choice((64, 128, 128, 256 if bits == 2 else 32)), rng.choice(("fp16", "fp16", "bf16")),
                    0 if kind == "call" else rng.choice((0, max(8, k // 100))), 0 if kind == "call" else rng.choice((0, 8, 8, rng.randint(1, 16))),
                    rng.random() < 0.4, kind)
    del c["name"]
    return c


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    g = _generator(seed)
    n, k = case["n"], case["k"]
    w = torch.empty((n, k), dtype=torch.float16, device="cuda").normal_(0, 0.02, generator=g)
    if case["kind"] == "pack":
        rms = torch.empty(k, device="cuda").log_normal_(0, 1, generator=g)
        return {"case": case, "w": w, "rms": rms}
    dtype = DTYPES[case["dtype"]]
    x = torch.empty((case["m"], k), device="cuda").normal_(0, 1, generator=g)
    rms = None
    if case["outliers"]:
        rms = torch.empty(k, device="cuda").log_normal_(0, 1, generator=g)
        x = x * rms
    x = x.to(dtype)
    bias = torch.empty(n, dtype=torch.float16, device="cuda").normal_(0, 0.01, generator=g) if case["bias"] else None
    if case["kind"] == "call":
        pack = pack_groupwise_int2 if case["bits"] == 2 else pack_groupwise_int4
        pw = pack(w, case["group"])
        x = torch.nn.functional.pad(x, (0, pw.padded_k - k))
        return {"case": case, "x": x, "pw": pw, "bias": bias}
    cls = HybridInt2Linear if case["bits"] == 2 else HybridInt4Linear
    if case["outliers"]:
        # the outlier columns are picked with the activation statistics; the codes by magnitude (see ``pack`` for the other way)
        idx = torch.topk(w.float().square().mean(0).sqrt() * rms, snap_outlier_count(case["outliers"], k)).indices
        columns = w[:, idx].contiguous()
        w[:, idx] = 0
        pw = (pack_groupwise_int2 if case["bits"] == 2 else pack_groupwise_int4)(w, case["group"])
        module = cls.from_buffers(pw.packed, pw.scales, k, case["group"], idx.to(torch.int32), columns, bias)
    else:
        source = nn.Linear(k, n, bias=False, device="meta")
        source.weight = nn.Parameter(w, requires_grad=False)
        source.bias = None if bias is None else nn.Parameter(bias, requires_grad=False)
        module = cls(source, case["group"])
    if case["rank"]:
        module.set_residual(torch.empty((n, case["rank"]), device="cuda").normal_(0, 0.01, generator=g),
                            torch.empty((case["rank"], k), device="cuda").normal_(0, 0.01, generator=g))
    return {"case": case, "x": x, "module": module}


def _prepare_step(case, seed):
    device = torch.device("cuda")
    context, batch = case["context"], case["batch"]
    max_len = context + 72                                       # room for the tokens still to be generated
    probs = (0.7, 0.3, 0.0) if case["shape"] == "llama-3-70b" else (0.6, 0.3, 0.1)
    model, _ = model_tools.build_mixed_model_streaming(case["shape"], device, 1, case["layers"], seed, max_len, probs)
    if case["fused"]:
        fuse_decoder_siblings(model)
    g = _generator(seed)
    vocab = model_tools.SHAPES[case["shape"]]["vocab"]
    ids = torch.randint(0, vocab, (batch, context), generator=g, device=device)
    decoder = StaticGraphDecoder(model, batch, max_len, device=device)
    decoder.prefill(ids)
    tok = torch.randint(0, vocab, (batch, 1), generator=g, device=device)
    pos = torch.full((1,), context, dtype=torch.long, device=device)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            decoder.native.step(tok, pos)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = decoder.native.step(tok, pos)
    caches = [t for pair in decoder.native.kv for t in pair]
    return {"case": case, "decoder": decoder, "graph": graph, "tok": tok, "pos": pos, "logits": logits, "caches": caches}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "call":
        call = decode_int2_linear if case["bits"] == 2 else decode_int4_linear
        return call(state["x"], state["pw"], state["bias"])
    if kind == "step":
        state["graph"].replay()
        return {"logits": state["logits"], "caches": state["caches"]}
    pack = pack_groupwise_int2 if case["bits"] == 2 else pack_groupwise_int4
    pw = pack(state["w"], case["group"], state["rms"])
    return [pw.packed, pw.scales]


def _linear_bytes(bits, n, k, group, outliers, rank, bias):
    if bits == 16:
        return n * k * 2 + (n * 2 if bias else 0)
    kpad = -(-k // group) * group
    oc = snap_outlier_count(outliers, k)
    return (n * kpad * bits // 8 + n * (kpad // group) * 2 + (n * oc * 2 + oc * 4 if oc else 0) + (n + k) * rank * 2 + (n * 2 if bias else 0))


def work(case):
    if case["kind"] == "pack":
        n, k = case["n"], case["k"]
        candidates = 13 if case["bits"] == 2 else 11
        return {"bytes": n * k * 2 + _linear_bytes(case["bits"], n, k, case["group"], 0, 0, False) + 4 * k, "flops": 8 * candidates * n * k}
    if case["kind"] == "step":
        s = model_tools.SHAPES[case["shape"]]
        b, layers, h = case["batch"], case["layers"], s["hidden"]
        q, kv = s["heads"] * s["head_dim"], s["kv_heads"] * s["head_dim"]
        probs = {2: 0.7, 4: 0.3} if case["shape"] == "llama-3-70b" else {2: 0.6, 4: 0.3, 16: 0.1}      # expectation over plans
        weights = activations = macs = 0
        for n, k, bias in ((q, h, s["qkv_bias"]), (kv, h, s["qkv_bias"]), (kv, h, s["qkv_bias"]), (h, q, False),
                           (s["inter"], h, False), (s["inter"], h, False), (h, s["inter"], False)):
            weights += sum(p * _linear_bytes(bits, n, k, 128, k // 100, 8, bias) for bits, p in probs.items())
            macs += b * n * k
        cache = 2 * b * kv * (case["context"] + 1) * 2
        head = s["vocab"] * h
        return {"bytes": layers * (weights + cache + 2 * h * 2) + head * 2 + b * (s["vocab"] + h) * 2,
                "flops": 2 * (layers * (macs + 2 * b * q * (case["context"] + 1)) + b * head)}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": _linear_bytes(case["bits"], n, k, case["group"], case["outliers"], case["rank"], case["bias"]) + m * (n + k) * 2,
            "flops": 2 * m * (n * k + case["rank"] * (n + k))}


def tolerance(case):
    if case["kind"] == "pack":
        # candidate scales whose errors agree to the last bits of a 32-bit sum may be picked either way: a handful of groups
        return {"rel": 1e-3, "max": 0.2, "differ": 1e-4}
    if case["kind"] == "step":
        return {"rel": 1e-2}                                     # 16-bit values rounded at every layer of the decoder
    if case["m"] > 16:                                           # weights and the three terms of the sum rounded to 16 bits
        return {"rel": 6e-3 if case["dtype"] == "bf16" else 2e-3}
    return {"rel": 4e-3 if case["dtype"] == "bf16" else 1e-3}    # 16-bit results of 32-bit sums
