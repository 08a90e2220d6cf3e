"""Performance cases: the work that users of this library have it do, through its public entry points.

Four kinds of call:

- ``linear``: `Context.int4_matmul_dev`, the packed-int4 matmul on device memory as an ONNX runner calls it
  once per MatMul node, with weights that stay resident. A pass walks ``count`` weight matrices of one shape,
  as a decoder walks its layers, so that matrices come from HBM where a model's would.
- ``linear_host``: `Context.int4_matmul`, the same operator with activations and outputs in (page-locked)
  host memory: what a CPU runner that uploaded its weights at load time calls.
- ``int8``: `Context.matmul_integer_dev`, `Context.qlinear_matmul_dev` and
  `Context.int8_matmul_requant_per_channel_dev` (pointwise QLinearConv over NHWC pixels).
- ``decode`` / ``prefill``: one greedy step (a replay of the captured graph) and one prompt pass of
  `Int4Decoder`, the llm-bench loop. The caches of a decode step are filled with seeded rows.

Shapes are those of the repository's benchmark configurations and kernel tables.
"""
from __future__ import annotations

import math

import torch

from yscv_b200 import Context
from yscv_b200.decoder import LLAMA3_70B, TINYLLAMA_1B, Int4Decoder

MODELS = {"tinyllama": TINYLLAMA_1B, "llama70b": LLAMA3_70B}


def listed():
    return [
        # the smallest call: an attention output projection of a 1B decoder for one token; launch latency
        {"name": "w4_m1_2048x2048", "kind": "linear", "m": 1, "n": 2048, "k": 2048, "count": 1},
        # the headline: one token through an MLP matrix of a 7B/8B decoder, matrix after matrix
        {"name": "w4_m1_14336x4096", "kind": "linear", "m": 1, "n": 14336, "k": 4096, "count": 16},
        # a small decode batch through the widest matrix of a 70B decoder
        {"name": "w4_m16_57344x8192", "kind": "linear", "m": 16, "n": 57344, "k": 8192, "count": 1},
        # a prompt whose length is no multiple of any tile
        {"name": "w4_m1000_14336x4096", "kind": "linear", "m": 1000, "n": 14336, "k": 4096, "count": 1},
        # the headline's operator called with host activations and outputs
        {"name": "w4_host_m1_14336x4096", "kind": "linear_host", "m": 1, "n": 14336, "k": 4096, "count": 4},
        # MatMulInteger of a small quantised layer
        {"name": "i8_i32_64x1024x1024", "kind": "int8", "m": 64, "n": 1024, "k": 1024, "out": "i32"},
        # QLinearMatMul prefill
        {"name": "i8_u8_2048x4096x4096", "kind": "int8", "m": 2048, "n": 4096, "k": 4096, "out": "u8"},
        # greedy decoding with a 1B decoder after a prompt of 128: one conversation, a few, a full server batch
        {"name": "tinyllama_decode_b1", "kind": "decode", "model": "tinyllama", "layers": 22, "batch": 1,
         "cached": 200, "kv_int8": False},
        {"name": "tinyllama_decode_b8", "kind": "decode", "model": "tinyllama", "layers": 22, "batch": 8,
         "cached": 200, "kv_int8": False},
        {"name": "tinyllama_decode_b32", "kind": "decode", "model": "tinyllama", "layers": 22, "batch": 32,
         "cached": 200, "kv_int8": False},
        # a full server batch at the 70B layer shape over long contexts (4 of its layers, the whole vocabulary)
        {"name": "llama70b_decode_b64", "kind": "decode", "model": "llama70b", "layers": 4, "batch": 64,
         "cached": 2048, "kv_int8": True},
        # a long prompt at the 70B layer shape (4 of its layers)
        {"name": "llama70b_prefill_2048", "kind": "prefill", "model": "llama70b", "layers": 4, "batch": 1,
         "prompt": 2048, "kv_int8": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear_host", "int8", "int8", "decode", "decode", "prefill"])
    if kind == "linear":
        m = rng.choice([1, _log(rng, 1, 16), _log(rng, 17, 128), _log(rng, 129, 2048)])
        n, k = _log(rng, 256, 57344), 256 * _log(rng, 1, 112)
        if rng.random() < 0.25 and m <= 64:  # a depth that is no multiple of the decode kernel's 256
            k = max(64, k - 32 * rng.randint(1, 7))
        while n * k > 57344 * 8192:
            n //= 2
        while m * n * k > 2048 * 8192 * 28672:
            m //= 2
        count = max(1, min(16, (1 << 29) // (n * k))) if m <= 16 else 1
        return {"kind": kind, "m": m, "n": n, "k": k, "count": count}
    if kind == "linear_host":
        n, k = _log(rng, 512, 28672), 256 * _log(rng, 4, 44)
        return {"kind": kind, "m": rng.choice([1, _log(rng, 1, 64)]), "n": n, "k": k, "count": 4}
    if kind == "int8":
        out = rng.choice(["i32", "u8", "i8"])
        if out == "i8":  # pixels x input channels -> output channels
            return {"kind": kind, "m": _log(rng, 49, 25088), "n": 8 * _log(rng, 8, 256), "k": 8 * _log(rng, 8, 128),
                    "out": out}
        m, n, k = _log(rng, 1, 4096), _log(rng, 64, 11008), _log(rng, 64, 11008)
        return {"kind": kind, "m": m, "n": n, "k": k, "out": out}
    if kind == "decode":
        kv_int8 = rng.random() < 0.5
        if rng.random() < 0.3:
            return {"kind": kind, "model": "llama70b", "layers": rng.randint(2, 4), "batch": _log(rng, 1, 64),
                    "cached": _log(rng, 16, 2048), "kv_int8": kv_int8}
        return {"kind": kind, "model": "tinyllama", "layers": 22, "batch": _log(rng, 1, 64),
                "cached": _log(rng, 16, 1900), "kv_int8": kv_int8}
    model = rng.choice(["tinyllama", "llama70b"])
    prompt = _log(rng, 8, 2048)
    batch = _log(rng, 1, max(1, min(32, 2048 // prompt)))
    return {"kind": kind, "model": model, "layers": 22 if model == "tinyllama" else rng.randint(2, 4), "batch": batch,
            "prompt": prompt, "kv_int8": rng.random() < 0.5}


_PROGRAM = {}


def _program():
    """The stream and the context that a program makes once."""
    if not _PROGRAM:
        _PROGRAM["stream"] = torch.cuda.Stream()
        _PROGRAM["ctx"] = Context(0, stream=_PROGRAM["stream"].cuda_stream)
    return _PROGRAM["ctx"], _PROGRAM["stream"]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def prepare(case, seed):
    ctx, stream = _program()
    with torch.cuda.stream(stream):
        state = {"linear": _prepare_linear, "linear_host": _prepare_linear, "int8": _prepare_int8,
                 "decode": _prepare_decode, "prefill": _prepare_prefill}[case["kind"]](ctx, stream, case, seed)
    stream.synchronize()
    return state


def _prepare_linear(ctx, stream, case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    g = _generator(seed)
    calls = []
    for _ in range(case["count"]):
        w = torch.randn(n, k, device="cuda", generator=g) * 0.02
        packed = torch.empty(n, k // 2, dtype=torch.uint8, device="cuda")
        scales = torch.empty(n, k // 32, device="cuda")
        ctx.pack_int4_dev(w.data_ptr(), n, k, 32, packed.data_ptr(), scales.data_ptr())
        handle = ctx.int4_weight_wrap(packed.data_ptr(), scales.data_ptr(), n, k, 32)
        x = torch.randn(m, k, device="cuda", generator=g)
        y = torch.empty(m, n, device="cuda")
        if case["kind"] == "linear_host":
            x, y = x.cpu().pin_memory(), torch.empty(m, n).pin_memory()
        calls.append({"w": handle, "x": x, "y": y, "keep": (packed, scales)})
    run = _run_linear
    if case["kind"] == "linear_host":
        run = _run_linear_host
        for c in calls:
            c["x_np"], c["y_np"] = c["x"].numpy(), c["y"].numpy()
    return {"run": run, "ctx": ctx, "m": m, "calls": calls}


def _run_linear(s):
    for c in s["calls"]:
        s["ctx"].int4_matmul_dev(c["w"], c["x"].data_ptr(), c["y"].data_ptr(), s["m"])
    return [c["y"] for c in s["calls"]]


def _run_linear_host(s):
    return [s["ctx"].int4_matmul(c["w"], c["x_np"], s["m"], out=c["y_np"]) for c in s["calls"]]


def _prepare_int8(ctx, stream, case, seed):
    m, n, k, out = case["m"], case["n"], case["k"], case["out"]
    g = _generator(seed)
    b = torch.clamp(torch.round(torch.randn(k, n, device="cuda", generator=g) * 28), -127, 127).to(torch.int8)
    s = {"run": _run_int8, "ctx": ctx, "m": m, "out": out, "b": ctx.pack_i8_b_dev(b.data_ptr(), k, n)}
    x = torch.round(torch.randn(m, k, device="cuda", generator=g) * (127 / 3))
    if out == "i8":
        s["a"] = torch.clamp(x, -128, 127).to(torch.int8)
        s["corr"] = torch.randint(-4000, 4000, (n,), dtype=torch.int32, device="cuda", generator=g)
        spread = 0.5 + torch.rand(n, device="cuda", generator=g)
        s["composite"] = (40 / (28 * 42 * math.sqrt(k))) * spread
        s["y"] = torch.empty(m, n, dtype=torch.int8, device="cuda")
    else:
        s["a"] = torch.clamp(x + 128, 0, 255).to(torch.uint8)
        s["rq"] = ctx.requant(40 / (28 * 42 * math.sqrt(k)), 128.0, 0, 255, a_unsigned=True, a_zp=128)
        s["y"] = torch.empty(m, n, dtype=torch.int32 if out == "i32" else torch.uint8, device="cuda")
    return s


def _run_int8(s):
    ctx, a, y = s["ctx"], s["a"].data_ptr(), s["y"].data_ptr()
    if s["out"] == "i32":
        ctx.matmul_integer_dev(a, True, 128, s["b"], s["m"], y)
    elif s["out"] == "u8":
        ctx.qlinear_matmul_dev(a, s["b"], s["m"], s["rq"], y)
    else:
        ctx.int8_matmul_requant_per_channel_dev(a, s["b"], s["m"], s["corr"].data_ptr(), s["composite"].data_ptr(), -2.0, y)
    return s["y"]


def _float_state(dec):
    """The decoder's updated state: its caches, or the row scales of int8 caches. The int8 rows themselves are
    no result to compare: a value next to a rounding boundary of its row's grid lands on either side, and behind
    the first layer of a bf16 chain most values are next to one for some correct summation order."""
    return dec.kscale + dec.vscale if dec.kv_int8 else dec.kcache + dec.vcache


def _prepare_decode(ctx, stream, case, seed):
    cfg, batch, cached = MODELS[case["model"]], case["batch"], case["cached"]
    dec = Int4Decoder(ctx, cfg, batch, cached + 130, stream, seed=seed, layers=case["layers"], kv_int8=case["kv_int8"])
    g = _generator(seed)
    for l in range(case["layers"]):
        for cache in (dec.kcache[l], dec.vcache[l]):
            if case["kv_int8"]:
                cache[:, :cached] = torch.randint(-127, 128, cache[:, :cached].shape, dtype=torch.int8, device="cuda", generator=g)
            else:
                cache[:, :cached].normal_(generator=g)
        if case["kv_int8"]:
            for scale in (dec.kscale[l], dec.vscale[l]):
                scale[:, :cached].uniform_(0.01, 0.03, generator=g)
    tokens = torch.randint(0, cfg.vocab, (batch,), dtype=torch.int32, device="cuda", generator=g)
    pos = torch.full((1,), cached, dtype=torch.int32, device="cuda")
    dec.pos.copy_(pos)
    dec.next_tokens.copy_(tokens)
    logits = dec.forward(dec.next_tokens, 1)
    dec.capture_decode_step()
    written = [c[:, cached] for c in _float_state(dec)]
    return {"run": _run_decode, "dec": dec, "stream": stream, "tokens": tokens, "pos": pos, "out": [logits, *written]}


def _run_decode(s):
    dec = s["dec"]
    with torch.cuda.stream(s["stream"]):
        dec.pos.copy_(s["pos"])
        dec.next_tokens.copy_(s["tokens"])
    dec.decode(1)
    return s["out"]


def _prepare_prefill(ctx, stream, case, seed):
    cfg, batch, prompt = MODELS[case["model"]], case["batch"], case["prompt"]
    dec = Int4Decoder(ctx, cfg, batch, prompt + 130, stream, seed=seed, layers=case["layers"], kv_int8=case["kv_int8"])
    tokens = torch.randint(0, cfg.vocab, (batch, prompt), dtype=torch.int32, device="cuda", generator=_generator(seed))
    written = [c[:, :prompt] for c in _float_state(dec)]
    return {"run": _run_prefill, "dec": dec, "tokens": tokens, "written": written}


def _run_prefill(s):
    s["dec"].reset()
    return [s["dec"].prefill(s["tokens"]), *s["written"]]


def run(state):
    return state["run"](state)


def work(case):
    """Bytes: every weight, activation, cache row and output once. Operations: two per weight and row, and the
    attention's two contractions."""
    if case["kind"] in ("linear", "linear_host"):
        m, n, k, c = case["m"], case["n"], case["k"], case["count"]
        return {"bytes": c * (n * k / 2 + n * k / 8 + 4 * m * (n + k)), "flops": 2.0 * c * m * n * k}
    if case["kind"] == "int8":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": m * k + n * k + m * n * (4 if case["out"] == "i32" else 1), "flops": 2.0 * m * n * k}
    cfg, layers, batch = MODELS[case["model"]], case["layers"], case["batch"]
    seq = case.get("prompt", 1)
    keys = seq * (seq + 1) / 2 if "prompt" in case else case["cached"] + 1  # (query, key) pairs of a head
    d, rows = cfg.head_dim, batch * seq
    weights = layers * ((cfg.n_q + 2 * cfg.n_kv) * d * cfg.hidden + cfg.hidden * cfg.n_q * d + 3 * cfg.mlp * cfg.hidden)
    row = 2 * cfg.n_kv * d * (1 if case["kv_int8"] else 4)
    cache = layers * batch * row * (seq if "prompt" in case else case["cached"] + 1)
    head = cfg.vocab * cfg.hidden
    return {"bytes": weights * 0.625 + 4 * head + cache + 4 * rows * cfg.hidden + 4 * batch * cfg.vocab,
            "flops": 2.0 * weights * rows + 2.0 * head * batch + 4.0 * layers * batch * keys * cfg.n_q * d}


def tolerance(case):
    kind = case["kind"]
    if kind == "int8":
        return "exact"
    if kind in ("linear", "linear_host"):
        # against float64: 5.4e-7 with 32-bit sums up to 16 rows, 2.7e-3 above, where products are bf16
        return {"rel": 2.5e-6} if case["m"] <= 16 else {"rel": 1e-2}
    if case["batch"] * case.get("prompt", 1) > 16:
        # Up to 4 of the 70B or 22 of the 1B layers with bf16 products: the embedding off by 1e-6 moves the logits by
        # 0.004 to 0.016 (bf16 roundings flip), the fp32-exact chain is 0.02 to 0.05 away
        return {"rel": 0.03}
    # 32-bit sums: one-launch step against operator chain, or the embedding off by 1e-6: 1.1e-5 after 22 layers; with
    # int8 caches a value on a rounding boundary moves by a step of its row's grid: 4.5e-5
    return {"rel": 5e-4} if case["kv_int8"] else {"rel": 4.5e-5}
