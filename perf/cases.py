"""Timed workloads of the engine and of the multiply operators it is made of.

A case is one request as a user sends it: a prompt generated from greedily, a host-sampled
conversation, a batch of ragged prompts decoded together, or one Q8_0 multiply through the
operator ABI.  Models are the decoder shapes of ``tuckmill_b200.testing``; their weights are random,
fixed per model, and loaded once (an engine outlives its requests); what a seed chooses is the prompt.

The artifacts behave like trained models in the one way that greedy decoding feels: the next token
wins by a wide margin.  Every token's embedding points at one successor row of the head and the
layers add a disturbance of about the embedding's own size, so a greedy stream does not hang on the
last bit of a sum, while the returned logits still depend on every layer.
"""
from __future__ import annotations

import collections
import dataclasses
import math
import os
import struct
import tempfile

import numpy as np
import torch

from tuckmill_b200 import cuda, engine, testing

# shape, context the engine is loaded for, the same with several sequences, rows of a prefill chunk
# (0: the default), embedding scale (makes the embedding's share of the residual stream about half)
_MODELS = {
    "qwen3-0.6b": (testing.QWEN3_0_6B, 4096, 1024, 0, 0.9),
    "gemma3-1b": (testing.GEMMA3_1B, 4096, 1024, 0, 0.06),
    # the 8B shape with 8 of its 36 layers: the same work per layer, a file that is written in seconds
    "qwen3-8b-8l": (dataclasses.replace(testing.QWEN3_8B, layers=8), 4096, 1024, 2048, 2.6),
}


def _generate(name, model, prompt, new, exact=False, f16=False):
    return {"name": name, "kind": "generate", "model": model, "prompt": prompt, "new": new, "exact": exact, "f16": f16}


def listed():
    return [
        # The first token of a short chat turn: the smallest request there is, all latency.
        _generate("0.6b first token", "qwen3-0.6b", 19, 1),
        # The standard request: 512 tokens in, 256 out.
        _generate("0.6b request", "qwen3-0.6b", 512, 256),
        # A document pasted into the prompt: several prefill chunks, the last one ragged.
        _generate("0.6b long prompt", "qwen3-0.6b", 3001, 8),
        # A caller that samples on the host: every step's logits come back before the next token goes in.
        {"name": "0.6b host sampling", "kind": "sample", "model": "qwen3-0.6b", "prompt": 128, "new": 24},
        # Bit-reproducible serving (prefill equals token-by-token decode).
        _generate("0.6b exact", "qwen3-0.6b", 70, 32, exact=True),
        # The unquantised twin of a model.
        _generate("0.6b f16 weights", "qwen3-0.6b", 64, 32, f16=True),
        # A server's batch: ragged prompts, all sequences decoded together.
        {"name": "0.6b 32 sequences", "kind": "batch", "model": "qwen3-0.6b", "sequences": 32, "prompt": 400, "new": 64},
        # Sliding-window layers, head size 256, GeGLU, a tied 262144-row head.
        _generate("gemma 1b request", "gemma3-1b", 700, 64),
        # Wide matrices: a 2048-token prompt in one chunk, decode bound by the weights' bytes.
        _generate("8b request", "qwen3-8b-8l", 2048, 32),
        {"name": "8b 32 sequences", "kind": "batch", "model": "qwen3-8b-8l", "sequences": 32, "prompt": 200, "new": 48},
        # One multiply through the operator ABI: a small projection of one token, ...
        {"name": "multiply 3072x1024 m1", "kind": "multiply", "rows": 3072, "cols": 1024, "tokens": 1},
        # ... and a wide one of a full prefill chunk.
        {"name": "multiply 12288x4096 m8192", "kind": "multiply", "rows": 12288, "cols": 4096, "tokens": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_one(rng):
    kind = rng.choice(["generate", "generate", "generate", "sample", "batch", "batch", "multiply"])
    model = rng.choice(sorted(_MODELS))
    if kind == "generate":
        form = rng.choice(["", "", "", "exact", "f16"])
        small = form != ""
        prompt = _log_int(rng, 1, 300 if small else 3500)
        if form == "f16":  # rows go to the F16 kernel in slices of 8, 2 and 1
            prompt -= prompt & 4 if prompt > 4 else prompt - 1
        return {"kind": kind, "model": "qwen3-0.6b" if small else model, "prompt": prompt,
                "new": _log_int(rng, 1, 64 if small else 256), "exact": form == "exact", "f16": form == "f16"}
    if kind == "sample":
        return {"kind": kind, "model": model, "prompt": _log_int(rng, 1, 1000), "new": _log_int(rng, 4, 40)}
    if kind == "batch":
        return {"kind": kind, "model": model, "sequences": _log_int(rng, 2, 48), "prompt": _log_int(rng, 4, 600),
                "new": _log_int(rng, 4, 64)}
    # projections and heads of the shapes above, token counts of decode batches and prefill chunks
    rows, cols = rng.choice([(3072, 1024), (4096, 1024), (6144, 1024), (1024, 3072), (1152, 6912), (13824, 1152),
                             (4096, 4096), (12288, 4096), (24576, 4096), (4096, 12288), (151936, 1024)])
    return {"kind": kind, "rows": rows, "cols": cols, "tokens": _log_int(rng, 1, 8192)}


def draw(rng):
    most = max(_cost(work(c)) for c in listed())
    while True:
        case = _draw_one(rng)
        if case["kind"] == "multiply" and case["rows"] * case["tokens"] > 12288 * 8192:
            continue  # the output alone would be larger than the largest listed one's
        if _cost(work(case)) <= most:
            return case


# ---- artifacts ------------------------------------------------------------------------------------

_DEV = "cuda"


def _gen(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(seed)
    return g


def _quants(g, rows, cols):
    return torch.randint(-127, 128, (rows, cols // 32, 32), dtype=torch.int8, device=_DEV, generator=g)


def _scales(g, rows, cols, sigma):
    """One |N(0, sigma)| / 127 per 32-quant block, in f16."""
    return (torch.randn(rows, cols // 32, device=_DEV, generator=g).abs() * (sigma / 127.0)).half()


def _raw(q, d):
    """Raw Q8_0 blocks [rows, cols/32, 34] of quants and scales."""
    return torch.cat([d.unsqueeze(-1).view(torch.uint8), q.view(torch.uint8)], dim=-1)


def _layout(shape):
    """(name, dims) of every tensor in file order; a matrix's dims are [columns, rows]."""
    yield "token_embd.weight", [shape.hidden, shape.vocab]
    yield "output_norm.weight", [shape.hidden]
    if not shape.tied_head:
        yield "output.weight", [shape.hidden, shape.vocab]
    for layer in range(shape.layers):
        yield from ((name, [cols, rows]) for name, rows, cols in shape.matrices(layer))
        yield from ((name, [n]) for name, n in shape.norms(layer))


def _values(shape, embed_sigma):
    """The tensors of _layout in its order: (quants, scales) of a matrix, a vector of a norm."""
    g = _gen(1)
    q, d = _quants(g, shape.vocab, shape.hidden), _scales(g, shape.vocab, shape.hidden, embed_sigma)
    last = torch.ones(shape.hidden, device=_DEV)
    if shape.tied_head:
        # Pairs (v, v ^ 1) differ by the signs the final norm applies: each names the other next.
        sign = (1 - 2 * torch.randint(0, 2, (shape.hidden,), device=_DEV, generator=g)).to(torch.int8)
        q[1::2] = q[0::2] * sign.view(-1, 32)
        d[1::2] = d[0::2]
        last = sign.float()
    for name, dims in _layout(shape):
        if name == "token_embd.weight":
            yield q, d
        elif name == "output.weight":  # row v is the embedding of the token that v follows
            before = torch.randperm(shape.vocab, device=_DEV, generator=g)
            yield q[before], (d[before].float() * (0.02 / embed_sigma)).half()
        elif len(dims) == 2:
            yield _quants(g, dims[1], dims[0]), _scales(g, dims[1], dims[0], 0.02)
        else:
            v = 1.0 + 0.1 * torch.randn(dims[0], device=_DEV, generator=g)
            yield v * last if name == "output_norm.weight" else v * 0.1 if ".post_" in name else v


def _write_gguf(path, shape, embed_sigma, f16):
    text = lambda s: struct.pack("<Q", len(s)) + s.encode()  # noqa: E731
    meta = {"block_count": shape.layers, "context_length": shape.context, "embedding_length": shape.hidden,
            "feed_forward_length": shape.ffn, "attention.head_count": shape.heads,
            "attention.head_count_kv": shape.kv_heads, "attention.key_length": shape.head_dim,
            "attention.value_length": shape.head_dim, "attention.layer_norm_rms_epsilon": float(shape.eps),
            "rope.freq_base": float(shape.rope_base)}
    if shape.arch == "gemma3":
        meta["attention.sliding_window"] = shape.window
    layout = list(_layout(shape))
    head = struct.pack("<IIQQ", 0x46554747, 3, len(layout), len(meta) + 1)
    head += text("general.architecture") + struct.pack("<I", 8) + text(shape.arch)
    for key, v in meta.items():
        head += text(shape.arch + "." + key)
        head += struct.pack("<If", 6, v) if isinstance(v, float) else struct.pack("<II", 4, v)
    off = 0
    for name, dims in layout:
        kind = testing.GGML_F32 if len(dims) == 1 else testing.GGML_F16 if f16 else testing.GGML_Q8_0
        size = dims[0] * 4 if len(dims) == 1 else dims[0] * dims[1] * 2 if f16 else dims[1] * (dims[0] // 32) * 34
        head += text(name) + struct.pack("<I%dQIQ" % len(dims), len(dims), *dims, kind, off)
        off += size + -size % 32
    with open(path, "wb") as f:
        f.write(head + b"\0" * (-len(head) % 32))
        for v in _values(shape, embed_sigma):
            data = v if torch.is_tensor(v) else v[0].half() * v[1].unsqueeze(-1) if f16 else _raw(*v)
            host = data.reshape(-1).view(torch.uint8).cpu().numpy()
            host.tofile(f)
            f.write(b"\0" * (-host.size % 32))


_ENGINES = collections.OrderedDict()  # the server's loaded models, the longest unused one given up first
_MOST_ENGINES = 8


def _engine(case):
    key = (case["model"], bool(case.get("exact")), bool(case.get("f16")), case.get("sequences", 1))
    if key in _ENGINES:
        _ENGINES.move_to_end(key)
        return _ENGINES[key]
    shape, context, batch_context, chunk, embed_sigma = _MODELS[case["model"]]
    while len(_ENGINES) >= _MOST_ENGINES:
        _ENGINES.popitem(last=False)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "model.gguf")
        _write_gguf(path, shape, embed_sigma, key[2])
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        _ENGINES[key] = engine.Engine(path, context=context if key[3] == 1 else batch_context, exact=key[1],
                                      sequences=key[3], prefill_batch=chunk)
    return _ENGINES[key]


# ---- the cases ------------------------------------------------------------------------------------


class _DeviceArray:
    """A library buffer as torch sees it, for filling it and for reading it where it lies."""

    def __init__(self, buf, shape):
        self._buf = buf  # keeps the storage
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (buf.device_ptr(), False),
                                         "version": 3}


_CONTEXT = []


def _prepare_multiply(case, seed):
    if not _CONTEXT:
        _CONTEXT.append(cuda.CudaContext(0))
    ctx, (m, rows, cols) = _CONTEXT[0], (case["tokens"], case["rows"], case["cols"])
    g = _gen(seed)
    raw = _raw(_quants(g, rows, cols), _scales(g, rows, cols, 0.02)).cpu().numpy()
    w = ctx.q8_0_matrix(raw, rows, cols)
    x, y = ctx.buffer(m * cols * 4), ctx.buffer(m * rows * 4)
    torch.as_tensor(_DeviceArray(x, (m, cols)), device=_DEV).copy_(torch.randn(m, cols, device=_DEV, generator=g))
    torch.cuda.synchronize()
    return {"case": case, "ctx": ctx, "w": w, "x": x, "y": y,
            "out": torch.as_tensor(_DeviceArray(y, (m, rows)), device=_DEV)}


def _lengths(case):
    """Ragged prompt lengths of a batch, from a quarter of the longest to the longest."""
    n = case["prompt"]
    return [max(1, n - int(0.75 * n * ((s * 0.6180339887) % 1.0))) for s in range(case["sequences"])]


def prepare(case, seed):
    if case["kind"] == "multiply":
        return _prepare_multiply(case, seed)
    eng = _engine(case)
    rng = np.random.default_rng(seed)
    ids = lambda n: rng.integers(0, eng.vocab, n, dtype=np.uint32)  # noqa: E731
    if case["kind"] == "batch":
        return {"case": case, "engine": eng, "prompts": [ids(n) for n in _lengths(case)]}
    return {"case": case, "engine": eng, "prompt": ids(case["prompt"]), "forced": ids(case["new"])}


def run(state):
    case = state["case"]
    if case["kind"] == "multiply":
        args = (state["w"], state["x"], state["y"], case["rows"], case["cols"])
        if case["tokens"] == 1:
            state["ctx"].q8_0_gemv(*args)
        else:
            state["ctx"].q8_0_gemm_mma(*args, case["tokens"])
        return state["out"]
    eng = state["engine"]
    if case["kind"] == "batch":
        tokens, _ = eng.generate_batch(state["prompts"], case["new"])
        return {"tokens": tokens[:32], "more tokens": [np.concatenate(tokens[32:])] if len(tokens) > 32 else [],
                "logits of sequence 0": eng.logits()}
    if case["kind"] == "sample":
        eng.reset()
        eng.prefill(state["prompt"])
        return [eng.logits()] + [eng.step(int(t)) for t in state["forced"]]
    tokens, _ = eng.generate(state["prompt"], case["new"])
    return {"tokens": tokens, "logits": eng.logits()}


def work(case):
    """Weights once for every pass that depends on the one before it (a prefill is one such pass, a decode
    step another: on-chip memory does not hold a model), the cached keys and values every step reads,
    inputs and results once; two operations a weight and token, four a cached position and head element."""
    if case["kind"] == "multiply":
        m, rows, cols = case["tokens"], case["rows"], case["cols"]
        return {"bytes": rows * (cols // 32) * 34 + 4 * m * (rows + cols), "flops": 2 * m * rows * cols}
    s = _MODELS[case["model"]][0]
    per = 2.0 if case.get("f16") else 34 / 32
    layer_weights = sum(rows * cols for _, rows, cols in s.matrices(0)) * s.layers
    head_weights = s.vocab * s.hidden
    lengths = _lengths(case) if case["kind"] == "batch" else [case["prompt"]]
    steps = case["new"] if case["kind"] == "sample" else case["new"] - 1
    # a sixth of a windowed model's layers see every position
    full = s.layers if not s.window else s.layers // 6
    seen = lambda p: full * p + (s.layers - full) * min(p, s.window or p)  # noqa: E731  positions over all layers
    kv_row, head_width = 2 * 2 * s.kv_heads * s.head_dim, s.heads * s.head_dim
    nbytes = (layer_weights + head_weights) * per * (1 + steps)
    flops = 0.0
    for n in lengths:
        chunk_seen = sum(seen(p + 1) for p in range(n))
        step_seen = sum(seen(n + i + 1) for i in range(steps))
        nbytes += kv_row * (s.layers * (n + steps) + step_seen)
        flops += 2.0 * layer_weights * (n + steps) + 2.0 * head_weights * (1 + steps) + 4.0 * head_width * (chunk_seen + step_seen)
    rows_out = 1 + (steps if case["kind"] == "sample" else 0)
    return {"bytes": nbytes + 4.0 * s.vocab * rows_out, "flops": flops}


def _cost(w):
    return max(w["bytes"], w["flops"] / 200)


def tolerance(case):
    if case["kind"] == "multiply":
        # one token: f32 products and sums; more: operands rounded to f16 once each, f32 sums
        return {"rel": 1e-5 if case["tokens"] == 1 else 1e-3}
    if case.get("exact") or case.get("f16"):
        # f32 arithmetic; a last-bit difference can move a cached key or value by one f16 step
        return {"rel": 3e-4, "differ": 0.002}
    # f16 operands in every prefill and batch multiply, carried through all layers
    return {"rel": 5e-3, "differ": 0.002}
