"""What the performance of this repository is measured on: the linear layers of decoder models whose
weights are GGUF blocks, driven through `brotensor_b200.ops` as an inference program drives them.

A case is one of four kinds of pass:

  step    one decode step of `layers` layers for `rows` sequences and, with `vocab`, the LM head. A decode
          loop captures its step once and replays it per token, so `prepare` captures and `run` replays.
          fused = False: one call per projection (the op interface of brotensor); fused = True: q/k/v in
          one launch with the RMSNorm of their input, gate/up in one launch with the SwiGLU gate.
  prompt  one chunk of `tokens` prompt tokens: embedding rows gathered from the quantized table, the seven
          projections of each layer, the LM head on the last token. Prompts differ in length, so the
          calls are made one by one and results are allocated by the calls.
  decode  the blocks of one layer's matrices decoded to a dense type (fine-tuning, export, checks).
  call    a single call from Python on a small matrix: latency.

Shapes. A layer has q (hidden x hidden), k and v (kv x hidden), o (hidden x hidden), gate and up
(ffn x hidden) and down (hidden x ffn). K-quant rows are whole 256-element blocks, so hidden and ffn are
multiples of 256 and otherwise arbitrary. `mix` names the formats as GGUF files combine them: "q4_k_m" is
Q4_K with down, LM head and embedding in Q6_K; the others use one format throughout.
"""
from __future__ import annotations

import math

import torch

from brotensor_b200 import ops, synth

_DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_MIX = {"q4_k_m": (synth.Q4_K, synth.Q6_K), "q6_k": (synth.Q6_K, synth.Q6_K), "q8_0": (synth.Q8_0, synth.Q8_0),
        "q5_k": (synth.Q5_K, synth.Q5_K), "q4_0": (synth.Q4_0, synth.Q4_0)}
_STREAMED = ("q4_k_m", "q6_k", "q8_0")


def listed():
    return [
        # One user's chat on an 8B-class model: a decode step of eight layers and the head, call by call in FP32.
        dict(name="step1", kind="step", hidden=4096, ffn=14336, kv=1024, layers=8, vocab=128256, mix="q4_k_m", rows=1, dtype="f32", bias=False, fused=False, repack=False),
        # The same kind of model in a program that uses the fused forms, FP16 activations, down_proj regrouped at load.
        dict(name="step1_fused", kind="step", hidden=4096, ffn=14336, kv=1024, layers=8, vocab=32000, mix="q4_k_m", rows=1, dtype="f16", bias=False, fused=True, repack=True),
        # A smaller model whose widths are not powers of two and whose vocabulary is odd, with q/k/v biases.
        dict(name="step1_ragged", kind="step", hidden=2560, ffn=6912, kv=640, layers=8, vocab=32003, mix="q4_k_m", rows=1, dtype="f16", bias=True, fused=False, repack=False),
        # Six concurrent sequences (a small server).
        dict(name="step6", kind="step", hidden=4096, ffn=14336, kv=1024, layers=4, vocab=32000, mix="q4_k_m", rows=6, dtype="f16", bias=False, fused=False, repack=False),
        # Three sequences on 8-bit weights, BF16 activations.
        dict(name="step3_q8", kind="step", hidden=4096, ffn=12288, kv=1024, layers=4, vocab=32000, mix="q8_0", rows=3, dtype="bf16", bias=False, fused=False, repack=False),
        # A file in one of the formats outside the three main ones.
        dict(name="step1_q5k", kind="step", hidden=4096, ffn=12288, kv=1024, layers=4, vocab=32000, mix="q5_k", rows=1, dtype="f16", bias=False, fused=False, repack=False),
        # A chat turn of a few dozen tokens.
        dict(name="prompt_45", kind="prompt", hidden=4096, ffn=14336, kv=1024, layers=2, vocab=32000, mix="q4_k_m", tokens=45, dtype="f16", bias=False),
        # The usual prefill chunk.
        dict(name="prompt_512", kind="prompt", hidden=4096, ffn=14336, kv=1024, layers=1, vocab=128256, mix="q4_k_m", tokens=512, dtype="f16", bias=False),
        # A long document, ragged length, 8-bit weights.
        dict(name="prompt_2000", kind="prompt", hidden=4096, ffn=14336, kv=1024, layers=1, vocab=32000, mix="q8_0", tokens=2000, dtype="bf16", bias=False),
        # A prompt on one of the other formats.
        dict(name="prompt_96_q5k", kind="prompt", hidden=4096, ffn=12288, kv=1024, layers=1, vocab=32000, mix="q5_k", tokens=96, dtype="f16", bias=False),
        # A layer's weights decoded to BF16.
        dict(name="decode_layer", kind="decode", hidden=4096, ffn=14336, kv=1024, mix="q4_k_m", dtype="bf16"),
        # The smallest call: one projection of one token.
        dict(name="call", kind="call", n=1024, k=4096, fmt="q4_k_m", rows=1, dtype="f16", bias=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _widths(rng, top):
    hidden = 256 * round(_log(rng, 1024, top) / 256)
    ffn = 256 * round(hidden * rng.uniform(2.5, 3.5) / 256)
    kv = 64 * max(1, round(hidden / rng.choice((1, 2, 4, 8)) / 64))
    return dict(hidden=hidden, ffn=ffn, kv=kv)


def draw(rng):
    kind = rng.choice(("step", "step", "step", "prompt", "prompt", "decode", "call"))
    dtype = rng.choice(("f32", "f16", "f16", "bf16"))
    mix = rng.choice(("q4_k_m", "q4_k_m", "q6_k", "q8_0", "q5_k", "q4_0"))
    bias = rng.random() < 0.3
    vocab = int(_log(rng, 8000, 128256))
    if kind == "step":
        w = _widths(rng, 5120)
        rows = rng.choice((1, 1, 1, 2, 3, 4, 5, 6, 7, 8))
        fused = rows == 1 and mix in ("q4_k_m", "q8_0") and rng.random() < 0.5
        per_layer = w["hidden"] * (2 * w["hidden"] + 2 * w["kv"] + 3 * w["ffn"])  # weights
        layers = max(2, min(8, round(1.2e9 / per_layer)))
        return dict(kind=kind, **w, layers=layers, vocab=vocab, mix=mix, rows=rows, dtype=dtype, bias=bias and not fused, fused=fused,
                    repack=fused and w["ffn"] % 2048 == 0)
    if kind == "prompt":
        w = _widths(rng, 4096)
        tokens = int(_log(rng, 9, 2000 if mix in _STREAMED else 128))
        return dict(kind=kind, **w, layers=1 if tokens > 256 else 2, vocab=vocab, mix=mix, tokens=tokens, dtype=dtype, bias=bias)
    if kind == "decode":
        return dict(kind=kind, **_widths(rng, 4096), mix=mix, dtype=dtype)
    k = 256 * round(_log(rng, 512, 8192) / 256)
    return dict(kind=kind, n=int(_log(rng, 64, 8192)), k=k, fmt=mix, rows=rng.choice((1, 1, 2, 5, 16)), dtype=dtype, bias=bias)


# ---- inputs ----------------------------------------------------------------------------------------------

class _Draw:
    """Blocks and activations on the GPU from one seed, with the statistics of brotensor_b200.synth."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def _bytes(self, n, b):
        return torch.randint(-2 ** 31, 2 ** 31, ((n * b + 3) // 4,), dtype=torch.int32, device="cuda", generator=self.g).view(torch.uint8)[:n * b].view(n, b)

    def _scale(self, n, s):
        return (torch.randn(n, 1, device="cuda", generator=self.g).abs() * s).half().view(torch.uint8)

    def weight(self, fmt, rows, k):
        n = rows * (k // synth.BLOCK_ELEMS[fmt])
        w = self._bytes(n, synth.BLOCK_BYTES[fmt])
        if fmt in (synth.Q4_K, synth.Q5_K):
            w[:, 0:2] = self._scale(n, 0.002)
            w[:, 2:4] = self._scale(n, 0.002)
        elif fmt == synth.Q6_K:
            w[:, 192:208] = torch.randint(-32, 32, (n, 16), dtype=torch.int8, device="cuda", generator=self.g).view(torch.uint8)
            w[:, 208:210] = self._scale(n, 0.001)
        else:
            w[:, 0:2] = self._scale(n, 0.005)
        return w.reshape(-1)

    def normal(self, m, k, dtype):
        """Post-norm activations: N(0, 1) with a few channels an order of magnitude larger."""
        x = torch.randn(m, k, device="cuda", generator=self.g)
        x[:, torch.randint(0, k, (max(1, k // 512),), device="cuda", generator=self.g)] *= 8
        return x.to(dtype)

    def gated(self, m, k, dtype):
        """The input of down_proj: silu(gate) * up."""
        a, b = (torch.randn(m, k, device="cuda", generator=self.g) for _ in range(2))
        return (torch.nn.functional.silu(a) * b).to(dtype)


def _layer(case):
    """(name, format, N, K) of a layer's seven matrices."""
    h, f, kv = case["hidden"], case["ffn"], case["kv"]
    a, b = _MIX[case["mix"]]
    return [("q", a, h, h), ("k", a, kv, h), ("v", a, kv, h), ("o", a, h, h), ("gate", a, f, h), ("up", a, f, h), ("down", b, h, f)]


def _biases(d, case, dtype):
    return {n: d.normal(1, rows, dtype).view(-1) if case["bias"] and n in "qkv" else None for n, _, rows, _ in _layer(case)}


def _step_inputs(case, d):
    """Raw GGUF weights and biases of each layer, the head and the activations, in the order they are drawn."""
    dt, m, h, f = _DT[case["dtype"]], case["rows"], case["hidden"], case["ffn"]
    layers = []
    for _ in range(case["layers"]):
        W = {n: d.weight(fmt, rows, k) for n, fmt, rows, k in _layer(case)}
        layers.append((W, _biases(d, case, dt)))
    head = d.weight(_MIX[case["mix"]][1], case["vocab"], h)
    x, a, hf = d.normal(m, h, dt), d.normal(m, h, dt), d.gated(m, f, dt)
    gamma = (torch.rand(h, device="cuda", generator=d.g) + 0.5).to(dt)
    return layers, head, x, a, hf, gamma


def _prepare_step(case, d):
    dt, m = _DT[case["dtype"]], case["rows"]
    h, f, L = case["hidden"], case["ffn"], case["layers"]
    head_fmt = _MIX[case["mix"]][1]
    specs = _layer(case)
    raw, head, x, a, hf, gamma = _step_inputs(case, d)
    layers = []
    for W, B in raw:
        F = {n: fmt for n, fmt, _, _ in specs}
        if case["repack"]:  # a program that never reads the weights back regroups them once, at load
            W["down"], F["down"] = ops.repack(F["down"], W["down"], h, f), ops.repacked_fmt(F["down"], f)
        layers.append((W, F, B))
    yt = torch.float16 if dt == torch.float16 else torch.float32
    names = [("act", f) if n == "gate" else (n, rows) for n, _, rows, _ in specs if n != "up"] if case["fused"] else [(n, rows) for n, _, rows, _ in specs]
    Y = {n: torch.empty(L, m, rows, dtype=yt, device="cuda") for n, rows in names}
    logits = torch.empty(m, case["vocab"], dtype=yt, device="cuda")

    def step():
        for i, (W, F, B) in enumerate(layers):
            if case["fused"]:
                ops.gemv_multi_rmsnorm(F["q"], [W["q"], W["k"], W["v"]], x.view(-1), gamma, 1e-5, [h, case["kv"], case["kv"]], outs=[Y["q"][i], Y["k"][i], Y["v"][i]])
                ops.gemv(F["o"], W["o"], a, h, out=Y["o"][i])
                ops.gemv_swiglu(F["gate"], W["gate"], W["up"], x, f, out=Y["act"][i])
                ops.gemv(F["down"], W["down"], hf, h, out=Y["down"][i])
            else:
                for n, _, rows, _ in specs:
                    ops.gemv(F[n], W[n], a if n == "o" else hf if n == "down" else x, rows, bias=B[n], out=Y[n][i])
        ops.gemv(head_fmt, head, x, case["vocab"], out=logits)

    step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return dict(graph=graph, out=[Y[n] for n, _ in names] + [logits], keep=(layers, head, x, a, hf, gamma))


def _prepare_prompt(case, d):
    dt, t = _DT[case["dtype"]], case["tokens"]
    h, f = case["hidden"], case["ffn"]
    layers = [({n: d.weight(fmt, rows, k) for n, fmt, rows, k in _layer(case)}, _biases(d, case, dt)) for _ in range(case["layers"])]
    fmt = _MIX[case["mix"]][1]
    table, head = d.weight(fmt, case["vocab"], h), d.weight(fmt, case["vocab"], h)
    ids = torch.randint(0, case["vocab"], (t,), dtype=torch.int32, device="cuda", generator=d.g)
    return dict(case=case, dt=dt, layers=layers, table=table, head=head, ids=ids, x=d.normal(t, h, dt), a=d.normal(t, h, dt), hf=d.gated(t, f, dt))


def _run_prompt(s):
    case, dt = s["case"], s["dt"]
    h, fmt = case["hidden"], _MIX[case["mix"]][1]
    out = [ops.embedding_gather(fmt, s["table"], s["ids"], case["vocab"], h, out_dtype=dt)]
    for W, B in s["layers"]:
        for n, f, rows, _ in _layer(case):
            out.append(ops.linear(f, W[n], s["a"] if n == "o" else s["hf"] if n == "down" else s["x"], rows, bias=B[n], out_dtype=dt))
    out.append(ops.linear(fmt, s["head"], s["x"][-1:], case["vocab"], out_dtype=torch.float32))
    return out


def _prepare_call(case, d):
    fmt, dt = _MIX[case["fmt"]][0], _DT[case["dtype"]]
    return dict(kind="call", fmt=fmt, n=case["n"], w=d.weight(fmt, case["n"], case["k"]), x=d.normal(case["rows"], case["k"], dt),
                b=d.normal(1, case["n"], dt).view(-1) if case["bias"] else None)


def prepare(case, seed):
    d = _Draw(seed)
    if case["kind"] == "step":
        return dict(kind="step", **_prepare_step(case, d))
    if case["kind"] == "prompt":
        return dict(kind="prompt", **_prepare_prompt(case, d))
    if case["kind"] == "decode":
        return dict(kind="decode", dt=_DT[case["dtype"]], mats=[(fmt, d.weight(fmt, n, k), n, k) for _, fmt, n, k in _layer(case)])
    return _prepare_call(case, d)


def run(s):
    if s["kind"] == "step":
        s["graph"].replay()
        return s["out"]
    if s["kind"] == "prompt":
        return _run_prompt(s)
    if s["kind"] == "decode":
        return [ops.dequant(fmt, w, n, k, s["dt"]) for fmt, w, n, k in s["mats"]]
    return ops.linear(s["fmt"], s["w"], s["x"], s["n"], bias=s["b"])


# ---- the same passes in 64 bits ---------------------------------------------------------------------------

def _f16(b):
    return b.contiguous().view(torch.float16).double()


def _k_scales(b):
    """The eight 6-bit scales and mins in the 12 bytes of a Q4_K / Q5_K block."""
    s0, s1, s2 = b[:, 4:8], b[:, 8:12], b[:, 12:16]
    sc = torch.cat([s0 & 63, (s2 & 15) | (s0 >> 6) << 4], 1)
    m = torch.cat([s1 & 63, (s2 >> 4) | (s1 >> 6) << 4], 1)
    return sc.double(), m.double()


def _rows64(fmt, raw, n, k):
    """Blocks (the block formats of ggml) -> (n, k) in 64 bits."""
    b = raw.view(-1, synth.BLOCK_BYTES[fmt])
    if fmt == synth.Q8_0:
        w = _f16(b[:, 0:2]) * b[:, 2:].contiguous().view(torch.int8).double()
    elif fmt == synth.Q4_0:
        w = _f16(b[:, 0:2]) * (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).double() - 8)
    elif fmt == synth.Q6_K:
        ql, qh = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 32)
        q = torch.stack([(ql[:, :, j & 1] >> 4 * (j >> 1) & 15) | (qh >> 2 * j & 3) << 4 for j in range(4)], 2).double() - 32
        sc = b[:, 192:208].contiguous().view(torch.int8).double()
        w = q.reshape(-1, 16, 16) * (_f16(b[:, 208:210]) * sc).unsqueeze(2)
    else:
        sc, m = _k_scales(b)
        qs = b[:, -128:].reshape(-1, 4, 1, 32)
        q = torch.cat([qs & 15, qs >> 4], 2).reshape(-1, 8, 32)
        if fmt == synth.Q5_K:
            q = q | torch.stack([b[:, 16:48] >> j & 1 for j in range(8)], 1) << 4
        w = (_f16(b[:, 0:2]) * sc).unsqueeze(2) * q.double() - (_f16(b[:, 2:4]) * m).unsqueeze(2)
    return w.reshape(n, k)


def _linear64(fmt, raw, x, n, bias=None):
    k = x.shape[1]
    y, step = [], max(1, (1 << 24) // k)
    blocks = raw.view(n, -1)
    for r in range(0, n, step):
        part = blocks[r:r + step]
        y.append(x.double() @ _rows64(fmt, part.reshape(-1), part.shape[0], k).T)
    y = torch.cat(y, 1)
    return y if bias is None else y + bias.double()


def exact(case, seed):
    d = _Draw(seed)
    if case["kind"] == "decode":
        return [_rows64(fmt, d.weight(fmt, n, k), n, k) for _, fmt, n, k in _layer(case)]
    if case["kind"] == "call":
        s = _prepare_call(case, d)
        return _linear64(s["fmt"], s["w"], s["x"], s["n"], s["b"])
    fmt = _MIX[case["mix"]][1]
    if case["kind"] == "prompt":
        s = _prepare_prompt(case, d)
        rows = s["table"].view(case["vocab"], -1)[s["ids"].long()]
        out = [_rows64(fmt, rows.reshape(-1), rows.shape[0], case["hidden"])]
        for W, B in s["layers"]:
            out += [_linear64(f, W[n], s["a"] if n == "o" else s["hf"] if n == "down" else s["x"], rows, B[n]) for n, f, rows, _ in _layer(case)]
        return out + [_linear64(fmt, s["head"], s["x"][-1:], case["vocab"])]
    layers, head, x, a, hf, gamma = _step_inputs(case, d)
    x64 = x.double()
    normed = x64 * torch.rsqrt(x64.square().mean(1, keepdim=True) + 1e-5) * gamma.double()
    Y = {}
    for W, B in layers:
        for n, f, rows, _ in _layer(case):
            src = a if n == "o" else hf if n == "down" else normed if case["fused"] and n in "qkv" else x
            Y.setdefault(n, []).append(_linear64(f, W[n], src, rows, B[n]))
    if case["fused"]:
        Y["gate"] = [torch.nn.functional.silu(g) * u for g, u in zip(Y["gate"], Y.pop("up"))]
    return [torch.stack(v) for v in Y.values()] + [_linear64(fmt, head, x, case["vocab"])]


# ---- what a pass cannot do without -----------------------------------------------------------------------

def _size(dtype):
    return 4 if dtype == "f32" else 2


def work(case):
    xs = _size(case["dtype"])
    if case["kind"] == "call":
        fmt, n, k, m = _MIX[case["fmt"]][0], case["n"], case["k"], case["rows"]
        return {"bytes": synth.packed_bytes(fmt, n, k) + xs * m * k + (2 if xs == 2 and case["dtype"] == "f16" else 4) * m * n, "flops": 2 * m * n * k}
    mats = _layer(case)
    if case["kind"] == "decode":
        return {"bytes": sum(synth.packed_bytes(f, n, k) + xs * n * k for _, f, n, k in mats), "flops": 0}
    h, f = case["hidden"], case["ffn"]
    m = case["rows"] if case["kind"] == "step" else case["tokens"]
    ys = (2 if case["dtype"] == "f16" else 4) if case["kind"] == "step" else xs
    rows_out = sum(n for _, _, n, _ in mats) - (f if case.get("fused") else 0)
    b = sum(synth.packed_bytes(fm, n, k) for _, fm, n, k in mats) * case["layers"] + xs * m * (2 * h + f) + ys * m * rows_out * case["layers"]
    fl = sum(2 * m * n * k for _, _, n, k in mats) * case["layers"]
    fmt = _MIX[case["mix"]][1]
    hm = m if case["kind"] == "step" else 1
    b += synth.packed_bytes(fmt, case["vocab"], h) + (ys * m if case["kind"] == "step" else 4) * case["vocab"]
    fl += 2 * hm * case["vocab"] * h
    if case["kind"] == "prompt":  # the gathered rows
        b += m * (synth.packed_bytes(fmt, 1, h) + 4 + xs * h)
    return {"bytes": b, "flops": fl}


def tolerance(case):
    """Decoding blocks is exact. A product carries the rounding of its operands - FP16 weights and activations in
    the GEMM, 15-bit fixed point with a shared exponent in the decode GEMV: up to 3e-4 over a row against a
    64-bit sum for the three main formats, 4e-7 for the two that are multiplied in FP32 - and of the
    result's type (2.1e-4 for FP16, 1.7e-3 for BF16); four times that is stated."""
    if case["kind"] == "decode":
        return "exact"
    result = case["dtype"] if case["kind"] == "prompt" else "f16" if case["dtype"] == "f16" else "f32"
    if result == "bf16":
        return {"rel": 7e-3}
    if result == "f32" and case.get("mix", case.get("fmt")) in ("q5_k", "q4_0"):
        return {"rel": 1e-5}
    return {"rel": 1.2e-3}
