"""The work a program has this library do, as measurable cases.

Three kinds of case:

* ``layers``: one pass of `m` token rows through the quantized part of a few transformer layers (embedding gather,
  then per layer norm, q/k/v projection, output projection with the residual, norm, gated MLP with the residual).
  m = 1 is single-stream decode, 2..8 batched decode, more a prompt. Attention itself is not part of the library, so
  its output is an input here. A program that decodes in a loop keeps the step in a CUDA graph (``graph``) or makes
  the calls one by one in encode-only mode.
* ``q4``: a single 4-bit projection, routed by m as `Q4Weight.matmul` does: GEMV, small-batch GEMM, prefill GEMM.
* ``q8`` / ``q8_signed``: a single 8-bit projection in MLX's format (m <= 8) or with signed codes and f32 tables (m = 1).
"""
from __future__ import annotations

import math

import torch

from tessl_b200 import nn

VOCAB = 32000  # rows of the embedding table of the ``layers`` cases: a pass reads m of them
EPS = 1e-6


def _layers(name, m, hidden, inter, q, kv, layers, group=64, graph=False, banks=False):
    return dict(name=name, kind="layers", m=m, hidden=hidden, inter=inter, q=q, kv=kv, layers=layers, group=group,
                graph=graph, banks=banks)


def _q4(name, m, rows, cols, group=64, bf16=False, resid=False):
    return dict(name=name, kind="q4", m=m, rows=rows, cols=cols, group=group, bf16=bf16, resid=resid)


def listed():
    return [
        # a lone K or V projection of a small layer: nothing but the latency of one call
        _q4("gemv_small", 1, 1024, 1024),
        # single-stream decode of a small dense model, calls made one by one, q/k/v in separate banks
        _layers("decode_eager", 1, 2048, 6144, 2048, 512, 2, banks=True),
        # single-stream decode at the headline width, the step kept in a CUDA graph
        _layers("decode_graph", 1, 4096, 12288, 4096, 1024, 4, graph=True),
        # five streams decoded together at a width that is no power of two, the step kept in a CUDA graph
        _layers("decode_batch_2560", 5, 2560, 9216, 4096, 1024, 2, graph=True),
        # eight streams decoded together, calls made one by one
        _layers("decode_batch", 8, 4096, 12288, 4096, 1024, 2),
        # the logits of one token, and of eight
        _q4("lm_head", 1, 151936, 4096),
        _q4("lm_head_batch", 8, 151936, 4096, bf16=True),
        # a long prompt through the MLP's up projection
        _q4("prefill_up", 2048, 12288, 4096, bf16=True),
        # a short ragged prompt through a down projection
        _q4("prefill_short", 77, 4096, 12288),
        # a middling ragged prompt through whole layers
        _layers("prefill_layer", 509, 2048, 6144, 2048, 512, 1),
        # 8-bit banks: a small batch in MLX's format, and one row with signed codes
        dict(name="q8_batch", kind="q8", m=4, rows=14336, cols=4096, group=64, bf16=True),
        dict(name="q8_signed", kind="q8_signed", m=1, rows=4096, cols=4096, group=64),
    ]


def _between(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    what = rng.choice(("decode", "batch", "prompt", "gemv", "gemm", "prefill", "prefill", "q8", "q8_signed"))
    group = rng.choice((32, 64, 64, 64, 128))
    if what in ("decode", "batch", "prompt"):
        m = {"decode": 1, "batch": rng.randint(2, 8), "prompt": _between(rng, 9, 420)}[what]
        hidden = rng.choice((1024, 2048, 4096)) if m == 1 else _between(rng, 1024, 5120, 256)
        inter = _between(rng, max(2 * hidden, 4352), max(4 * hidden, 6144) if hidden <= 4096 else 17408, 256)
        c = _layers("", m, hidden, inter, _between(rng, 1024, 4096, 256),
                    _between(rng, 256, 1024, 128), rng.randint(1, 3) if m <= 8 else 1, group=group,
                    graph=m <= 8 and rng.random() < 0.6, banks=m == 1 and rng.random() < 0.5)
    elif what in ("gemv", "gemm"):
        m = 1 if what == "gemv" else rng.randint(2, 8)
        cols = rng.choice((1024, 2048, 4096, 4096, 8192, 12288, _between(rng, 1024, 17408, 128)))
        rows = _between(rng, 257, min(151936, (151936 * 4096) // cols))
        c = _q4("", m, rows, cols, group=group, bf16=rng.random() < 0.5, resid=rng.random() < 0.3)
    elif what == "prefill":
        c = _q4("", _between(rng, 9, 2048), _between(rng, 512, 12288), _between(rng, 1024, 4096, 128), group=group,
                bf16=rng.random() < 0.5)
    else:
        c = dict(name="", kind=what, m=rng.randint(1, 8) if what == "q8" else 1, rows=_between(rng, 512, 14336),
                 cols=rng.choice((1024, 2048, 4096, _between(rng, 1024, 4096, 128))), group=rng.choice((32, 64, 64)))
        if what == "q8":
            c["bf16"] = rng.random() < 0.5
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs ---

_runtime = []


def runtime():
    """The process's runtime, in encode-only mode: calls return once they are on the runtime's stream."""
    if not _runtime:
        rt = nn.Runtime()
        rt.set_encode_only(True)
        _runtime.append((rt, torch.cuda.ExternalStream(rt.stream)))
    return _runtime[0]


class _Maker:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.keep = []

    def buf(self, t):
        return nn.GpuBuffer.from_torch(t)

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, device="cuda", generator=self.gen) * (hi - lo) + lo

    def normal(self, *shape, std=1.0):
        return torch.randn(shape, device="cuda", generator=self.gen) * std

    def bytes(self, *shape):
        return torch.randint(0, 256, shape, device="cuda", dtype=torch.uint8, generator=self.gen)

    def bank(self, rows, cols, group):
        """4-bit codes of any value, scales U(0.002, 0.02), biases about -8 scales, as MLX's quantizer leaves them."""
        scale = self.uniform((rows, cols // group), 0.002, 0.02).bfloat16()
        bias = (-8.0 * scale.float() + self.normal(rows, cols // group, std=0.001)).bfloat16()
        packed, sb = self.bytes(rows, cols // 2), torch.stack((scale, bias), dim=-1).contiguous()
        return nn.Q4MlxBank(self.buf(packed), self.buf(sb))


def _empty(*shape, bf16=False):
    return torch.zeros(shape, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)


def _project(rt, bank, x, y, shape, m, resid=None, bf16=False):
    if m == 1:
        nn.gemv_q4_mlx_simd(rt, bank, x, y, shape, resid=resid, y_as_bf16=bf16)
    elif m <= nn.GEMM_Q4_MLX_MAX_M:
        nn.gemm_q4_mlx(rt, bank, x, y, shape, m, resid=resid, y_as_bf16=bf16)
    else:
        nn.gemm_q4_mlx_tensorops(rt, bank, x, y, shape, m, y_as_bf16=bf16)


class _Layers:
    """Weights and buffers of a few layers, and the step over them."""

    def __init__(self, c, seed):
        mk = _Maker(seed)
        self.rt, self.stream = runtime()
        m, h, i, q, kv, g = self.m, self.h, self.i, self.q, self.kv, self.g = tuple(c[k] for k in ("m", "hidden", "inter", "q", "kv", "group"))
        buf = mk.buf
        self.ids = buf(torch.randint(0, VOCAB, (m,), device="cuda", dtype=torch.int32, generator=mk.gen))
        self.table = mk.bank(VOCAB, h, g)
        self.attn = buf(mk.normal(m, q).bfloat16())
        self.layers = []
        for _ in range(c["layers"]):
            w = {"norm1": buf(mk.normal(h, std=0.1)), "norm2": buf(mk.normal(h, std=0.1)), "o": mk.bank(h, q, g),
                 "gate": mk.bank(i, h, g), "up": mk.bank(i, h, g), "down": mk.bank(h, i, g)}
            if c["banks"]:
                w["q"], w["k"], w["v"] = mk.bank(q, h, g), mk.bank(kv, h, g), mk.bank(kv, h, g)
                w["out"] = [_empty(q), _empty(kv), _empty(kv)]
                w["qkv_out"] = nn.QkvOutputs(*(buf(t) for t in w["out"]))
            else:
                w["qkv"] = mk.bank(q + 2 * kv, h, g)
                w["out"] = [_empty(m, q + 2 * kv)]
                w["qkv_out"] = buf(w["out"][0])
            self.layers.append(w)
        self.final = buf(mk.normal(h, std=0.1))
        self.resid_t, self.last_t = _empty(m, h), _empty(m, h, bf16=True)
        self.resid, self.last, self.x = buf(self.resid_t), buf(self.last_t), buf(_empty(m, h, bf16=True))
        self.mid = buf(_empty(m, i, bf16=True))
        if m > 1:
            self.gate, self.up = buf(_empty(m, i)), buf(_empty(m, i))
        if m > nn.GEMM_Q4_MLX_MAX_M:
            self.y = buf(_empty(m, h))
        self.s_qkv, self.s_o, self.s_up, self.s_down = (nn.QuantShape(r, k, g) for r, k in ((q + 2 * kv, h), (h, q), (i, h), (h, i)))
        self.outputs = {"resid": self.resid_t, "last": self.last_t, "qkv": [w["out"] for w in self.layers]}
        torch.cuda.synchronize()
        self.graph = None
        if c["graph"]:
            self.step()  # buffers the library grows on demand are grown before the capture
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=self.stream):
                self.step()

    def step(self):
        rt, m = self.rt, self.m
        nn.embed_lookup_q4_mlx(rt, self.table, self.ids, self.resid, VOCAB, self.h, self.g, m)
        fused = m <= nn.GEMM_Q4_MLX_MAX_M  # those kernels add the residual themselves
        y = self.resid if fused else self.y
        add = False  # y still has to be added to the residual stream
        for w in self.layers:
            self.norm(add, w["norm1"], self.x)
            if "q" in w:
                nn.gemv_q4_mlx_qkv(rt, w["q"], w["k"], w["v"], self.x, w["qkv_out"], self.q, self.kv, self.h, self.g)
            else:
                _project(rt, w["qkv"], self.x, w["qkv_out"], self.s_qkv, m)
            _project(rt, w["o"], self.attn, y, self.s_o, m, resid=self.resid if fused else None)
            self.norm(not fused, w["norm2"], self.x)
            if m == 1:
                nn.gemv_q4_mlx_gate_up_silu(rt, w["gate"], w["up"], self.x, self.mid, self.s_up, True)
            else:
                _project(rt, w["gate"], self.x, self.gate, self.s_up, m)
                _project(rt, w["up"], self.x, self.up, self.s_up, m)
                nn.swiglu(rt, self.gate, self.up, self.mid, m * self.i, True)
            _project(rt, w["down"], self.mid, y, self.s_down, m, resid=self.resid if fused else None)
            add = not fused
        self.norm(add, self.final, self.last)

    def norm(self, add, w, out):
        if add:
            nn.qwen35_add_rms_norm(self.rt, self.y, self.resid, w, out, True, self.m, self.h, EPS)
        else:
            nn.qwen35_rms_norm(self.rt, self.resid, w, out, True, self.m, self.h, EPS)

    def run(self):
        if self.graph is None:
            self.step()
        else:
            with torch.cuda.stream(self.stream):
                self.graph.replay()
        return self.outputs


class _Single:
    """One projection: its bank, its input and its output."""

    def __init__(self, c, seed):
        mk = _Maker(seed)
        rt, _ = runtime()
        m, rows, cols, g = c["m"], c["rows"], c["cols"], c["group"]
        buf, kind, bf16 = mk.buf, c["kind"], c.get("bf16", False)
        self.out = _empty(m, rows, bf16=bf16)
        y, shape = buf(self.out), nn.QuantShape(rows, cols, g)
        if kind == "q4":
            bank, x = mk.bank(rows, cols, g), buf(mk.normal(m, cols).bfloat16())
            resid = buf(mk.normal(m, rows)) if c["resid"] else None
            self.call = lambda: _project(rt, bank, x, y, shape, m, resid=resid, bf16=bf16)
        elif kind == "q8":
            scale = mk.uniform((rows, cols // g), 0.0005, 0.005).bfloat16()
            sb = buf(torch.stack((scale, -128.0 * scale), dim=-1).bfloat16().contiguous())
            codes, x = buf(mk.bytes(rows, cols)), buf(mk.normal(m, cols).bfloat16())
            self.call = lambda: nn.gemm_q8_mlx(rt, codes, sb, x, y, shape, m, bf16)
        else:
            scales, zeros = buf(mk.uniform((rows, cols // g), 0.0005, 0.005)), buf(mk.normal(rows, cols // g, std=4.0))
            codes, x = buf(mk.bytes(rows, cols)), buf(mk.normal(cols))
            self.call = lambda: nn.gemv_q8(rt, codes, scales, zeros, x, y, rows, cols, g)
        torch.cuda.synchronize()

    def run(self):
        self.call()
        return self.out


def prepare(case, seed):
    return (_Layers if case["kind"] == "layers" else _Single)(case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work ---

def _bank_bytes(rows, cols, group, bits=4):
    return rows * cols * bits // 8 + rows * (cols // group) * 4


def work(case):
    m, g = case["m"], case["group"]
    if case["kind"] == "layers":
        h, i, q, kv = case["hidden"], case["inter"], case["q"], case["kv"]
        shapes = ((q + 2 * kv, h), (h, q), (i, h), (i, h), (h, i))
        per = sum(_bank_bytes(r, k, g) for r, k in shapes) + 2 * h * 4 + m * (q * 2 + (q + 2 * kv) * 4)
        return {"bytes": case["layers"] * per + m * (_bank_bytes(1, h, g) + h * 4 + h * 2) + h * 4,
                "flops": 2 * m * case["layers"] * sum(r * k for r, k in shapes)}
    rows, cols = case["rows"], case["cols"]
    if case["kind"] == "q8_signed":
        nbytes = rows * cols + rows * (cols // g) * 8 + cols * 4 + rows * 4
    else:
        nbytes = _bank_bytes(rows, cols, g, 4 if case["kind"] == "q4" else 8) + m * cols * 2
        nbytes += m * rows * ((2 if case["bf16"] else 4) + (4 if case.get("resid") else 0))
    return {"bytes": nbytes, "flops": 2 * m * rows * cols}


def tolerance(case):
    """Another order of the f32 sums, from what each path differs by from the same product in 64 bits: up to 5e-7 (2-norm)
    for the small batches and 1.4e-5 (largest 5e-5) for the prefill GEMM over 12288 columns, whose tensor cores truncate as
    they add. A bf16 result that falls the other way differs by one step, 2^-7 of its value; in a chain of layers, whose
    activations are bf16 between projections, up to 1.2e-3 of the 2-norm."""
    if case["kind"] == "layers":
        return {"rel": 5e-3, "max": 5e-2}
    if case.get("bf16"):
        return {"rel": 1e-3, "max": 1e-2}
    return {"rel": 6e-5, "max": 3e-4} if case["m"] > nn.GEMM_Q4_MLX_MAX_M else {"rel": 5e-6, "max": 5e-5}
