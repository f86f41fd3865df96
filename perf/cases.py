"""The work that is timed: attention forward (prefill, cross attention, decode against a key/value cache, FP8), attention
forward + backward, the H2O score, linear layers with fused epilogues, batched products, rowwise programs, and a Llama-style
decoder layer compiled through ``heddle_b200.frontend.tilelang_backend``.

Sizes are those of this repository's own configurations (heddle_b200/bench_configs.py, tests/) or generic ones.  ``listed()``
names twelve of them, ``draw()`` gives more of the same ranges.  ``prepare`` makes what a program has in hand before the call,
``run`` is one pass through the public entry points.
"""
from __future__ import annotations

import math

import torch

from heddle_b200 import ops
from heddle_b200.frontend import tilelang_backend

# every layer shape is compiled once per process, however many there are
torch._dynamo.config.recompile_limit = 256
torch._dynamo.config.accumulated_recompile_limit = 1024

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_MAX_FLOPS = 4.0e12  # of a drawn case: below the largest listed one
_MAX_BYTES = 2.0e9


# ------------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------------
def _attention(B, Hq, Hkv, Sq, Skv, D, dtype, causal, layout="bhsd", lse=False, capacity=0):
    """``capacity``: rows of the key/value buffers that the call sees a prefix of (0: exactly Skv rows)."""
    return dict(kind="attention", B=B, Hq=Hq, Hkv=Hkv, Sq=Sq, Skv=Skv, D=D, dtype=dtype, causal=causal, layout=layout, lse=lse,
                capacity=capacity)


def _train(B, Hq, Hkv, Sq, Skv, D, dtype, causal, layout="bhsd"):
    return dict(kind="train", B=B, Hq=Hq, Hkv=Hkv, Sq=Sq, Skv=Skv, D=D, dtype=dtype, causal=causal, layout=layout)


def _h2o(B, Hq, Hkv, S, D, dtype):
    return dict(kind="h2o", B=B, Hq=Hq, Hkv=Hkv, Sq=S, Skv=S, D=D, dtype=dtype, causal=True)


def _linear(M, N, K, epilogue, dtype, row_scale=False, bias=False, residual=False):
    return dict(kind="linear", M=M, N=N, K=K, epilogue=epilogue, dtype=dtype, row_scale=row_scale, bias=bias, residual=residual)


def _bmm(B, M, N, K, dtype, b_layout):
    """``b_layout``: "kn" = row-major [B, K, N] storage, "nk" = a transposed view of [B, N, K] storage."""
    return dict(kind="bmm", B=B, M=M, N=N, K=K, dtype=dtype, b_layout=b_layout)


def _rowwise(rows, cols, program, dtype):
    return dict(kind="rowwise", rows=rows, cols=cols, program=program, dtype=dtype)


def _layer(B, S, hidden, heads, inter):
    return dict(kind="layer", B=B, S=S, hidden=hidden, heads=heads, inter=inter, dtype="bf16")


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # prompt processing, the headline shape of bench.py
        named("prefill causal", _attention(4, 32, 32, 4096, 4096, 128, "bf16", True)),
        # quantised long-context prompt processing (configuration 4 of bench_configs.py)
        named("prefill fp8", _attention(4, 32, 32, 8192, 8192, 128, "e4m3", False)),
        # the smallest calls: a short ragged sequence of a small model, one launch per call
        named("short ragged", _attention(1, 8, 8, 197, 197, 64, "fp16", False, layout="bshd")),
        # one new token per sequence against a grouped-query cache that is not full
        named("decode gqa", _attention(16, 64, 8, 1, 6001, 128, "bf16", True, capacity=8192)),
        # attention of one training step of a large model
        named("train causal", _train(4, 32, 32, 4096, 4096, 128, "bf16", True)),
        # attention of a training step of a small model: ragged, head_dim 64, (B, S, H, D) tensors
        named("train ragged", _train(8, 12, 12, 577, 577, 64, "fp16", False, layout="bshd")),
        # attention with the H2O cache-eviction score, grouped queries, ragged prompt
        named("h2o gqa", _h2o(2, 32, 8, 3000, 128, "bf16")),
        # the gate / up projection of a decode step: few rows, every weight read once
        named("decode swiglu", _linear(24, 2 * 11008, 4096, "swiglu", "bf16", row_scale=True)),
        # per-head score-like products (bmm of bench_configs.py)
        named("batched product", _bmm(64, 2048, 2048, 128, "bf16", "kn")),
        # a normalisation with two row reductions over a step's activations
        named("rowwise norm", _rowwise(16384, 4096, "norm", "bf16")),
        # the decoder layer of bench_configs.py on a full batch of prompts, and on one short prompt
        named("layer prompts", _layer(8, 2048, 4096, 32, 11008)),
        named("layer short", _layer(1, 120, 4096, 32, 11008)),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    v = max(lo, min(hi, v))
    return max(multiple, v // multiple * multiple) if multiple > 1 else v


def _draw_once(rng):
    kind = rng.choice(["prefill", "prefill", "fp8", "decode", "decode", "train", "train", "h2o", "linear", "linear", "bmm", "rowwise",
                       "layer"])
    dtype = rng.choice(["bf16", "fp16"])
    D = rng.choice([64, 128, 128])
    Hkv = rng.choice([1, 2, 4, 8, 12, 16, 32])
    group = rng.choice([1, 1, 2, 4, 8])
    layout = rng.choice(["bhsd", "bshd"])
    causal = rng.random() < 0.6
    if kind == "prefill":
        Sq = _log_int(rng, 16, 8192)
        Skv = Sq if rng.random() < 0.6 else Sq + _log_int(rng, 1, 4096)
        return _attention(_log_int(rng, 1, 16), Hkv * group, Hkv, Sq, Skv, D, dtype, causal, layout, rng.random() < 0.3)
    if kind == "fp8":
        Sq = _log_int(rng, 256, 8192)
        return _attention(_log_int(rng, 1, 8), Hkv * group, Hkv, Sq, Sq, 128, "e4m3", causal)
    if kind == "decode":
        Skv = _log_int(rng, 64, 32768)
        Sq = min(Skv, rng.choice([1, 1, 1, 2, 3, 4, 8]))
        return _attention(_log_int(rng, 1, 64), Hkv * group, Hkv, Sq, Skv, D, dtype, True, layout, False,
                          Skv + rng.choice([0, _log_int(rng, 1, 2048)]))
    if kind == "train":
        Sq = _log_int(rng, 64, 8192)
        return _train(_log_int(rng, 1, 16), Hkv * group, Hkv, Sq, Sq, D, dtype, causal, layout)
    if kind == "h2o":
        return _h2o(_log_int(rng, 1, 8), Hkv * group, Hkv, _log_int(rng, 64, 8192), D, dtype)
    if kind == "linear":
        M, K = _log_int(rng, 1, 16384), _log_int(rng, 512, 12288, 8)
        epilogue = rng.choice(["none", "none", "silu", "gelu_tanh", "swiglu"])
        N = _log_int(rng, 512, 16384, 16) * (2 if epilogue == "swiglu" else 1)
        plain = epilogue == "none"
        return _linear(M, N, K, epilogue, dtype, rng.random() < 0.3, rng.random() < 0.3, plain and rng.random() < 0.5)
    if kind == "bmm":
        return _bmm(_log_int(rng, 2, 128), _log_int(rng, 16, 4096), _log_int(rng, 64, 4096, 8), _log_int(rng, 64, 2048, 8), dtype,
                    rng.choice(["kn", "nk"]))
    if kind == "rowwise":
        return _rowwise(_log_int(rng, 16, 65536), _log_int(rng, 128, 16384, 8), rng.choice(["norm", "silu_mul", "softmax"]), dtype)
    heads = rng.choice([8, 16, 32])
    return _layer(_log_int(rng, 1, 8), _log_int(rng, 16, 2048), 128 * heads, heads, 344 * heads)


def draw(rng):
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["flops"] <= _MAX_FLOPS and w["bytes"] <= _MAX_BYTES:
            return case


# ------------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------------
class _DecoderLayer(torch.nn.Module):
    """Pre-norm Llama block (RMSNorm, rotate-half RoPE, causal attention, SwiGLU); the rotary tables are buffers."""

    def __init__(self, hidden, heads, inter, positions):
        super().__init__()

        def lin(i, o):
            return torch.nn.Linear(i, o, bias=False)

        self.hidden, self.heads, self.head_dim = hidden, heads, hidden // heads
        self.wq, self.wk, self.wv, self.wo = lin(hidden, hidden), lin(hidden, hidden), lin(hidden, hidden), lin(hidden, hidden)
        self.wg, self.wu, self.wd = lin(hidden, inter), lin(hidden, inter), lin(inter, hidden)
        self.g1, self.g2 = torch.nn.Parameter(torch.ones(hidden)), torch.nn.Parameter(torch.ones(hidden))
        half = self.head_dim // 2
        self.register_buffer("cos", torch.empty(positions, half))
        self.register_buffer("sin", torch.empty(positions, half))

    def fill(self, gen):
        with torch.no_grad():
            for p in self.parameters():
                if p.dim() == 2:
                    p.normal_(0.0, 0.02, generator=gen)
                else:
                    p.uniform_(0.5, 1.5, generator=gen)
            half = self.head_dim // 2
            inv = 1.0 / (10000.0 ** (torch.arange(half, dtype=torch.float32, device=self.cos.device) / half))
            angle = torch.arange(self.cos.shape[0], dtype=torch.float32, device=self.cos.device)[:, None] * inv[None, :]
            self.cos.copy_(angle.cos())
            self.sin.copy_(angle.sin())
        return self.requires_grad_(False)

    @staticmethod
    def norm(x, g):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * g

    def rope(self, x):
        d = self.head_dim // 2
        x1, x2 = x[..., :d], x[..., d:]
        return torch.cat([x1 * self.cos - x2 * self.sin, x2 * self.cos + x1 * self.sin], dim=-1)

    def forward(self, x):
        B, S, _ = x.shape
        h = self.norm(x, self.g1)
        q, k, v = (w(h).view(B, S, self.heads, self.head_dim).transpose(1, 2) for w in (self.wq, self.wk, self.wv))
        a = torch.nn.functional.scaled_dot_product_attention(self.rope(q), self.rope(k), v, is_causal=True)
        x = x + self.wo(a.transpose(1, 2).reshape(B, S, self.hidden))
        h = self.norm(x, self.g2)
        return x + self.wd(torch.nn.functional.silu(self.wg(h)) * self.wu(h))


_NORM = (("load", "input", 0, 0.0), ("reduce_mean", None, 0, 0.0), ("sub", "reduced", 0, 0.0), ("store_tmp", None, 0, 0.0),
         ("mul", "tmp", 0, 0.0), ("reduce_mean", None, 1, 0.0), ("load", "reduced", 1, 0.0), ("add", "imm", 0, 1e-5),
         ("rsqrt", None, 0, 0.0), ("mul", "tmp", 0, 0.0), ("store_out", None, 0, 0.0))
_SILU_MUL = (("load", "input", 0, 0.0), ("silu", None, 0, 0.0), ("mul", "input", 1, 0.0), ("store_out", None, 0, 0.0))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def heads(H, S, dtype, capacity=0):
        """A [B, H, S, D] (or [B, S, H, D]) tensor, a prefix of a longer buffer when ``capacity`` says so."""
        B, D, rows = case["B"], case["D"], max(S, capacity)
        if case.get("layout") == "bshd":
            return randn(B, rows, H, D).to(dtype)[:, :S]
        return randn(B, H, rows, D).to(dtype)[:, :, :S]

    kind, c = case["kind"], case
    state = dict(case)
    if kind in ("attention", "train", "h2o"):
        fp8 = c["dtype"] == "e4m3"
        dtype = torch.float32 if fp8 else _DTYPES[c["dtype"]]
        q = heads(c["Hq"], c["Sq"], dtype)
        k, v = (heads(c["Hkv"], c["Skv"], dtype, c.get("capacity", 0)) for _ in range(2))
        if fp8:
            scales = [float(t.abs().max()) / 448.0 for t in (q, k, v)]
            q, k, v = ((t / s).to(torch.float8_e4m3fn) for t, s in zip((q, k, v), scales))
            state["scales"] = tuple(scales)
        state.update(q=q, k=k, v=v)
        if kind == "train":
            state["grad"] = heads(c["Hq"], c["Sq"], dtype)
    elif kind == "linear":
        dtype, n_out = _DTYPES[c["dtype"]], c["N"] // 2 if c["epilogue"] == "swiglu" else c["N"]
        state["x"] = randn(c["M"], c["K"]).to(dtype)
        state["w"] = (randn(c["N"], c["K"]) * 0.02).to(dtype)
        state["row_scale_t"] = torch.rand(c["M"], generator=gen, device="cuda") + 0.5 if c["row_scale"] else None
        state["bias_t"] = randn(c["N"]).to(dtype) if c["bias"] else None
        state["residual_t"] = randn(c["M"], n_out).to(dtype) if c["residual"] else None
    elif kind == "bmm":
        dtype = _DTYPES[c["dtype"]]
        state["a"] = randn(c["B"], c["M"], c["K"]).to(dtype)
        if c["b_layout"] == "kn":
            state["b"] = randn(c["B"], c["K"], c["N"]).to(dtype)
        else:
            state["b"] = randn(c["B"], c["N"], c["K"]).to(dtype).transpose(1, 2)
    elif kind == "rowwise":
        dtype = _DTYPES[c["dtype"]]
        state["inputs"] = [randn(c["rows"], c["cols"]).to(dtype) for _ in range(2 if c["program"] == "silu_mul" else 1)]
    elif kind == "layer":
        dtype = _DTYPES[c["dtype"]]
        with torch.device("cuda"):
            prev = torch.get_default_dtype()
            torch.set_default_dtype(dtype)
            try:
                layer = _DecoderLayer(c["hidden"], c["heads"], c["inter"], c["S"])
            finally:
                torch.set_default_dtype(prev)
        layer.fill(gen)
        state["layer"] = torch.compile(layer, backend=tilelang_backend, dynamic=False)
        state["x"] = randn(c["B"], c["S"], c["hidden"]).to(dtype)
    else:
        raise ValueError(kind)
    return state


# ------------------------------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------------------------------
def run(state):
    s, kind = state, state["kind"]
    if kind == "attention":
        if "scales" in s:
            return ops.fa_fwd(s["q"], s["k"], s["v"], causal=s["causal"], layout=s["layout"], scales=s["scales"])
        return ops.fa_fwd(s["q"], s["k"], s["v"], causal=s["causal"], layout=s["layout"], return_lse=s["lse"])
    if kind == "train":
        out, lse = ops.fa_fwd(s["q"], s["k"], s["v"], causal=s["causal"], layout=s["layout"], return_lse=True)
        dq, dk, dv = ops.fa_bwd(s["q"], s["k"], s["v"], out, s["grad"], lse, causal=s["causal"], layout=s["layout"])
        return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if kind == "h2o":
        out, lse = ops.fa_fwd(s["q"], s["k"], s["v"], causal=True, return_lse=True)
        return out, ops.h2o_score(s["q"], s["k"], lse, causal=True)
    if kind == "linear":
        return ops.gemm_epilogue(s["x"], s["w"], s["epilogue"], bias=s["bias_t"], row_scale=s["row_scale_t"], residual=s["residual_t"])
    if kind == "bmm":
        return ops.bmm(s["a"], s["b"])
    if kind == "rowwise":
        if s["program"] == "softmax":
            return ops.row_softmax(s["inputs"][0], 0.125)
        return ops.rowwise_program(_NORM if s["program"] == "norm" else _SILU_MUL, s["inputs"])
    return s["layer"](s["x"])


# ------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations may be apart
# ------------------------------------------------------------------------------------------------------------------------
def _pairs(c):
    """(query, key) pairs that take part, of one head."""
    Sq, Skv = c["Sq"], c["Skv"]
    if not c["causal"]:
        return Sq * Skv
    return Sq * (Skv - Sq) + Sq * (Sq + 1) // 2


def work(case):
    c, kind = case, case["kind"]
    if kind in ("attention", "train", "h2o"):
        es = 1 if c["dtype"] == "e4m3" else 2
        q = c["B"] * c["Hq"] * c["Sq"] * c["D"]
        kv = c["B"] * c["Hkv"] * c["Skv"] * c["D"]
        product = 2.0 * c["B"] * c["Hq"] * _pairs(c) * c["D"]  # one of Q K^T, P V, ...
        stats = 4.0 * c["B"] * c["Hq"] * c["Sq"]
        if kind == "train":  # q, k, v, dO in; O, LSE, dQ, dK, dV out
            return {"bytes": 2.0 * (4 * q + 4 * kv) + stats, "flops": 7 * product}
        if kind == "h2o":  # Q K^T, P V and the column sums of P; the score is [B, Hq, Skv] fp32
            return {"bytes": 2.0 * (2 * q + 2 * kv) + 4.0 * c["B"] * c["Hq"] * c["Skv"], "flops": 2 * product}
        return {"bytes": float(es * q + 2 * es * kv + 2 * q) + (stats if c["lse"] else 0.0), "flops": 2 * product}
    if kind == "linear":
        n_out = c["N"] // 2 if c["epilogue"] == "swiglu" else c["N"]
        extra = (4.0 * c["M"] if c["row_scale"] else 0) + (2.0 * c["N"] if c["bias"] else 0) + (2.0 * c["M"] * n_out if c["residual"] else 0)
        return {"bytes": 2.0 * (c["M"] * c["K"] + c["N"] * c["K"] + c["M"] * n_out) + extra, "flops": 2.0 * c["M"] * c["N"] * c["K"]}
    if kind == "bmm":
        return {"bytes": 2.0 * c["B"] * (c["M"] * c["K"] + c["K"] * c["N"] + c["M"] * c["N"]), "flops": 2.0 * c["B"] * c["M"] * c["N"] * c["K"]}
    if kind == "rowwise":
        n = c["rows"] * c["cols"]
        return {"bytes": 2.0 * n * (3 if c["program"] == "silu_mul" else 2), "flops": 0.0}
    rows, h, inter = c["B"] * c["S"], c["hidden"], c["inter"]
    weights = 4 * h * h + 3 * h * inter
    pairs = c["S"] * (c["S"] + 1) // 2
    return {"bytes": 2.0 * (weights + 2 * h + 2 * rows * h), "flops": 2.0 * rows * weights + 4.0 * c["B"] * pairs * h}


def tolerance(case):
    """About four times the distance from the same path in fp64 (measured at the listed sizes; the figures in brackets)."""
    kind, dtype = case["kind"], case["dtype"]
    if dtype == "e4m3":  # P in e4m3 [rel 2.7e-2, max 0.14]: the cap of what can be stated
        return {"rel": 3e-2, "max": 0.6}
    if kind in ("rowwise", "linear", "bmm"):  # fp32 arithmetic, one rounding at the store [bf16 1.7e-3, 3.9e-3; fp16 2.2e-4, 4.9e-4]
        return {"rel": 6.6e-3, "max": 1.6e-2} if dtype == "bf16" else {"rel": 9e-4, "max": 2e-3}
    if kind == "layer":  # five 16-bit intermediates [5.4e-3, 2.5e-2]
        return {"rel": 2e-2, "max": 0.1}
    # 16-bit P and dS [bf16 2.6e-3, 5.3e-2; fp16 3e-4, 1.4e-3]; the score and the LSE are fp32 [2e-6]
    return {"rel": 1e-2, "max": 0.2} if dtype == "bf16" else {"rel": 1.2e-3, "max": 6e-3}


# ------------------------------------------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ------------------------------------------------------------------------------------------------------------------------
def _exact_head(c, q, k, v, grad=None):
    """One (batch, query head): O, LSE, the column sums of P and, with ``grad``, dQ, dK, dV."""
    s = (q @ k.T) / math.sqrt(c["D"])
    if c["causal"]:
        Sq, Skv = s.shape
        s.masked_fill_(torch.ones(Sq, Skv, dtype=torch.bool, device=s.device).triu_(Skv - Sq + 1), float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - lse[:, None])
    out = p @ v
    r = dict(out=out, lse=lse, score=p.sum(0))
    if grad is not None:
        ds = p * (grad @ v.T - (grad * out).sum(-1, keepdim=True)) / math.sqrt(c["D"])
        r.update(dq=ds @ k, dk=ds.T @ q, dv=p.T @ grad)
    return r


def _exact_attention(c, state):
    b_h_s_d = (lambda t: t.transpose(1, 2)) if c.get("layout") == "bshd" else (lambda t: t)
    q, k, v = (b_h_s_d(state[n]) for n in "qkv")
    grad = b_h_s_d(state["grad"]) if "grad" in state else None
    scales = state.get("scales", (1.0, 1.0, 1.0))
    f64 = dict(dtype=torch.float64, device=q.device)
    B, Hq, Hkv, group = c["B"], c["Hq"], c["Hkv"], c["Hq"] // c["Hkv"]
    full = dict(out=torch.empty(q.shape, **f64), lse=torch.empty(q.shape[:3], **f64), score=torch.empty(B, Hq, c["Skv"], **f64))
    if grad is not None:
        full.update(dq=torch.empty(q.shape, **f64), dk=torch.zeros(k.shape, **f64), dv=torch.zeros(v.shape, **f64))
    for b in range(B):
        for h in range(Hkv):
            kh, vh = k[b, h].double() * scales[1], v[b, h].double() * scales[2]
            for g in range(h * group, (h + 1) * group):
                r = _exact_head(c, q[b, g].double() * scales[0], kh, vh, None if grad is None else grad[b, g].double())
                for name, t in r.items():
                    if name in ("dk", "dv"):
                        full[name][b, h] += t
                    else:
                        full[name][b, g] = t
    out = {n: b_h_s_d(t) if t.dim() == 4 else t for n, t in full.items()}
    if c["kind"] == "train":
        return {n: out[n] for n in ("out", "lse", "dq", "dk", "dv")}
    if c["kind"] == "h2o":
        return out["out"], out["score"]
    return (out["out"], out["lse"]) if c["lse"] else out["out"]


def exact(case, seed):
    c, state = case, prepare(case, seed)
    if c["kind"] in ("attention", "train", "h2o"):
        return _exact_attention(c, state)
    if c["kind"] == "linear":
        y = state["x"].double() @ state["w"].double().T
        if c["row_scale"]:
            y = y * state["row_scale_t"].double()[:, None]
        if c["bias"]:
            y = y + state["bias_t"].double()
        if c["epilogue"] == "swiglu":
            gate, up = y.chunk(2, -1)
            y = torch.nn.functional.silu(gate) * up
        elif c["epilogue"] == "silu":
            y = torch.nn.functional.silu(y)
        elif c["epilogue"] == "gelu_tanh":
            y = torch.nn.functional.gelu(y, approximate="tanh")
        return y + state["residual_t"].double() if c["residual"] else y
    if c["kind"] == "bmm":
        return torch.stack([a.double() @ b.double() for a, b in zip(state["a"], state["b"])])
    if c["kind"] == "rowwise":
        x = [t.double() for t in state["inputs"]]
        if c["program"] == "softmax":
            return torch.softmax(0.125 * x[0], -1)
        if c["program"] == "silu_mul":
            return torch.nn.functional.silu(x[0]) * x[1]
        x = x[0] - x[0].mean(-1, keepdim=True)
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    layer = state["layer"]._orig_mod.double()
    return torch.cat([layer(x[None].double()) for x in state["x"]])
