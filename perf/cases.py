"""The work this backend is timed on: one pass per case through the public ops.

Sizes are those of this repository's shape corpora (``ayla_b200/corpus_shapes.json``), its suite
(``ayla_b200/suite.py``) and its whole-graph driver (``ayla_b200/bench_torch_compile.py``).  A case
names an op, its extents (``out[batch, m, n]`` from a depth of ``k``), the element type and, where
the op has them, an activation.
"""

from __future__ import annotations

import math

import torch

from ayla_b200 import gemm_act_mul_op, gemm_act_op, gemm_op, swiglu_op
from ayla_b200.rmsnorm_linear import fold_norm_weight, rms_norm_linear

_TORCH_DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}


def _case(op: str, dtype: str, batch: int, m: int, n: int, k: int, activation: str = "none", **extra) -> dict:
    return {**extra, "op": op, "dtype": dtype, "batch": batch, "m": m, "n": n, "k": k, "activation": activation}


def listed() -> list[dict]:
    return [
        # A linear layer of a small encoder on one short sequence: latency and launches are all there is.
        _case("addmm", "float16", 1, 256, 1024, 1024, name="addmm_small"),
        # One decoding step of eight sequences through an MLP weight: a stream of the weight.
        _case("mm", "bfloat16", 1, 8, 14336, 4096, name="mm_decode"),
        # A short prompt (or a large decoding batch) through an attention projection; the projection
        # most often seen in the corpora.
        _case("mm", "bfloat16", 1, 128, 4096, 4096, name="mm_prompt"),
        # The up projection of a transformer MLP, bias and GELU fused.
        _case("act", "float16", 1, 8192, 3072, 768, "gelu", name="mlp_up_gelu"),
        # The square product the benchmark is quoted on.
        _case("mm", "bfloat16", 1, 4096, 4096, 4096, name="mm_square"),
        # Backward: the weight gradient of a projection, a deep reduction over the tokens.
        _case("mm", "bfloat16", 1, 1024, 1024, 8192, name="mm_weight_grad"),
        # A projection of a vocabulary-sized dimension that is a multiple of 8 and of nothing more.
        _case("mm", "bfloat16", 1, 4096, 2560, 8008, name="mm_ragged_depth"),
        # Attention scores of 64 heads.
        _case("bmm", "bfloat16", 64, 2048, 2048, 128, name="bmm_scores"),
        # Window attention: thousands of small products.
        _case("bmm", "float16", 8192, 56, 32, 56, name="bmm_windows"),
        # A pointwise convolution as a product: very many rows, few columns, shallow.
        _case("mm", "float16", 1, 200704, 96, 24, name="mm_pointwise"),
        # RMSNorm and the fused query/key/value projection of a prompt.
        _case("rmsnorm", "bfloat16", 1, 4096, 6144, 4096, name="rmsnorm_projection"),
        # The gated MLP of an 8B-class decoder on a long prompt, the largest.
        _case("swiglu", "bfloat16", 1, 8192, 14336, 4096, name="swiglu_prompt"),
    ]


def _log_int(rng, low: int, high: int, multiple: int = 1) -> int:
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(multiple, round(value / multiple) * multiple)


def draw(rng) -> dict:
    """A case of the same ranges.  Three in four have columns and depth in multiples of 64, the rest
    in multiples of 8 (what the ops take); rows are any number."""
    while True:
        multiple = rng.choice((64, 64, 64, 8))
        dtype = rng.choice(("float16", "bfloat16"))
        kind = rng.choice(("decode", "decode", "projection", "projection", "fused", "weight_grad", "scores", "values",
                           "windows", "thin", "rmsnorm", "swiglu"))
        batch, activation = 1, "none"
        if kind == "decode":
            op = rng.choice(("mm", "mm", "addmm", "gated", "swiglu"))
            m, n, k = _log_int(rng, 1, 64), _log_int(rng, 1024, 14336, multiple), _log_int(rng, 1024, 14336, multiple)
            activation = "sigmoid" if op == "gated" else "none"
        elif kind == "projection":
            op = rng.choice(("mm", "addmm"))
            m, n, k = (_log_int(rng, 64, 16384), _log_int(rng, 256, 8192, multiple), _log_int(rng, 256, 8192, multiple))
        elif kind == "fused":
            op = rng.choice(("act", "gated"))
            activation = rng.choice(("relu", "silu", "gelu")) if op == "act" else rng.choice(("sigmoid", "silu"))
            m, n, k = (_log_int(rng, 64, 16384), _log_int(rng, 256, 8192, multiple), _log_int(rng, 256, 4096, multiple))
        elif kind == "weight_grad":
            op = "mm"
            m, n = _log_int(rng, 128, 4096, 8), _log_int(rng, 128, 4096, multiple)
            k = _log_int(rng, 2048, 65536, multiple)
        elif kind in ("scores", "values"):
            op, batch = "bmm", _log_int(rng, 8, 128)
            long, short = _log_int(rng, 128, 2048, 8), rng.choice((64, 80, 96, 128))
            m = _log_int(rng, 128, 2048)
            n, k = (long, short) if kind == "scores" else (short, long)
        elif kind == "windows":
            op, batch = "bmm", _log_int(rng, 256, 8192)
            m, n, k = _log_int(rng, 8, 128), _log_int(rng, 8, 128, 8), _log_int(rng, 8, 128, 8)
        elif kind == "thin":
            op = rng.choice(("mm", "addmm"))
            m, n, k = _log_int(rng, 16384, 262144), _log_int(rng, 16, 128, 8), _log_int(rng, 16, 128, 8)
        elif kind == "rmsnorm":
            op = "rmsnorm"
            m, n, k = _log_int(rng, 16, 8192), _log_int(rng, 1024, 8192, multiple), _log_int(rng, 1024, 8192, multiple)
        else:
            op = "swiglu"
            m, n, k = _log_int(rng, 64, 8192), _log_int(rng, 1024, 14336, multiple), _log_int(rng, 1024, 4096, multiple)
        case = _case(op, dtype, batch, m, n, k, activation)
        cost = work(case)
        if cost["flops"] <= 1.0e12 and cost["bytes"] <= 1.0e9:
            return case


def prepare(case: dict, seed: int) -> dict:
    """Activations ~ N(0, 1), weights ~ N(0, 1/k), biases ~ N(0, 0.1), and the output buffer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _TORCH_DTYPES[case["dtype"]]
    op, m, n, k = case["op"], case["m"], case["n"], case["k"]
    lead = (case["batch"],) if op == "bmm" else ()

    def normal(*shape: int, scale: float = 1.0) -> torch.Tensor:
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)

    a, bt = normal(*lead, m, k), normal(*lead, n, k, scale=k ** -0.5)
    out = torch.empty(*lead, m, n, dtype=dtype, device="cuda")
    if op in ("mm", "bmm"):
        return {"call": gemm_op(op, case["dtype"]), "args": (a, bt, out)}
    if op == "addmm":
        return {"call": gemm_op(op, case["dtype"]), "args": (normal(n, scale=0.1), a, bt, out)}
    if op == "act":
        return {"call": gemm_act_op("addmm", case["activation"], case["dtype"]),
                "args": (normal(n, scale=0.1), a, bt, out)}
    if op == "gated":
        return {"call": gemm_act_mul_op("mm", case["activation"], case["dtype"]), "args": (a, bt, normal(m, n), out)}
    if op == "swiglu":
        return {"call": swiglu_op(case["dtype"]), "args": (a, bt, normal(n, k, scale=k ** -0.5), out)}
    norm_weight = (1.0 + 0.1 * torch.randn(k, device="cuda", generator=g)).to(dtype)
    return {"x": a, "folded": fold_norm_weight(bt, norm_weight), "args": (out,)}


def run(state: dict) -> torch.Tensor:
    out = state["args"][-1]
    if "x" in state:
        rms_norm_linear(state["x"], state["folded"], out=out)
    else:
        state["call"](*state["args"])
    return out


def work(case: dict) -> dict:
    batch, m, n, k = case["batch"], case["m"], case["n"], case["k"]
    weights = 2 if case["op"] == "swiglu" else 1
    elements = batch * (m * k + weights * n * k + m * n)
    if case["op"] in ("addmm", "act"):
        elements += n
    elif case["op"] == "gated":
        elements += m * n
    return {"bytes": 2 * elements, "flops": 2 * weights * batch * m * n * k}


def tolerance(case: dict) -> dict:
    return {"rel": 7e-3 if case["dtype"] == "bfloat16" else 9e-4}
