"""RMSNorm followed by a projection as one row reduction and one GEMM.

``rmsnorm(x) @ W.T`` with ``rmsnorm(x) = x * rsqrt(mean(x^2) + eps) * g`` equals
``r[:, None] * (x @ (W * g).T)`` with ``r = rsqrt(mean(x^2) + eps)``: the norm's weight vector ``g``
moves into the projection weight once (``fold_norm_weight``), and the per-row factor ``r`` is applied
to the fp32 accumulator in the GEMM's epilogue (``gemm_act_rowmul_op``), so the normalised activations
are never written to or read back from memory.  The reference lists epilogue fusion as an aim
(README.md:6-7) and has no kernel of this form.
"""

from __future__ import annotations

from functools import cache

import torch

from . import _lib, native_dispatch
from .gemm_jit import _SHORT_DTYPES, _TORCH_DTYPES, gemm_act_rowmul_op
from .torch_custom_call import DEFAULT_NAMESPACE, _library

_DTYPE_NAMES = {torch_dtype: name for name, torch_dtype in _TORCH_DTYPES.items() if name in _SHORT_DTYPES}


def fold_norm_weight(weight: torch.Tensor, norm_weight: torch.Tensor) -> torch.Tensor:
    """``W * g`` along the input features, computed in fp32 and rounded once: ``weight`` is
    ``[out_features, in_features]``, ``norm_weight`` is ``[in_features]``."""
    return (weight.float() * norm_weight.float()).to(weight.dtype)


@cache
def _row_factors_op(dtype: str) -> torch._ops.OpOverload:
    """Torch op ``(x, eps, factors) -> ()`` writing ``factors[r, 0] = rsqrt(mean(x[r] ** 2) + eps)``."""
    name = f"rms_row_factors_{_SHORT_DTYPES[dtype]}"

    def cuda_impl(x: torch.Tensor, eps: float, factors: torch.Tensor) -> None:
        if x.dim() != 2:
            raise ValueError(f"{name}: expected a rank-2 tensor, got shape {tuple(x.shape)}")
        if x.dtype != _TORCH_DTYPES[dtype] or factors.dtype != x.dtype:
            raise ValueError(f"{name}: expected dtype {_TORCH_DTYPES[dtype]}, got {x.dtype} and {factors.dtype}")
        if not (x.is_contiguous() and factors.is_contiguous()):
            raise ValueError(f"{name}: all tensors must be contiguous")
        if factors.device != x.device or factors.numel() != x.shape[0]:
            raise ValueError(f"{name}: factors must hold one element per row of x on its device")
        with torch.cuda.device(x.device):
            _lib.init(x.device.index)
            _lib.rms_factors(dtype, x.data_ptr(), factors.data_ptr(), x.shape[0], x.shape[1], eps,
                             torch.cuda.current_stream().cuda_stream)

    lib = _library(DEFAULT_NAMESPACE)
    lib.define(f"{name}(Tensor arg0, float eps, Tensor(a1!) arg1) -> ()")
    if native_dispatch.load() is not None:
        native_dispatch.register_rms_factors(DEFAULT_NAMESPACE, name, dtype, _TORCH_DTYPES[dtype], cuda_impl)
    else:
        lib.impl(name, cuda_impl, "CUDA")
    lib.impl(name, lambda x, eps, factors: None, "Meta")
    return getattr(getattr(torch.ops, DEFAULT_NAMESPACE), name).default


@cache
def _rms_linear_op(dtype: str, activation: str) -> torch._ops.OpOverload:
    """Torch op ``(x, eps, weight, out) -> ()``: the row factors of ``x``, then ``out = activation(x @ weight^T)`` times
    them.  Shapes that have not been specialised go through the two ops one after the other."""
    row_factors = _row_factors_op(dtype)
    projection = gemm_act_rowmul_op("mm", activation, dtype)
    projection_name = projection._schema.name.split("::")[1]
    name = projection_name.replace("jit_mm", "rms_linear").replace("_rowmul", "")

    def cuda_impl(x: torch.Tensor, eps: float, weight: torch.Tensor, out: torch.Tensor) -> None:
        factors = torch.empty(x.shape[0], 1, dtype=x.dtype, device=x.device)
        row_factors(x, eps, factors)
        projection(x, weight, factors, out)

    lib = _library(DEFAULT_NAMESPACE)
    lib.define(f"{name}(Tensor arg0, float eps, Tensor arg1, Tensor(a2!) arg2) -> ()")
    if native_dispatch.load() is not None:
        native_dispatch.register_rms_linear(DEFAULT_NAMESPACE, name, projection_name, cuda_impl)
    else:
        lib.impl(name, cuda_impl, "CUDA")
    lib.impl(name, lambda x, eps, weight, out: None, "Meta")
    return getattr(getattr(torch.ops, DEFAULT_NAMESPACE), name).default


def rms_norm_linear(x: torch.Tensor, folded_weight: torch.Tensor, eps: float = 1e-5, activation: str = "none",
                    out: torch.Tensor | None = None) -> torch.Tensor:
    """``activation(rmsnorm(x) @ W.T)`` for ``x`` of shape ``[tokens, in_features]`` and
    ``folded_weight = fold_norm_weight(W, g)``.  The row factors are computed in fp32 and handed to
    the kernel in the operands' type; ``activation`` other than ``"none"`` is only equivalent to
    activating the scaled product when it is positively homogeneous (``"relu"``)."""
    if x.dtype not in _DTYPE_NAMES:
        raise ValueError(f"unsupported dtype {x.dtype}")
    if activation not in ("none", "relu"):
        raise ValueError("only 'none' and 'relu' commute with the per-row scale")
    tokens = x.shape[0]
    if out is None:
        out = torch.empty(tokens, folded_weight.shape[0], dtype=x.dtype, device=x.device)
    dtype = _DTYPE_NAMES[x.dtype]
    _rms_linear_op(dtype, activation)(x, eps, folded_weight, out)
    return out
