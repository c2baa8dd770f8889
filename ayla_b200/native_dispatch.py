"""The compiled CUDA kernels of the torch ops (``csrc/torch_dispatch.cpp``).

An op registered here runs without entering Python whenever its shapes have been specialised; everything else
-- an unseen shape, refused operands, a reported timeout, another stream's workspace -- goes to the Python
fallback it was registered with.
"""

from __future__ import annotations

import ctypes
import importlib.util
import warnings
from collections.abc import Callable
from functools import cache
from pathlib import Path
from types import ModuleType

import torch

from . import _lib
from .jit_compiler import ShapeSpecializingJITCompiler
from .torch_custom_call import OperandKind

_PATH = Path(__file__).resolve().parent / "lib" / "_torch_dispatch.so"


@cache
def load() -> ModuleType | None:
    """The compiled dispatcher.  ``None``, with a warning, where it is missing or does not load (it is built for one
    torch and one Python): the ops keep their Python implementation then, which launches the same kernels at some
    8 us of host time more per call."""
    try:
        spec = importlib.util.spec_from_file_location("_torch_dispatch", _PATH)
        assert spec is not None and spec.loader is not None
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        return module
    except (ImportError, OSError) as error:
        warnings.warn(f"the compiled op dispatcher cannot be used, calls go through Python: {error}; "
                      "build it with `python -m ayla_b200.build`", RuntimeWarning, stacklevel=2)
        return None


_MAX_OPERANDS = 5  # kMaxOperands of the compiled dispatcher
_DISPATCHERS: dict[tuple[str, str], object] = {}  # those of the ops registered here


def serves(launcher, kinds: list[OperandKind]) -> bool:
    """Whether the compiled dispatcher can stand in for ``launcher``: a per-shape dispatcher itself (a subclass
    may do something else on a call), whose operands are the op's arguments, all of one dtype, the last one
    written -- and it is there to do so."""
    if type(launcher) is not ShapeSpecializingJITCompiler:
        return False
    signature = launcher.signature
    return (len(signature) <= _MAX_OPERANDS and len({spec.dtype for spec in signature}) == 1 and
            kinds == [OperandKind.R] * (len(signature) - 1) + [OperandKind.RW] and load() is not None)


def register(namespace: str, name: str, compiler: ShapeSpecializingJITCompiler) -> None:
    """Register the CUDA kernel of ``namespace::name``, backed by a compiler that ``serves`` accepts."""
    [dtype] = {spec.dtype for spec in compiler.signature}
    dispatcher = None

    offered: set[int] = set()  # launchers the dispatcher has been given, which it keeps alive

    def fallback(*tensors: torch.Tensor) -> None:
        launcher = compiler._launcher(tensors)
        launcher(*tensors)
        if id(launcher) in offered:
            return
        native_call: Callable[[], dict | None] | None = getattr(launcher, "native_call", None)
        fields = native_call() if native_call is not None else None
        if fields is not None:
            offered.add(id(launcher))
            dispatcher.insert(list(tensors), launcher, fields)

    dispatcher = load().register_op(namespace, name, len(compiler.signature), dtype, fallback)
    _DISPATCHERS[namespace, name] = dispatcher


def register_rms_factors(namespace: str, name: str, dtype: str, torch_dtype: torch.dtype, fallback) -> None:
    """Register the CUDA kernel of the row-factors op ``(x, eps, factors) -> ()``."""
    entry = ctypes.cast(_lib.load().ayla_b200_rms_factors, ctypes.c_void_p).value
    load().register_rms_factors(namespace, name, entry, _lib.DTYPE_CODES[dtype], torch_dtype, fallback)


def register_rms_linear(namespace: str, name: str, projection: str, fallback) -> None:
    """Register the CUDA kernel of ``(x, eps, weight, out) -> ()``, whose projection is the op ``projection``."""
    entry = ctypes.cast(_lib.load().ayla_b200_rms_factors, ctypes.c_void_p).value
    load().register_rms_linear(namespace, name, entry, _DISPATCHERS[namespace, projection], fallback)
