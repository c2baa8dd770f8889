"""Custom-op glue on the meta device -- mirrors the reference's
tests/test_torch_custom_call.py:8-53."""

from pathlib import Path

import pytest
import torch

from ayla_b200 import native_dispatch
from ayla_b200.jit_compiler import OpTemplate, ShapeSpecializingJITCompiler
from ayla_b200.torch_custom_call import OperandKind, TensorSpec, make_schema, make_torch_custom_call


def test_out_only_custom_call_has_meta_kernel():
    class Launcher:
        name = "out_only_meta_test"
        signature = [TensorSpec.build([4, 8], torch.bfloat16), TensorSpec.build([4, 16], torch.bfloat16)]

        def __call__(self, *args):
            raise AssertionError("Meta dispatch must not launch the kernel")

    op = make_torch_custom_call(Launcher(), [OperandKind.R, OperandKind.RW], namespace="ayla_b200_out_only_meta_test")
    src = torch.empty((4, 8), dtype=torch.bfloat16, device="meta")
    out = torch.empty((4, 16), dtype=torch.bfloat16, device="meta")
    assert op(src, out) is None


def test_result_shape_can_be_inferred_from_inputs():
    class Launcher:
        name = "dynamic_result_meta_test"
        signature = [TensorSpec.build([1, 8], torch.bfloat16), TensorSpec.build([1, 16], torch.bfloat16)]

        def __call__(self, *args):
            raise AssertionError("Meta dispatch must not launch the kernel")

    op = make_torch_custom_call(
        Launcher(),
        [OperandKind.R, OperandKind.RESULT],
        namespace="ayla_b200_dynamic_result_meta_test",
        infer_result_shapes=lambda src: [(src.shape[0], 16)],
    )
    src = torch.empty((7, 8), dtype=torch.bfloat16, device="meta")
    result = op(src)
    assert result.shape == (7, 16) and result.dtype == torch.bfloat16 and result.device.type == "meta"


def test_schema_rendering():
    kinds = [OperandKind.R, OperandKind.R, OperandKind.RW]
    assert make_schema("jit_mm_bf16", kinds) == "jit_mm_bf16(Tensor arg0, Tensor arg1, Tensor(a2!) arg2) -> ()"
    assert make_schema("f", [OperandKind.R, OperandKind.RESULT]) == "f(Tensor arg0) -> Tensor"
    assert make_schema("g", [OperandKind.RESULT, OperandKind.RESULT]) == "g() -> (Tensor, Tensor)"


def test_dynamic_m_op_infers_its_result_on_meta():
    from ayla_b200.dynamic_m import make_dynamic_m_matmul

    op = make_dynamic_m_matmul(256, 64, namespace="ayla_b200_dynamic_m_meta_test")
    lhs = torch.empty((3, 64), dtype=torch.bfloat16, device="meta")
    rhs = torch.empty((256, 64), dtype=torch.bfloat16, device="meta")
    out = op(lhs, rhs)
    assert out.shape == (3, 256) and out.dtype == torch.bfloat16 and out.device.type == "meta"


class _Counting(ShapeSpecializingJITCompiler):
    def __call__(self, *tensors):
        raise AssertionError("Meta dispatch must not launch the kernel")


_BF16, _F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("name, cls, dtypes, written", [
    ("mixed_dtypes", ShapeSpecializingJITCompiler, (_BF16, _F32), 1),
    ("six_operands", ShapeSpecializingJITCompiler, (_BF16,) * 6, 5),
    ("first_written", ShapeSpecializingJITCompiler, (_BF16,) * 3, 0),
    ("subclass", _Counting, (_BF16,) * 3, 2),
    ("plain", ShapeSpecializingJITCompiler, (_BF16,) * 5, 4),
])
def test_per_shape_dispatchers_of_any_signature_become_ops(name, cls, dtypes, written, monkeypatch):
    """Only a signature that the compiled dispatcher handles goes to it; the others keep the Python one."""
    compiled = []
    register = native_dispatch.register
    monkeypatch.setattr(native_dispatch, "register", lambda *args: (compiled.append(args[1]), register(*args)))
    compiler = cls(OpTemplate(name, tuple(TensorSpec(dtype, (None, None)) for dtype in dtypes)), lambda bound, device: None)
    kinds = [OperandKind.RW if i == written else OperandKind.R for i in range(len(dtypes))]
    op = make_torch_custom_call(compiler, kinds, namespace="ayla_b200_signatures_test")
    assert op(*[torch.empty(4, 8, dtype=dtype, device="meta") for dtype in dtypes]) is None
    assert torch._C._dispatch_has_kernel_for_dispatch_key(f"ayla_b200_signatures_test::{name}", "CUDA")
    assert compiled == (["plain"] if name == "plain" else [])


_WITHOUT_THE_EXTENSION = """
import sys, warnings
from pathlib import Path
import torch
from ayla_b200 import native_dispatch
path = Path(sys.argv[1])
if sys.argv[2] == "broken":
    path.write_bytes(b"not a shared object")
native_dispatch._PATH = path
with warnings.catch_warnings(record=True) as caught:
    warnings.simplefilter("always")
    from ayla_b200 import gemm_op, swiglu_op
    from ayla_b200.rmsnorm_linear import rms_norm_linear
    def empty(*shape):
        return torch.empty(*shape, dtype=torch.bfloat16, device="meta")
    assert gemm_op("mm", "bfloat16")(empty(8, 64), empty(16, 64), empty(8, 16)) is None
    assert swiglu_op("bfloat16")(empty(8, 64), empty(16, 64), empty(16, 64), empty(8, 16)) is None
    assert rms_norm_linear(empty(8, 64), empty(16, 64)).shape == (8, 16)
assert sum("go through Python" in str(w.message) for w in caught) == 1, [str(w.message) for w in caught]
for name in ("jit_mm_bf16", "swiglu_bf16", "rms_row_factors_bf16"):
    assert torch._C._dispatch_has_kernel_for_dispatch_key("ayla::" + name, "CUDA")
"""


@pytest.mark.parametrize("state", ["missing", "broken"])
def test_ops_without_the_compiled_dispatcher(state, tmp_path):
    """A missing or unloadable extension is reported once; the ops keep their Python implementation."""
    import subprocess
    import sys

    subprocess.run([sys.executable, "-c", _WITHOUT_THE_EXTENSION, str(tmp_path / "_torch_dispatch.so"), state],
                   check=True, cwd=Path(__file__).resolve().parent.parent)


def test_the_compiled_dispatcher_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
    import types

    from ayla_b200 import build

    (tmp_path / "source.cpp").write_text("")
    for name, path in (("DISPATCH_SOURCE", "source.cpp"), ("DISPATCH_PATH", "out.so"), ("DISPATCH_STAMP", "stamp")):
        monkeypatch.setattr(build, name, tmp_path / path)
    built = []

    def compile_it(cmd, **kwargs):
        built.append(cmd)
        (tmp_path / "out.so").write_text("")
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(build.subprocess, "run", compile_it)
    build.build_dispatch()
    build.build_dispatch()
    assert len(built) == 1
    monkeypatch.setattr(torch, "__version__", "0.0")
    build.build_dispatch()
    assert len(built) == 2
