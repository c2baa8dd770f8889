"""The compiled CUDA kernels of the ops: the plain repeated call, and that all else still reaches Python."""

import threading

import pytest
import torch

from ayla_b200 import _lib, gemm_act_mul_op, gemm_jit, gemm_op, gemm_op_compiler, swiglu_op
from ayla_b200.gemm_jit import _DEFAULTS, GemmLauncher, GemmScheduleSeed
from ayla_b200.jit_compiler import ShapeSpecializingJITCompiler
from ayla_b200.rmsnorm_linear import rms_norm_linear
from oracle import gemm_oracle as O
from tests.test_gpu_parity import assert_parity

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _mm(m, n, k, seed=0):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    return a, bt, O.mm_ref32(a, bt)


@pytest.mark.parametrize("op", ["mm", "addmm", "bmm", "gated", "swiglu"])
def test_repeated_calls_on_new_operands(op, monkeypatch):
    """Every operand layout: the first call specialises in Python, later ones, on other buffers, do not enter it."""
    monkeypatch.delenv("AYLA_B200_DEBUG", raising=False)
    g = torch.Generator().manual_seed(3)
    for seed in range(3):
        a = torch.randn(40, 136, generator=g).bfloat16()
        bt, up = ((torch.randn(72, 136, generator=g) * 136 ** -0.5).bfloat16() for _ in range(2))
        bias, mul = torch.randn(72, generator=g).bfloat16(), torch.randn(40, 72, generator=g).bfloat16()
        if op == "bmm":
            a, bt = torch.stack([a, a * 2]), torch.stack([bt, up])
        call, args, want = {
            "mm": lambda: (gemm_op("mm", "bfloat16"), (a, bt), O.mm_ref32(a, bt)),
            "addmm": lambda: (gemm_op("addmm", "bfloat16"), (bias, a, bt), O.addmm_ref32(bias, a, bt)),
            "bmm": lambda: (gemm_op("bmm", "bfloat16"), (a, bt), O.bmm_ref32(a, bt)),
            "gated": lambda: (gemm_act_mul_op("mm", "sigmoid", "bfloat16"), (a, bt, mul),
                              O.act_ref32("sigmoid", O.gemm_ref32("mm", a, bt)) * mul.float()),
            "swiglu": lambda: (swiglu_op("bfloat16"), (a, bt, up), O.swiglu_ref32(a, bt, up)),
        }[op]()
        out = torch.full(want.shape, float("nan"), dtype=torch.bfloat16, device=DEV)
        assert call(*[t.to(DEV) for t in args], out) is None
        assert_parity(out.cpu(), want, f"{op} call {seed}")
        monkeypatch.setattr(ShapeSpecializingJITCompiler, "_launcher", _no_python)


def _no_python(*args, **kwargs):
    raise AssertionError("a repeated call entered Python")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_repeated_row_factors_do_not_enter_python(dtype, monkeypatch):
    weight = torch.randn(64, 264, device=DEV).to(dtype)
    for seed in range(3):
        x = torch.randn(24, 264, generator=torch.Generator().manual_seed(seed)).to(dtype)
        out = rms_norm_linear(x.to(DEV), weight)
        factors = torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5).to(dtype).float()
        assert_parity(out.cpu(), (x.float() @ weight.cpu().float().T) * factors, f"call {seed}")
        monkeypatch.setattr(_lib, "rms_factors", _no_python)
        monkeypatch.setattr(ShapeSpecializingJITCompiler, "_launcher", _no_python)


def test_another_streams_k_split_launch_enters_python(monkeypatch):
    """Only the stream that a workspace belongs to is served without Python."""
    monkeypatch.delenv("AYLA_B200_DEBUG", raising=False)
    m, n, k = 128, 192, 8192
    a, bt, want = _mm(m, n, k, 6)
    a, bt = a.to(DEV), bt.to(DEV)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    captured = {**_DEFAULTS, "tile_n": 64, "cta_group": 1, "split_k": 4}
    seed = GemmScheduleSeed(captured, {key: int(captured[key]) for key in _lib.Config.FIELDS}, (), None)
    monkeypatch.setattr(gemm_jit, "select_gemm_schedule", lambda *args: seed)
    op = gemm_op("mm", "bfloat16", "ayla_b200_k_split_test")
    op(a, bt, out)
    calls = []
    launch = GemmLauncher.__call__
    monkeypatch.setattr(GemmLauncher, "__call__", lambda self, *tensors: (calls.append(1), launch(self, *tensors))[1])
    op(a, bt, out)
    assert calls == []
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        op(a, bt, out)
    torch.cuda.synchronize()
    assert calls == [1]
    assert_parity(out.cpu(), want, "another stream")


def test_refusals_come_from_python_after_a_specialised_call():
    a, bt, want = _mm(48, 64, 128)
    a, bt = a.to(DEV), bt.to(DEV)
    out = torch.empty(48, 64, dtype=torch.bfloat16, device=DEV)
    op = gemm_op("mm", "bfloat16")
    for _ in range(2):
        op(a, bt, out)
    wide = torch.empty(48, 128, dtype=torch.bfloat16, device=DEV)[:, :64]
    for bad, message in (((a, bt, wide), "contiguous"), ((a.half(), bt, out), "expected dtype"),
                         ((a, bt[:, :64].contiguous(), out), "bt must be"), ((a[None], bt, out), "rank-2"),
                         ((a.view(-1)[4:4 + 47 * 128].view(47, 128), bt, out[:47]), "16-byte aligned")):
        with pytest.raises(ValueError, match=message):
            op(*bad)
    out.zero_()
    op(a, bt, out)
    assert_parity(out.cpu(), want, "the call after the refused ones")


def test_streams_threads_and_timeouts_of_a_k_split_shape():
    """A launch with a workspace: another stream gets its own from Python, threads share the record, and a
    launch that timed out is reported by the next call."""
    m, n, k = 128, 256, 8192
    a, bt, want = _mm(m, n, k, 5)
    a, bt = a.to(DEV), bt.to(DEV)
    op = gemm_op("mm", "bfloat16")
    outs = [torch.empty(m, n, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
    op(a, bt, outs[0])
    launcher = gemm_op_compiler("mm", "bfloat16")._launcher((a, bt, outs[0]))
    assert isinstance(launcher, GemmLauncher)
    torch.cuda.synchronize()

    def work(out):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                op(a, bt, out)
        torch.cuda.synchronize()

    threads = [threading.Thread(target=work, args=(out,)) for out in outs[1:]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out in outs:
        assert_parity(out.cpu(), want, "streams and threads")
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        op(a, bt, outs[0])
        torch.cuda.synchronize()
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    with pytest.raises(RuntimeError, match="timed out"):
        op(a, bt, outs[0])
    op(a, bt, outs[0])
    launcher.check_status()
    assert_parity(outs[0].cpu(), want, "after the report")


def test_capture_of_a_specialised_call_and_of_an_unseen_shape():
    a, bt, want = _mm(56, 80, 256, 9)
    a, bt = a.to(DEV), bt.to(DEV)
    out = torch.empty(56, 80, dtype=torch.bfloat16, device=DEV)
    op = gemm_op("mm", "bfloat16")
    op(a, bt, out)
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op(a, bt, out)
        with pytest.raises(RuntimeError, match="before capture"):
            op(a[:55], bt, out[:55])
    graph.replay()
    torch.cuda.synchronize()
    assert_parity(out.cpu(), want, "replayed")
