"""Parity of the CUDA path with the CPU oracle, on a B200.

Every test reaches the kernels through the C ABI (directly via ``ayla_b200._lib`` or
through the ``torch.ops.ayla`` ops, whose CUDA implementation is a ctypes call into
the same ABI).  Tolerance (the project's, written once in ``oracle.gemm_oracle``):
Frobenius relative error <= 5e-3 and max elementwise error <= 2e-2 * rms(ref) against
the CPU fp32 result rounded to the output type; elements that miss the second bound
while being the neighbouring representable value of the reference are rounding flips
of the last bit and are counted, not failed (``Parity.ok``).
"""

import json
import re

import pytest
import torch

from ayla_b200 import _lib, gemm_act_op, gemm_op, gemm_op_compiler, swiglu_op, swiglu_op_compiler
from ayla_b200.gemm_jit import gemm_jit_compiler, select_gemm_schedule
from oracle import gemm_oracle as O
from tests.conftest import load_golden_cases

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
TD = {"float16": torch.float16, "bfloat16": torch.bfloat16}


@pytest.fixture(scope="module")
def device_state():
    _lib.init(0)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    workspace = torch.zeros(64 << 20, dtype=torch.uint8, device=DEV)
    return status, workspace


def run_abi(operation, dtype, tensors, cfg, device_state, canary_rows=4):
    """Launch through the C ABI with an explicit schedule; returns (out, status)."""
    status, workspace = device_state
    status.zero_()
    dev = [t.to(DEV) for t in tensors]
    if operation == "swiglu":
        x, wg, wu = dev
        m, k = x.shape
        n = wg.shape[0]
        store = torch.full((m + canary_rows, n), float("nan"), dtype=x.dtype, device=DEV)
        out = store[:m]
        _lib.swiglu(dtype, x.data_ptr(), wg.data_ptr(), wu.data_ptr(), out.data_ptr(), m, n, k,
                    _lib.Config.from_dict(cfg) if cfg else None, status.data_ptr(),
                    torch.cuda.current_stream().cuda_stream)
    else:
        bias = dev[0] if operation == "addmm" else None
        a, bt = dev[-2:]
        batch = a.shape[0] if operation == "bmm" else 1
        m, k = a.shape[-2:]
        n = bt.shape[-2]
        rows = batch * m
        store = torch.full((rows + canary_rows, n), float("nan"), dtype=a.dtype, device=DEV)
        out = store[:rows].view(*a.shape[:-2], m, n)
        _lib.gemm(operation, dtype, bias.data_ptr() if bias is not None else 0, a.data_ptr(),
                  bt.data_ptr(), out.data_ptr(), batch, m, n, k,
                  _lib.Config.from_dict(cfg) if cfg else None, workspace.data_ptr(), workspace.numel(),
                  status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    # rows past the end of `out` must still hold their poison
    assert bool(torch.isnan(store[store.shape[0] - canary_rows:]).all()), "kernel wrote past the output"
    return out, int(status.item())


def launched_kernels(call, tmp_path):
    """(name, bytes of shared memory) of every kernel that ``call`` launches, as the profiler records them."""
    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        call()
        torch.cuda.synchronize()
    profile.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    kernels = [(e["name"], e["args"].get("shared memory")) for e in events if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("no kernels from the profiler")
    return kernels


def assert_parity(out, ref32, what=""):
    parity = O.compare(out, ref32)
    assert parity.ok, f"{what}: {parity}"
    return parity


# ------------------------------------------------------------------ golden vectors

@pytest.mark.parametrize("case", load_golden_cases(), ids=repr)
def test_ops_reproduce_golden_vectors(case):
    operands = [t.to(DEV) for t in case.operands()]
    want = case.expected()
    out = torch.full(want.shape, float("nan"), dtype=case.torch_dtype, device=DEV)
    if case.operation == "swiglu":
        assert swiglu_op(case.dtype)(*operands, out) is None
    else:
        assert gemm_op(case.operation, case.dtype)(*operands, out) is None
    torch.cuda.synchronize()
    got = out.cpu()
    parity = O.compare(got, want.float())
    assert parity.ok, parity
    # Beyond the project tolerance: a different fp32 summation order can only flip the
    # last bit, and only on a small fraction of elements.
    differing = int((got.view(torch.int16) != want.view(torch.int16)).sum())
    assert differing <= max(2, got.numel() // 200), (differing, got.numel())
    rms = float(want.float().pow(2).mean().sqrt())
    ulp = O._ulp(want.float().abs().clamp_min(1e-2 * rms), case.torch_dtype)
    assert bool(((got.float() - want.float()).abs() <= ulp * 1.0001).all())


# ------------------------------------- the reference's own GPU test, op for op

@pytest.mark.parametrize("operation", ["mm", "addmm", "bmm"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(96, 128, 128), (256, 256, 256)])
def test_jit_matches_torch_and_replays_cuda_graph(operation, dtype, m, n, k):
    """tests/test_gemm_jit.py:49-75 of the reference, same shapes and tolerances."""
    compiler = gemm_jit_compiler(operation, str(dtype).removeprefix("torch."))
    lead = (2,) if operation == "bmm" else ()
    a = torch.randn((*lead, m, k), device=DEV, dtype=dtype)
    bt = torch.randn((*lead, n, k), device=DEV, dtype=dtype)
    out = torch.empty((*lead, m, n), device=DEV, dtype=dtype)
    args = [a, bt, out]
    expected = a @ bt.transpose(-1, -2)
    if operation == "addmm":
        bias = torch.randn(n, device=DEV, dtype=dtype)
        args.insert(0, bias)
        expected = torch.addmm(bias, a, bt.T)
    compiler(*args)
    torch.testing.assert_close(out, expected, atol=0.125, rtol=0.02)
    assert compiler.cache_size == 1
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        compiler(*args)
    out.zero_()
    graph.replay()
    torch.testing.assert_close(out, expected, atol=0.125, rtol=0.02)
    assert compiler.cache_size == 1


def test_capture_time_cache_miss_is_an_error():
    compiler = gemm_jit_compiler("mm", "bfloat16")
    a = torch.randn(64, 64, device=DEV, dtype=torch.bfloat16)
    out = torch.empty(64, 64, device=DEV, dtype=torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError, match="before capture"):
        with torch.cuda.graph(graph):
            compiler(a, a, out)


# --------------------------------------------------- every kernel variant, ragged

ROW_MAJOR = [(tile_n, cta_group) for tile_n in (64, 128, 192, 256) for cta_group in (1, 2)]
SHAPES = [
    ("mm", 1, 128, 256, 64), ("mm", 1, 96, 128, 128), ("mm", 1, 333, 520, 200), ("mm", 1, 1, 8, 8),
    ("addmm", 1, 300, 264, 192), ("bmm", 3, 200, 136, 128), ("mm", 1, 1024, 768, 520),
]


@pytest.mark.parametrize("tile_n,cta_group", ROW_MAJOR)
@pytest.mark.parametrize("split_k", [1, 3])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_row_major_variants(tile_n, cta_group, split_k, dtype, device_state):
    torch.manual_seed(tile_n + cta_group + split_k)
    cfg = dict(tile_n=tile_n, cta_group=cta_group, split_k=split_k, group_m=3)
    for operation, batch, m, n, k in SHAPES:
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k)).to(TD[dtype])
        bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
        out, status = run_abi(operation, dtype, tensors, cfg, device_state)
        assert status == 0
        assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("k", [1024, 1016, 1000])  # rows of whole lines, starting inside a line, inside a sector
def test_cache_hints_change_no_bit(cta_group, k, device_state):
    g = torch.Generator().manual_seed(k)
    a = torch.randn(520, k, generator=g).bfloat16()
    bt = (torch.randn(264, k, generator=g) * k ** -0.5).bfloat16()
    outs = []
    for hint_a in (0, 1, 2):
        for hint_b in (0, 1, 2):
            cfg = dict(tile_n=128, cta_group=cta_group, l2_hint_a=hint_a, l2_hint_b=hint_b)
            out, status = run_abi("mm", "bfloat16", (a, bt), cfg, device_state)
            assert status == 0
            outs.append(out)
    assert_parity(outs[0], O.mm_ref32(a, bt))
    assert all(torch.equal(outs[0], out) for out in outs)


# (batch, m, n, k): one tile and several, extents inside a chunk and a lane quarter, depths that the splits do not share
# evenly; the last three fill whole waves first and split the depth of the tiles left over.
@pytest.mark.parametrize("batch, m, n, k, config", [
    (1, 128, 64, 1000, dict(tile_n=64, cta_group=1, split_k=7)),
    (1, 130, 136, 2056, dict(tile_n=64, cta_group=1, split_k=8)),
    (3, 257, 200, 1024, dict(tile_n=128, cta_group=2, split_k=4)),
    (1, 40, 128, 8192, dict(tile_n=128, cta_group=1, split_k=48)),
    (1, 300, 264, 3000, dict(tile_n=192, cta_group=2, split_k=5)),
    (1, 600, 520, 4096, dict(tile_n=256, cta_group=2, split_k=2)),
    (1, 512, 256, 4096, dict(tile_n=256, cta_group=1, split_k=32)),
    (2, 1024, 1000, 512, dict(tile_n=256, cta_group=1, split_k=3, split_tail=1, grid_ctas=54)),
    (1, 2100, 1000, 640, dict(tile_n=128, cta_group=2, split_k=2, split_tail=1, grid_ctas=60)),
    (1, 520, 520, 1032, dict(tile_n=64, cta_group=1, split_k=5, split_tail=1, grid_ctas=40)),
])
@pytest.mark.parametrize("bias", [False, True])
def test_shared_sum_of_a_split_depth(batch, m, n, k, config, bias, device_state):
    """The k-splits of a tile share its sum; an owner that does not wait leaves its pieces to the last of the others.
    Both add in split order, so they agree bit for bit."""
    lib = _lib.load()
    operation = "bmm" if batch > 1 else "addmm" if bias else "mm"
    g = torch.Generator().manual_seed(m + n + k)
    lead = (batch,) if batch > 1 else ()
    a = torch.randn((*lead, m, k), generator=g).bfloat16()
    bt = (torch.randn((*lead, n, k), generator=g) * k ** -0.5).bfloat16()
    tensors = [a, bt] if operation != "addmm" else [torch.randn(n, generator=g).bfloat16(), a, bt]
    out, status = run_abi(operation, "bfloat16", tensors, config, device_state)
    assert status == 0
    assert_parity(out, O.gemm_ref32(operation, *tensors), config)
    lib.ayla_b200_debug_set_flags(32)  # owners hand every piece over, to whoever is last or back to themselves
    try:
        for _ in range(3):
            handed, status = run_abi(operation, "bfloat16", tensors, config, device_state)
            assert status == 0
            assert torch.equal(handed, out)
    finally:
        lib.ayla_b200_debug_set_flags(0)
    again, _ = run_abi(operation, "bfloat16", tensors, config, device_state)  # the counters were left clean
    assert torch.equal(again, out)
    assert not bool(device_state[1][:65536].any())


@pytest.mark.parametrize("tile_n,cta_group", ROW_MAJOR)
def test_split_depths_summed_by_the_last_arriver(tile_n, cta_group, device_state):
    """More split units than the grid runs at once (few CTAs asked for), so that a CTA has several: the last to arrive
    sums a tile.  With a bias, an activation, factors per row, a gate and batches."""
    status, workspace = device_state
    config = dict(tile_n=tile_n, cta_group=cta_group, split_k=3, grid_ctas=6)
    torch.manual_seed(tile_n + cta_group)
    for operation, activation, gate, batch, m, n, k in (
            ("mm", "none", None, 1, 333, 520, 520), ("addmm", "none", None, 1, 300, 776, 264), ("bmm", "none", None, 4, 200, 136, 712),
            ("addmm", "gelu", None, 1, 520, 520, 200), ("mm", "relu", "row", 1, 300, 1032, 320), ("addmm", "silu", "full", 1, 700, 264, 392)):
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k)).bfloat16()
        bt = (torch.randn((*lead, n, k)) * k ** -0.5).bfloat16()
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n).bfloat16(), a, bt)
        assert -(-m // (128 * cta_group)) * -(-n // tile_n) * batch * 3 > 6 // cta_group
        want = O.gemm_ref32(operation, *tensors)
        if activation == "none" and gate is None:
            out, code = run_abi(operation, "bfloat16", tensors, config, device_state)
            out = out.cpu()
        else:
            want = O.act_ref32(activation, want)
            dev = [t.to(DEV) for t in tensors]
            out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
            status.zero_()
            mul = (torch.rand(m, 1 if gate == "row" else n) + 0.5).bfloat16()
            head = (operation, "bfloat16", activation, dev[0].data_ptr() if operation == "addmm" else 0, dev[-2].data_ptr(),
                    dev[-1].data_ptr())
            tail = (out.data_ptr(), 1, m, n, k, _lib.Config.from_dict(config), workspace.data_ptr(), workspace.numel(),
                    status.data_ptr(), torch.cuda.current_stream().cuda_stream)
            if gate is None:
                _lib.gemm_act(*head, *tail)
            else:
                want = want * mul.float()
                held = mul.to(DEV)
                (_lib.gemm_act_rowmul if gate == "row" else _lib.gemm_act_mul)(*head, held.data_ptr(), *tail)
            torch.cuda.synchronize()
            out, code = out.cpu(), int(status.item())
        assert code == 0
        assert_parity(out, want, f"{operation} {activation} {gate} {batch}x{m}x{n}x{k} {config}")
    assert not bool(workspace[:65536].any())


@pytest.mark.parametrize("tile_n", [16, 32, 64, 128])
@pytest.mark.parametrize("split_k", [1, 4])
def test_swapped_variants(tile_n, split_k, device_state):
    torch.manual_seed(tile_n * 7 + split_k)
    cfg = dict(tile_n=tile_n, cta_group=1, swap_ab=1, split_k=split_k, group_m=1)
    for dtype in ("bfloat16", "float16"):
        for operation, batch, m, n, k in (("mm", 1, 1, 256, 512), ("mm", 1, tile_n, 520, 264),
                                          ("addmm", 1, max(1, tile_n - 3), 264, 192),
                                          ("bmm", 3, tile_n, 136, 128), ("mm", 1, 3 * tile_n + 5, 1024, 512)):
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            out, status = run_abi(operation, dtype, tensors, cfg, device_state)
            assert status == 0
            assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")


@pytest.mark.parametrize("tile_rows", [8, 56, 97, 104, 120])
def test_swapped_tiles_with_fewer_rows(tile_rows, device_state):
    """tile_rows < 128: more, lighter tiles of bt; rows past the trimmed tile are never stored."""
    torch.manual_seed(tile_rows)
    for tile_n, split in ((16, dict()), (32, dict(split_k=2)), (64, dict(split_k=2, cluster_split=1)), (128, dict())):
        cfg = dict(tile_n=tile_n, cta_group=1, swap_ab=1, group_m=1, tile_rows=tile_rows, **split)
        for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, min(tile_n, 24), 1000, 512),
                                                 ("addmm", "float16", 1, tile_n, 776, 320),
                                                 ("bmm", "bfloat16", 2, max(1, tile_n - 5), 264, 256)):
            assert _lib.config_valid(_lib.Config.from_dict(cfg), operation, dtype, batch, m, n, k), cfg
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            out, status = run_abi(operation, dtype, tensors, cfg, device_state)
            assert status == 0
            assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")


@pytest.mark.parametrize("split_k", [2, 4, 8])
def test_cluster_split_k_variants(split_k, device_state):
    """k-splits as the CTAs of one cluster, reduced through distributed shared memory."""
    torch.manual_seed(split_k)
    for tile_n, swap in ((64, 0), (128, 0), (256, 0), (32, 1), (64, 1), (128, 1)):
        cfg = dict(tile_n=tile_n, cta_group=1, swap_ab=swap, split_k=split_k, cluster_split=1, group_m=1 if swap else 8)
        for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, 333 if not swap else tile_n - 3, 520, 1000),
                                                 ("addmm", "float16", 1, 256 if not swap else tile_n, 264, 1024),
                                                 ("bmm", "bfloat16", 2, 200 if not swap else 8, 136, 512)):
            if not _lib.config_valid(_lib.Config.from_dict(cfg), operation, dtype, batch, m, n, k):
                continue
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            out, status = run_abi(operation, dtype, tensors, cfg, device_state)
            assert status == 0
            assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")
    # deterministic: the partials are added in rank order
    op, tensors = O.make_inputs("C2b", "bfloat16", scale_down=4)
    cfg = dict(tile_n=64, cta_group=1, split_k=split_k, cluster_split=1)
    first, _ = run_abi(op, "bfloat16", tensors, cfg, device_state)
    again, _ = run_abi(op, "bfloat16", tensors, cfg, device_state)
    assert torch.equal(first, again)


@pytest.mark.parametrize("tile_n,cta_group", [(128, 1), (256, 1), (128, 2), (256, 2)])
@pytest.mark.parametrize("grid_ctas", [0, 10, 36])
def test_stream_k_variants(tile_n, cta_group, grid_ctas, device_state):
    """Equal contiguous shares of the (tile, k-block) sequence per CTA: tiles cut between CTAs are
    finished by the last contributor, summing in CTA order."""
    torch.manual_seed(tile_n + cta_group + grid_ctas)
    cfg = dict(tile_n=tile_n, cta_group=cta_group, stream_k=1, group_m=3, grid_ctas=grid_ctas)
    for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, 1024, 768, 520), ("addmm", "float16", 1, 300, 264, 1992),
                                             ("bmm", "bfloat16", 3, 200, 136, 1024), ("mm", "float16", 1, 333, 520, 4104)):
        assert _lib.config_valid(_lib.Config.from_dict(cfg), operation, dtype, batch, m, n, k), cfg
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k)).to(TD[dtype])
        bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
        out, status = run_abi(operation, dtype, tensors, cfg, device_state)
        assert status == 0
        assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")
        again, _ = run_abi(operation, dtype, tensors, cfg, device_state)
        assert torch.equal(out, again)


@pytest.mark.parametrize("split_k", [2, 4])
@pytest.mark.parametrize("tile_n", [64, 128, 256])
def test_paired_cluster_split_k_variants(split_k, tile_n, device_state):
    """k-splits of a 256-row tile as the CTA pairs of one cluster (4 or 8 CTAs)."""
    torch.manual_seed(split_k * 1000 + tile_n)
    cfg = dict(tile_n=tile_n, cta_group=2, split_k=split_k, cluster_split=1, group_m=2)
    for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, 333, 520, 1000), ("mm", "float16", 1, 256, 256, 512),
                                             ("addmm", "float16", 1, 512, 264, 1024), ("addmm", "bfloat16", 1, 130, 72, 2048),
                                             ("bmm", "bfloat16", 2, 200, 136, 512), ("mm", "bfloat16", 1, 1024, 1024, 4096)):
        assert _lib.config_valid(_lib.Config.from_dict(cfg), operation, dtype, batch, m, n, k)
        assert _lib.workspace_bytes(_lib.Config.from_dict(cfg), operation, batch, m, n, k) == 0
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k)).to(TD[dtype])
        bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
        out, status = run_abi(operation, dtype, tensors, cfg, device_state)
        assert status == 0
        assert_parity(out, O.gemm_ref32(operation, *tensors), f"{operation} {batch}x{m}x{n}x{k} {cfg}")
        again, _ = run_abi(operation, dtype, tensors, cfg, device_state)
        assert torch.equal(out, again)


@pytest.mark.parametrize("split_k", [1, 2, 4])
@pytest.mark.parametrize("tile_n", [128, 256])
def test_pairs_on_tiles_of_128_rows(tile_n, split_k, device_state):
    """Products of at most 128 rows on CTA pairs, whole and split through clusters: the same bits as with single CTAs, and
    the epilogue's bias, activation, row factors and gate on the half of the columns that each lane has."""
    torch.manual_seed(tile_n + split_k)
    status, workspace = device_state
    cfg = dict(tile_n=tile_n, cta_group=2, split_k=split_k, cluster_split=int(split_k > 1), group_m=8)
    for operation, dtype, activation, batch, m, n, k in (
            ("mm", "bfloat16", "none", 1, 128, 256, 512), ("mm", "float16", "none", 1, 65, 520, 1000),
            ("addmm", "float16", "gelu", 1, 97, 776, 2056), ("addmm", "bfloat16", "none", 1, 127, 136, 640),
            ("bmm", "float16", "silu", 5, 70, 264, 648), ("bmm", "bfloat16", "none", 40, 128, 392, 512),
            ("mm", "bfloat16", "relu", 1, 33, 72, 4096), ("mm", "float16", "none", 1, 3, 4096, 584)):
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k)).to(TD[dtype])
        bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
        what = f"{operation} {activation} {batch}x{m}x{n}x{k} {cfg}"
        out, code = run_abi(operation, dtype, tensors, cfg, device_state)
        assert code == 0
        ref = O.gemm_ref32(operation, *tensors)
        assert_parity(out, ref, what)
        single, code = run_abi(operation, dtype, tensors, dict(cfg, cta_group=1), device_state)
        assert code == 0 and torch.equal(out, single), what
        dev = [t.to(DEV) for t in tensors]
        row = (torch.rand((*lead, m, 1)) + 0.5).to(TD[dtype])
        gate = torch.randn((*lead, m, n)).to(TD[dtype])
        for entry, factors in ((_lib.gemm_act_rowmul, row), (_lib.gemm_act_mul, gate)):
            store = torch.full((batch * m + 4, n), float("nan"), dtype=TD[dtype], device=DEV)
            status.zero_()
            entry(operation, dtype, activation, dev[0].data_ptr() if operation == "addmm" else 0, dev[-2].data_ptr(),
                  dev[-1].data_ptr(), (factors_on_device := factors.to(DEV)).data_ptr(), store.data_ptr(), batch, m, n, k,
                  _lib.Config.from_dict(cfg), workspace.data_ptr(), workspace.numel(), status.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert int(status.item()) == 0 and bool(torch.isnan(store[batch * m:]).all()), what
            got = store[:batch * m].view(*lead, m, n).cpu()
            assert_parity(got, O.act_ref32(activation, ref) * factors.float(), f"{what} {entry.__name__}")


@pytest.mark.parametrize("m, flat", [(33, True), (128, True), (129, False)])
@pytest.mark.parametrize("operation, activation, tile_n, split_k", [("mm", "none", 128, 2), ("addmm", "gelu", 128, 1),
                                                                    ("mm", "silu", 256, 1), ("addmm", "none", 256, 2)])
def test_pairs_of_few_rows_run_the_kernel_of_64_rows_a_cta(operation, activation, tile_n, split_k, m, flat, device_state,
                                                           tmp_path):
    status, _ = device_state
    a, bt = (torch.zeros(rows, 1024, dtype=torch.bfloat16, device=DEV) for rows in (m, 512))
    out, bias = torch.empty(m, 512, dtype=torch.bfloat16, device=DEV), torch.zeros(512, dtype=torch.bfloat16, device=DEV)
    cfg = _lib.Config.from_dict(dict(tile_n=tile_n, cta_group=2, split_k=split_k, cluster_split=int(split_k > 1), group_m=8))

    def call():
        _lib.gemm_act(operation, "bfloat16", activation, bias.data_ptr(), a.data_ptr(), bt.data_ptr(), out.data_ptr(), 1, m, 512,
                      1024, cfg, 0, 0, status.data_ptr(), torch.cuda.current_stream().cuda_stream)

    [(name, _)] = launched_kernels(call, tmp_path)
    traits = re.search(r"GemmTraits<([^>]*)>", name).group(1).split(", ")
    assert traits[:2] == [str(tile_n), "2"] and (traits[6] == "3") == flat, name


@pytest.mark.parametrize("tile_n, split_k", [(128, 2), (128, 4), (256, 2), (256, 4)])
def test_pairs_of_few_rows_exchange_partial_sums_in_the_ring(tile_n, split_k, device_state):
    """The exchange area over ring slots that are still in use, which no schedule of theirs needs: all partial sums wait."""
    lib = _lib.load()
    g = torch.Generator().manual_seed(tile_n + split_k)
    cfg = dict(tile_n=tile_n, cta_group=2, split_k=split_k, cluster_split=1)
    for m, n, k in ((128, 520, 2048), (70, 264, 1992), (33, 136, 4096)):
        a = torch.randn(m, k, generator=g).bfloat16()
        bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
        want, code = run_abi("mm", "bfloat16", (a, bt), cfg, device_state)
        assert code == 0
        try:
            lib.ayla_b200_debug_set_flags(2)
            out, code = run_abi("mm", "bfloat16", (a, bt), cfg, device_state)
        finally:
            lib.ayla_b200_debug_set_flags(0)
        assert code == 0 and torch.equal(out, want)
        assert_parity(out, O.mm_ref32(a, bt), f"{m}x{n}x{k} {cfg}")


def test_launch_overlap_keeps_stream_order(device_state):
    """A chain of launches, each reading what the one before wrote, gives the same bits whether
    or not a launch may start its set-up under its predecessor's tail."""
    torch.manual_seed(5)
    n = 1024
    x0 = torch.randn(256, n).to(torch.bfloat16).to(DEV)
    weights = [(torch.randn(n, n) * n ** -0.5).to(torch.bfloat16).to(DEV) for _ in range(3)]
    ws = torch.zeros(64 << 20, dtype=torch.uint8, device=DEV)
    schedules = [dict(tile_n=128, cta_group=2), dict(tile_n=64, cta_group=1, split_k=4),
                 dict(tile_n=64, cta_group=1, split_k=4, cluster_split=1), dict(tile_n=128, cta_group=1, split_tail=2)]
    stream = torch.cuda.current_stream().cuda_stream

    def chain():
        bufs = [x0, torch.zeros_like(x0), torch.zeros_like(x0)]
        cur = 0
        for step in range(24):
            src, dst = bufs[cur], bufs[1 + (step % 2)]
            cfg = _lib.Config.from_dict(schedules[step % len(schedules)])
            _lib.gemm("mm", "bfloat16", 0, src.data_ptr(), weights[step % 3].data_ptr(), dst.data_ptr(),
                      1, 256, n, n, cfg, ws.data_ptr(), ws.numel(), 0, stream)
            cur = 1 + (step % 2)
        torch.cuda.synchronize()
        return bufs[cur].clone()

    try:
        _lib.set_launch_overlap(False)
        plain = chain()
        _lib.set_launch_overlap(True)
        overlapped = chain()
        out_buf = torch.zeros_like(x0)
        mid = torch.zeros_like(x0)
        cfg = _lib.Config.from_dict(schedules[0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            cap = torch.cuda.current_stream().cuda_stream
            _lib.gemm("mm", "bfloat16", 0, x0.data_ptr(), weights[0].data_ptr(), mid.data_ptr(), 1, 256, n, n,
                      cfg, 0, 0, 0, cap)
            _lib.gemm("mm", "bfloat16", 0, mid.data_ptr(), weights[1].data_ptr(), out_buf.data_ptr(), 1, 256, n, n,
                      cfg, 0, 0, 0, cap)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        _lib.set_launch_overlap(True)
    assert torch.equal(plain, overlapped)
    assert torch.isfinite(plain.float()).all()
    expect_mid = O.gemm_ref32("mm", x0.cpu(), weights[0].cpu()).to(torch.bfloat16)
    expect = O.gemm_ref32("mm", expect_mid, weights[1].cpu())
    assert_parity(out_buf.cpu(), expect, "two dependent launches in a graph")


@pytest.mark.parametrize("activation", ["relu", "sigmoid", "silu", "gelu", "gelu_tanh"])
def test_fused_activation_epilogue(activation, device_state):
    """act([bias +] a @ bt.T) through every kind of epilogue: bulk-store, transposed, workspace
    split-K, cluster split-K (bulk-store, lone-chunk and narrow-slice forms)."""
    torch.manual_seed(len(activation))
    status, workspace = device_state
    schedules = [dict(tile_n=256, cta_group=2), dict(tile_n=128, cta_group=1, split_k=2),
                 dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1),
                 dict(tile_n=128, cta_group=1, split_k=4, cluster_split=1),
                 dict(tile_n=64, cta_group=2, split_k=2, cluster_split=1),
                 dict(tile_n=16, cta_group=1, swap_ab=1, group_m=1),
                 dict(tile_n=32, cta_group=1, swap_ab=1, group_m=1, split_k=4, cluster_split=1),
                 dict(tile_n=128, cta_group=1, swap_ab=1, group_m=1, split_k=2, cluster_split=1),
                 dict(tile_n=64, cta_group=1, swap_ab=1, group_m=1, split_k=3)]
    for cfg in schedules:
        small = bool(cfg.get("swap_ab"))
        for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, 24 if small else 300, 520, 1024),
                                                 ("addmm", "float16", 1, 16 if small else 256, 264, 512),
                                                 ("bmm", "bfloat16", 2, 8 if small else 200, 136, 512)):
            config = _lib.Config.from_dict(cfg)
            assert _lib.config_valid(config, operation, dtype, batch, m, n, k), cfg
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            dev = [t.to(DEV) for t in tensors]
            out = torch.full((*lead, m, n), float("nan"), dtype=TD[dtype], device=DEV)
            status.zero_()
            _lib.gemm_act(operation, dtype, activation, dev[0].data_ptr() if operation == "addmm" else 0,
                          dev[-2].data_ptr(), dev[-1].data_ptr(), out.data_ptr(), batch, m, n, k, config,
                          workspace.data_ptr(), workspace.numel(), status.data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            want = O.act_ref32(activation, O.gemm_ref32(operation, *tensors))
            assert_parity(out.cpu(), want, f"{activation} {operation} {batch}x{m}x{n}x{k} {cfg}")


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("activation", ["sigmoid", "silu", "gelu", "gelu_tanh"])
def test_activations_at_every_16_bit_value(activation, dtype):
    """act(x @ I) over every finite value of the type (bf16 from 2^-100 up: its square and cube must not
    leave fp32's range at the bottom), against the function in double precision.  The bound is half an ulp
    for the one rounding, plus the relative error of the fp32 evaluation: 2^z with |z| <= 130 carries z's
    own rounding (130 * 2^-24 * ln 2 < 6e-6, three times that for the cubic argument of gelu_tanh), GELU's
    polynomial 3e-6 down to x = -5 and less than 6e-9 absolutely below (5e-6 of 5 * Phi(-5) = 1.4e-6 down to
    x = -6, where x * Phi(x) itself is 5.9e-9);
    results under 2^-100 may be flushed."""
    values = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(TD[dtype])
    values = values[torch.isfinite(values)]
    if dtype == "bfloat16":
        values = torch.where(values.float().abs() < 2.0 ** -100, torch.zeros_like(values), values)
    x = torch.cat([values, values.new_zeros(-values.numel() % 64)]).view(-1, 64)
    out = torch.full_like(x, float("nan"), device=DEV)
    gemm_act_op("mm", activation, dtype)(x.to(DEV), torch.eye(64, dtype=TD[dtype], device=DEV), out)
    x64 = x.double()
    want = {"sigmoid": lambda t: torch.special.expit(t), "silu": lambda t: t * torch.special.expit(t),
            "gelu": lambda t: 0.5 * t * torch.special.erfc(-t * 0.5 ** 0.5),
            "gelu_tanh": lambda t: t * torch.special.expit(2 * (2 / torch.pi) ** 0.5 * (t + 0.044715 * t ** 3)),
            }[activation](x64)
    got = out.cpu().double()
    half_ulp = 0.5 * O._ulp(want.float(), TD[dtype]).double()
    relative = {"gelu": 3e-6, "gelu_tanh": 2e-5}.get(activation, 7e-6)
    bound = 1.001 * half_ulp + relative * want.abs() + (6e-9 if activation == "gelu" else 2.0 ** -100)
    bad = ~((got - want).abs() <= bound)
    assert not bad.any(), [(x64[bad][i].item(), got[bad][i].item(), want[bad][i].item()) for i in range(min(5, int(bad.sum())))]


@pytest.mark.parametrize("activation, at_minus_infinity", [("relu", 0.0), ("sigmoid", 0.0), ("silu", float("nan")),
                                                           ("gelu", float("nan")), ("gelu_tanh", float("nan"))])
@pytest.mark.parametrize("m", [16, 256])
def test_activations_of_infinities_and_nan(activation, at_minus_infinity, m):
    """The formulas of the framework's own activations at the ends: x * sigmoid(x) and 0.5 x (1 + erf or tanh) are
    0 * inf at minus infinity.  (relu is max(x, 0) on the fp32 sum, whose result for a NaN is 0.)"""
    def run(rows):
        a = torch.zeros(m, 8).half()
        for i, row in enumerate(rows):
            a[i] = torch.tensor(row).half()
        out = torch.empty(m, 128, dtype=torch.float16, device=DEV)
        gemm_act_op("mm", activation, "float16")(a.to(DEV), torch.ones(128, 8).half().to(DEV), out)
        return out.cpu()[:len(rows)]

    top, nan, inf = 1.0 if activation == "sigmoid" else float("inf"), float("nan"), float("inf")
    got = run([[inf] + [0.0] * 7, [-inf] + [0.0] * 7, [nan] + [0.0] * 7, [65504.0] * 8, [-65504.0] * 8])
    want = torch.tensor([top, at_minus_infinity, 0.0 if activation == "relu" else nan, top, 0.0]).half()
    assert torch.equal(got.nan_to_num(nan=7.0, posinf=8.0, neginf=9.0),
                       want[:, None].expand(5, 128).nan_to_num(nan=7.0, posinf=8.0, neginf=9.0)), got[:, 0]


@pytest.mark.parametrize("activation", ["none", "sigmoid", "silu"])
def test_gated_activation_epilogue(activation, device_state):
    """act([bias +] a @ bt.T) * mul through the bulk-store, transposed, workspace split-K and cluster
    split-K epilogues (ragged shapes: the gate is read only where `out` is written)."""
    torch.manual_seed(3 + len(activation))
    status, workspace = device_state
    schedules = [dict(tile_n=256, cta_group=2), dict(tile_n=128, cta_group=1, split_k=2),
                 dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1),
                 dict(tile_n=128, cta_group=1, split_k=4, cluster_split=1),
                 dict(tile_n=64, cta_group=2, split_k=2, cluster_split=1),
                 dict(tile_n=16, cta_group=1, swap_ab=1, group_m=1),
                 dict(tile_n=32, cta_group=1, swap_ab=1, group_m=1, split_k=4, cluster_split=1),
                 dict(tile_n=64, cta_group=1, swap_ab=1, group_m=1, split_k=3)]
    for cfg in schedules:
        small = bool(cfg.get("swap_ab"))
        for operation, dtype, batch, m, n, k in (("mm", "bfloat16", 1, 24 if small else 300, 520, 1024),
                                                 ("addmm", "float16", 1, 16 if small else 256, 264, 512),
                                                 ("bmm", "bfloat16", 2, 8 if small else 200, 136, 512)):
            config = _lib.Config.from_dict(cfg)
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            mul = torch.randn((*lead, m, n)).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            dev = [t.to(DEV) for t in tensors]
            out = torch.full((*lead, m, n), float("nan"), dtype=TD[dtype], device=DEV)
            status.zero_()
            _lib.gemm_act_mul(operation, dtype, activation, dev[0].data_ptr() if operation == "addmm" else 0,
                              dev[-2].data_ptr(), dev[-1].data_ptr(), mul.to(DEV).data_ptr(), out.data_ptr(),
                              batch, m, n, k, config, workspace.data_ptr(), workspace.numel(), status.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            want = O.act_ref32(activation, O.gemm_ref32(operation, *tensors)) * mul.float()
            assert_parity(out.cpu(), want, f"{activation}*mul {operation} {batch}x{m}x{n}x{k} {cfg}")


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("tile_n", [64, 128, 192, 256])
def test_gated_tiles(tile_n, cta_group, device_state):
    """The kernels that load the gate through their staging rows: every tile width, many units per CTA (few
    CTAs asked for), a half-width last wave, ragged rows and columns, a bias, batches."""
    status, workspace = device_state
    g = torch.Generator().manual_seed(tile_n + cta_group)
    for operation, batch, m, n, k, grid, tail in (("mm", 1, 1000, 1096, 200, 6, 0), ("addmm", 1, 333, 520, 72, 4, 0),
                                                  ("bmm", 3, 200, 264, 136, 2, 0), ("mm", 1, 1500, 776, 64, 16, 2)):
        if tail and tile_n % 128 != 0:
            continue
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn(*lead, m, k, generator=g).bfloat16()
        bt = (torch.randn(*lead, n, k, generator=g) * k ** -0.5).bfloat16()
        mul = torch.randn(*lead, m, n, generator=g).bfloat16()
        tensors = (a, bt) if operation != "addmm" else (torch.randn(n, generator=g).bfloat16(), a, bt)
        dev, gate = [t.to(DEV) for t in tensors], mul.to(DEV)
        out = torch.full((batch * m * n + 64,), 7.0, dtype=torch.bfloat16, device=DEV)
        config = _lib.Config.from_dict(dict(tile_n=tile_n, cta_group=cta_group, grid_ctas=grid, split_tail=tail))
        status.zero_()
        for _ in range(2):
            _lib.gemm_act_mul(operation, "bfloat16", "silu", dev[0].data_ptr() if operation == "addmm" else 0,
                              dev[-2].data_ptr(), dev[-1].data_ptr(), gate.data_ptr(), out.data_ptr(), batch, m, n, k,
                              config, workspace.data_ptr(), workspace.numel(), status.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        want = O.act_ref32("silu", O.gemm_ref32(operation, *tensors)) * mul.float()
        assert_parity(out[:-64].view(*lead, m, n).cpu(), want, f"{operation} {batch}x{m}x{n}x{k} {config.to_dict()}")
        assert bool((out[-64:] == 7.0).all())


def test_row_factor_epilogue(device_state):
    """act([bias +] a @ bt.T) * row_mul[:, None] through the bulk-store, transposed, workspace split-K
    and cluster split-K epilogues."""
    torch.manual_seed(77)
    status, workspace = device_state
    schedules = [dict(tile_n=256, cta_group=2), dict(tile_n=192, cta_group=1), dict(tile_n=128, cta_group=1, split_k=2),
                 dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1),
                 dict(tile_n=128, cta_group=1, split_k=4, cluster_split=1),
                 dict(tile_n=64, cta_group=2, split_k=2, cluster_split=1),
                 dict(tile_n=16, cta_group=1, swap_ab=1, group_m=1),
                 dict(tile_n=32, cta_group=1, swap_ab=1, group_m=1, split_k=4, cluster_split=1),
                 dict(tile_n=128, cta_group=1, swap_ab=1, group_m=1, split_k=2, cluster_split=1),
                 dict(tile_n=64, cta_group=1, swap_ab=1, group_m=1, split_k=3)]
    for cfg in schedules:
        small = bool(cfg.get("swap_ab"))
        for operation, dtype, activation, batch, m, n, k in (
                ("mm", "bfloat16", "none", 1, 24 if small else 300, 520, 1024),
                ("addmm", "float16", "relu", 1, 16 if small else 256, 264, 512),
                ("bmm", "bfloat16", "silu", 3, 8 if small else 200, 136, 512)):
            config = _lib.Config.from_dict(cfg)
            lead = (batch,) if operation == "bmm" else ()
            a = torch.randn((*lead, m, k)).to(TD[dtype])
            bt = (torch.randn((*lead, n, k)) * k ** -0.5).to(TD[dtype])
            row_mul = (torch.rand((*lead, m, 1)) + 0.5).to(TD[dtype])
            tensors = (a, bt) if operation != "addmm" else (torch.randn(n).to(TD[dtype]), a, bt)
            dev = [t.to(DEV) for t in tensors]
            out = torch.full((*lead, m, n), float("nan"), dtype=TD[dtype], device=DEV)
            status.zero_()
            _lib.gemm_act_rowmul(operation, dtype, activation, dev[0].data_ptr() if operation == "addmm" else 0,
                                 dev[-2].data_ptr(), dev[-1].data_ptr(), row_mul.to(DEV).data_ptr(), out.data_ptr(),
                                 batch, m, n, k, config, workspace.data_ptr(), workspace.numel(), status.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            want = O.act_ref32(activation, O.gemm_ref32(operation, *tensors)) * row_mul.float()
            assert_parity(out.cpu(), want, f"{activation}*row {operation} {batch}x{m}x{n}x{k} {cfg}")


def test_rms_norm_linear_matches_the_unfused_form():
    """One row reduction + one GEMM against normalise-then-project in fp32 on the CPU, on a decode and
    a prefill token count, through whichever schedules selection gives them."""
    from ayla_b200 import gemm_act_rowmul_op
    from ayla_b200.rmsnorm_linear import fold_norm_weight, rms_norm_linear

    torch.manual_seed(5)
    assert gemm_act_rowmul_op("mm", "none", "bfloat16") is torch.ops.ayla.jit_mm_rowmul_bf16.default
    hidden, features = 1024, 1536
    g = (1.0 + 0.1 * torch.randn(hidden)).to(torch.bfloat16)
    w = (torch.randn(features, hidden) * hidden ** -0.5).to(torch.bfloat16)
    folded = fold_norm_weight(w.to(DEV), g.to(DEV))
    for tokens in (8, 300):
        x = (torch.randn(tokens, hidden) * 3.0).to(torch.bfloat16)
        got = rms_norm_linear(x.to(DEV), folded, eps=1e-5)
        x32 = x.float()
        normed = x32 * torch.rsqrt(x32.pow(2).mean(-1, keepdim=True) + 1e-5) * g.float()
        want = normed @ w.float().T
        rel = float((got.cpu().float() - want).norm() / want.norm())
        # Three roundings separate the two forms (folded weight, row factor, output): each at most 2^-9.
        assert rel < 6e-3, (tokens, rel)
    with pytest.raises(ValueError, match="row factors must be"):
        gemm_act_rowmul_op("mm", "none", "bfloat16")(x.to(DEV), folded, torch.ones(300, device=DEV, dtype=torch.bfloat16)
                                                     .view(1, 300), torch.empty(300, features, device=DEV,
                                                                                dtype=torch.bfloat16))


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("rows, k", [(1, 8), (9, 248), (7, 2040), (5, 2048), (3, 4096), (2, 8184), (2, 8200), (1, 65536)])
def test_rms_row_factors(rows, k, dtype):
    """Either side of each choice of threads per row, against double precision: half an ulp for the one
    rounding, and k * 2^-24 relative for the fp32 sum (halved by the root) with 2^-22 for rsqrt."""
    from ayla_b200.rmsnorm_linear import _row_factors_op

    torch.manual_seed(rows * k)
    x = (torch.randn(rows, k) * torch.linspace(0.1, 4.0, rows).view(-1, 1)).to(TD[dtype])
    factors = torch.full((rows + 1, 1), float("nan"), dtype=TD[dtype], device=DEV)
    _row_factors_op(dtype)(x.to(DEV), 1e-5, factors[:rows])
    want = torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5)
    bound = 0.5 * O._ulp(want.float(), TD[dtype]).double() + want * (0.5 * k * 2.0 ** -24 + 2.0 ** -22)
    assert ((factors[:rows].cpu().double() - want).abs() <= bound).all()
    assert torch.isnan(factors[rows])


@pytest.mark.parametrize("m, k", [(256, 1024), (2048, 512), (40, 8192)])
def test_rms_norm_linear_behind_the_launch_that_writes_its_input(m, k):
    """x is rewritten by a GEMM directly in front of every call: with launches overlapping, the row factors and
    the projection are those of the new x, bit for bit what serialised launches give."""
    from ayla_b200.rmsnorm_linear import rms_norm_linear

    g = torch.Generator().manual_seed(k)
    sources = [(torch.randn(m, 128, generator=g) * 4.0 ** (i % 4)).bfloat16().to(DEV) for i in range(6)]
    up = (torch.randn(k, 128, generator=g) * 128 ** -0.5).bfloat16().to(DEV)
    weight = (torch.randn(192, k, generator=g) * k ** -0.5).bfloat16().to(DEV)
    x = torch.empty(m, k, dtype=torch.bfloat16, device=DEV)
    mm = gemm_op("mm", "bfloat16")

    def chain():
        outs = []
        for source in sources * 4:
            mm(source, up, x)
            outs.append(rms_norm_linear(x, weight))
        torch.cuda.synchronize()
        return torch.stack(outs)

    try:
        _lib.set_launch_overlap(False)
        serial = chain()
    finally:
        _lib.set_launch_overlap(True)
    assert torch.equal(chain(), serial)
    x32 = O.gemm_ref32("mm", sources[-1].cpu(), up.cpu()).bfloat16().float()
    factors = torch.rsqrt(x32.pow(2).mean(-1, keepdim=True) + 1e-5).bfloat16().float()
    assert_parity(serial[-1].cpu(), (x32 @ weight.cpu().float().T) * factors, f"rms_norm_linear {m}x192x{k}")


@pytest.mark.parametrize("m, n, k", [(20, 1216, 1408), (300, 520, 1024), (130, 1536, 4104), (2048, 1024, 512)])
def test_rms_norm_linear_between_launches_that_write_its_operands_and_read_its_result(m, n, k):
    """Weight and input are rewritten in front of every call, its result is read behind it and then overwritten, the row
    factors' memory is given back with the call: the same bits as with serialised launches."""
    from ayla_b200.rmsnorm_linear import rms_norm_linear

    g = torch.Generator().manual_seed(m + n + k)
    rand = lambda *shape: (torch.randn(*shape, generator=g) * 64 ** -0.25).bfloat16().to(DEV)
    xs, ws = [rand(m, 64) for _ in range(4)], [rand(n, 64) for _ in range(4)]
    up, down = rand(k, 64), rand(136, n)
    x, w = torch.empty(m, k, dtype=torch.bfloat16, device=DEV), torch.empty(n, k, dtype=torch.bfloat16, device=DEV)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    mm = gemm_op("mm", "bfloat16")

    def chain():
        results = []
        for i in range(16):
            mm(ws[i % 4], up, w)
            mm(xs[(i + i // 4) % 4], up, x)
            rms_norm_linear(x, w, out=out)
            results.append(torch.empty(m, 136, dtype=torch.bfloat16, device=DEV))
            mm(out, down, results[-1])
        torch.cuda.synchronize()
        return torch.stack(results)

    try:
        _lib.set_launch_overlap(False)
        serial = chain()
    finally:
        _lib.set_launch_overlap(True)
    for _ in range(3):
        assert torch.equal(chain(), serial)


def test_rms_norm_linear_refuses_what_the_projection_refuses():
    from ayla_b200.rmsnorm_linear import rms_norm_linear

    x = torch.randn(16, 264, device=DEV).bfloat16()
    w = torch.randn(64, 264, device=DEV).bfloat16()
    for bad_x, bad_w in ((x[:, :256], w[:, :256].contiguous()), (x.view(2, 8, 264), w), (x[:0], w), (x, w[:, :256]),
                         (x.view(-1)[4:].narrow(0, 0, 15 * 264).view(15, 264), w),
                         (x[:, :260].contiguous(), w[:, :260].contiguous())):
        with pytest.raises(ValueError):
            rms_norm_linear(bad_x, bad_w)
    y = x.clone().requires_grad_()
    assert torch.equal(rms_norm_linear(y, w), rms_norm_linear(x, w))


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("m, n, k", [
    (1, 8, 8), (5, 72, 136), (16, 200, 520), (20, 136, 1032),     # 16 and 32 columns; no split, two, four
    (64, 264, 1032), (49, 1032, 520), (130, 1000, 1000),          # 64
    (100, 4104, 520), (128, 1032, 2056), (300, 1160, 2056)])      # 128, and several column tiles
def test_swapped_swiglu(m, n, k, dtype):
    """Shapes that run with the weights on the row side: remainders of the 64 weight rows per tile, of the
    columns and of the depth, every width and cluster split."""
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).to(TD[dtype])
    gate, up = ((torch.randn(n, k, generator=g) * k ** -0.5).to(TD[dtype]) for _ in range(2))
    guard = 128
    out = torch.full((m * n + guard,), 7.0, dtype=TD[dtype], device=DEV)
    swiglu_op(dtype)(x.to(DEV), gate.to(DEV), up.to(DEV), out[:-guard].view(m, n))
    assert_parity(out[:-guard].view(m, n).cpu(), O.swiglu_ref32(x, gate, up), f"swiglu {m}x{n}x{k}")
    assert bool((out[-guard:] == 7.0).all())


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize(
    "operation, batch, m, n, k",
    [
        # one matrix per accumulator: one row, row tiles with remainders, every operand swizzle, odd depths in
        # 16-byte pieces, the most columns and depth, several units per CTA
        ("mm", 1, 1, 8, 8), ("addmm", 1, 129, 24, 24), ("mm", 1, 257, 128, 128), ("addmm", 1, 300, 120, 40),
        ("mm", 1, 128, 104, 120), ("addmm", 1, 90001, 16, 16), ("mm", 1, 150003, 96, 72),
        ("bmm", 3, 65, 128, 72), ("bmm", 2, 200, 56, 16), ("bmm", 700, 100, 40, 104), ("bmm", 1, 70, 32, 48),
        ("mm", 1, 70938, 120, 48), ("addmm", 1, 100001, 40, 80), ("bmm", 84, 286, 112, 48), ("bmm", 37, 473, 56, 40),
        # two and four, the last unit partly filled
        ("bmm", 5, 64, 64, 128), ("bmm", 3, 33, 40, 8), ("bmm", 2049, 56, 32, 56), ("bmm", 3, 8, 48, 32),
        ("bmm", 7, 32, 32, 16), ("bmm", 6, 1, 8, 24), ("bmm", 4001, 17, 24, 40),
    ])
def test_packed_kernel_equals_the_general_one(operation, batch, m, n, k, dtype):
    """Both add the same products in the same order in fp32 and round once: every bit is the same."""
    _lib.init(0)
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    lead = (batch,) if operation == "bmm" else ()
    a = torch.randn(*lead, m, k, device=DEV, generator=g).to(TD[dtype])
    bt = torch.randn(*lead, n, k, device=DEV, generator=g).to(TD[dtype])
    bias = torch.randn(n, device=DEV, generator=g).to(TD[dtype])
    guard = 64
    out = torch.full((batch * m * n + guard,), 7.0, dtype=TD[dtype], device=DEV)
    want = torch.empty(*lead, m, n, dtype=TD[dtype], device=DEV)
    status = _lib.StatusWord()
    stream = torch.cuda.current_stream().cuda_stream
    _lib.gemm_packed(operation, dtype, bias.data_ptr(), a.data_ptr(), bt.data_ptr(), out.data_ptr(), batch, m, n, k,
                     status.ptr, stream)
    _lib.gemm(operation, dtype, bias.data_ptr(), a.data_ptr(), bt.data_ptr(), want.data_ptr(), batch, m, n, k,
              _lib.Config.from_dict(dict(tile_n=64)), 0, 0, status.ptr, stream)
    torch.cuda.synchronize()
    assert status.peek() == 0
    assert torch.equal(out[:-guard].view_as(want), want)
    assert bool((out[-guard:] == 7.0).all())


@pytest.mark.parametrize("offset", [0, 8])  # results on whole sectors (written by row where that is faster), or inside them
@pytest.mark.parametrize(
    "operation,batch,m,n,k",
    [
        # rows of one sector, of a half line, of others; the last rows of a quarter and a tile; a matrix per unit, two, four
        ("mm", 1, 1, 16, 8), ("addmm", 1, 130, 32, 32), ("addmm", 1, 20001, 48, 24), ("mm", 1, 257, 112, 128),
        ("mm", 1, 90003, 80, 88), ("bmm", 3, 33, 96, 72), ("bmm", 5, 64, 48, 40), ("bmm", 3, 31, 32, 16), ("bmm", 7, 1, 16, 24),
        # as many units as the SMs take at a time and more, in the chained form
        ("bmm", 700, 40, 80, 16), ("mm", 1, 76000, 48, 32), ("mm", 1, 75700, 72, 16), ("bmm", 1300, 20, 40, 24),
    ])
def test_packed_kernels_results_by_row(operation, batch, m, n, k, offset):
    _lib.init(0)
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    lead = (batch,) if operation == "bmm" else ()
    a = torch.randn(*lead, m, k, device=DEV, generator=g).bfloat16()
    bt = torch.randn(*lead, n, k, device=DEV, generator=g).bfloat16()
    bias = torch.randn(n, device=DEV, generator=g).bfloat16()
    store = torch.full((batch * m * n + 64 + offset,), 7.0, dtype=torch.bfloat16, device=DEV)
    out = store[offset:-64]
    want = torch.empty(*lead, m, n, dtype=torch.bfloat16, device=DEV)
    status = _lib.StatusWord()
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        _lib.gemm_packed(operation, "bfloat16", bias.data_ptr(), a.data_ptr(), bt.data_ptr(), out.data_ptr(), batch, m, n, k,
                         status.ptr, stream)
    _lib.gemm(operation, "bfloat16", bias.data_ptr(), a.data_ptr(), bt.data_ptr(), want.data_ptr(), batch, m, n, k,
              _lib.Config.from_dict(dict(tile_n=64)), 0, 0, status.ptr, stream)
    torch.cuda.synchronize()
    assert status.peek() == 0
    assert torch.equal(out.view_as(want), want)
    assert bool((store[:offset] == 7.0).all()) and bool((store[-64:] == 7.0).all())


def test_a_capture_without_memory_for_a_workspace_records_a_schedule_that_needs_none(monkeypatch):
    """A product whose depth is split where SMs would idle needs a workspace, which its graph may not get."""
    monkeypatch.setattr(_lib, "capture_workspace", lambda stream, size: None)
    m, n, k = 175, 2304, 8000
    g = torch.Generator().manual_seed(5)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    want = O.mm_ref32(a, bt)
    compiler = gemm_jit_compiler("mm", "bfloat16")
    a, bt, out = a.to(DEV), bt.to(DEV), torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    compiler(a, bt, out)
    assert next(iter(compiler._cache.values())).workspace is not None
    assert_parity(out, want, "split")
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        compiler(a, bt, out)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert_parity(out, want, "captured")


def _split_product(m=175, n=2304, k=8000):
    """A specialised mm whose depth is split through a workspace, its operands and its eager result."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    a = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    bt = (torch.randn(n, k, device=DEV, generator=g) * k ** -0.5).bfloat16()
    compiler = gemm_jit_compiler("mm", "bfloat16")
    out = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    compiler(a, bt, out)
    launcher = next(iter(compiler._cache.values()))
    assert launcher.workspace is not None
    return compiler, launcher, a, bt, out


@pytest.mark.parametrize("warm", [False, True])
def test_captured_launches_have_a_workspace_of_their_graph(warm):
    """Whether or not the stream they were captured on has one: a replay touches no stream's workspace, and gives what
    the eager launch gives, bit for bit."""
    compiler, launcher, a, bt, want = _split_product()
    stream = torch.cuda.Stream()
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    if warm:
        with torch.cuda.stream(stream):
            compiler(a, bt, out)
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        compiler(a, bt, out)
        compiler(a, bt, out)
    spaces = [launcher.workspace, *(workspace for workspace, _ in launcher._per_stream.values())]
    assert len(spaces) == 1 + warm
    header = _lib.workspace_counter_bytes(launcher.config, "mm", 1, *want.shape, a.shape[1])
    for workspace in spaces:
        workspace[header:] = 7
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    for workspace in spaces:
        assert not bool(workspace[:header].any()) and bool((workspace[header:] == 7).all())


def test_graphs_and_eager_launches_of_a_split_product_overlap():
    compiler, _, a, bt, want = _split_product()
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [torch.zeros_like(want) for _ in streams]
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        compiler(a, bt, outs[0])
    torch.cuda.synchronize()
    graphs = []
    for out in outs[1:]:  # both captured on the stream that the eager launches use
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            for _ in range(4):
                compiler(a, bt, out)
        graphs.append(graph)
    for _ in range(25):
        for stream, graph in zip(streams[1:], graphs):
            with torch.cuda.stream(stream):
                graph.replay()
        with torch.cuda.stream(streams[0]):
            for _ in range(4):
                compiler(a, bt, outs[0])
        torch.cuda.synchronize()
        for out in outs:
            assert torch.equal(out, want)
            out.zero_()
        torch.cuda.synchronize()


def test_many_row_counts_share_a_workspace():
    """A layer called with any number of tokens: every second count has a k-split schedule, all on one workspace."""
    n, k = 1024, 8192
    g = torch.Generator(device=DEV).manual_seed(2)
    a = torch.randn(1024, k, device=DEV, generator=g).bfloat16()
    bt = (torch.randn(n, k, device=DEV, generator=g) * k ** -0.5).bfloat16()
    out = torch.empty(1024, n, dtype=torch.bfloat16, device=DEV)
    want = a.float() @ bt.float().T
    compiler = gemm_jit_compiler("mm", "bfloat16")
    compiler(a, bt, out)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    counts = list(range(70, 1024, 9))
    for m in counts:
        compiler(a[:m], bt, out[:m])
    for m in counts[::10]:
        compiler(a[:m], bt, out[:m])
        # fp32 sums in another order than the reference's, then one rounding to bfloat16
        torch.testing.assert_close(out[:m].float(), want[:m], atol=0.02, rtol=2.0 ** -8)
    launchers = compiler._cache.values()
    assert sum(launcher.workspace is not None for launcher in launchers) > len(counts) // 2
    assert torch.cuda.memory_allocated() - before < 64 << 20


def test_workspaces_of_graphs_are_shared_along_a_stream_and_given_back():
    size = 8 << 20
    stream = torch.cuda.current_stream().cuda_stream
    assert _lib.capture_workspace(stream, size) is None  # not capturing
    with pytest.raises(ValueError, match="counters"):
        _lib.capture_workspace(stream, 1024)
    x = torch.zeros(8, device=DEV)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    here, other = torch.cuda.Stream(), torch.cuda.Stream()
    for i in range(40):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=here):
            first = _lib.capture_workspace(here.cuda_stream, size)
            assert first is not None
            assert _lib.capture_workspace(here.cuda_stream, size // 2) == first
            other.wait_stream(here)
            second = _lib.capture_workspace(other.cuda_stream, size)
            with torch.cuda.stream(other):
                x.add_(1)
            here.wait_stream(other)
            larger = _lib.capture_workspace(here.cuda_stream, 2 * size)
            assert len({first, second, larger}) == 3
            assert _lib.capture_workspace(here.cuda_stream, size) in (first, larger)
        graph.replay()
        torch.cuda.synchronize()
        del graph
    # 40 graphs of 32 MB each; the last one or two may still be held
    assert before - torch.cuda.mem_get_info()[0] < 256 << 20
    assert bool((x == 40).all())


# The packed kernel's piped form: one B and many, a depth of one piece and of an odd number, units with rows and matrices
# missing at the end, one ring slot more or less, units enough to use every slot and accumulator again.
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("operation, batch, m, n, k", [
    ("mm", 1, 32769, 8, 8), ("addmm", 1, 70000, 96, 24), ("addmm", 1, 40003, 128, 120), ("mm", 1, 90001, 16, 40),
    ("mm", 1, 33000, 128, 128), ("bmm", 260, 129, 72, 104), ("bmm", 301, 128, 128, 64), ("bmm", 1030, 17, 24, 88),
    ("bmm", 2055, 45, 16, 120), ("bmm", 600, 1, 96, 72),
])
def test_piped_packed_kernel_equals_the_general_one(operation, batch, m, n, k, dtype, device_state):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    lead = (batch,) if operation == "bmm" else ()
    a = torch.randn((*lead, m, k), device=DEV, generator=g).to(TD[dtype])
    bt = (torch.randn((*lead, n, k), device=DEV, generator=g) * k ** -0.5).to(TD[dtype])
    bias = torch.randn(n, device=DEV, generator=g).to(TD[dtype])
    status, workspace = device_state
    status.zero_()
    outs = [torch.full((batch * m + 4, n), float("nan"), dtype=TD[dtype], device=DEV) for _ in range(2)]
    stream = torch.cuda.current_stream().cuda_stream
    bias_ptr = bias.data_ptr() if operation == "addmm" else 0
    for _ in range(2):
        _lib.gemm_packed(operation, dtype, bias_ptr, a.data_ptr(), bt.data_ptr(), outs[0].data_ptr(), batch, m, n, k,
                         status.data_ptr(), stream)
    cfg = _lib.Config.from_dict(dict(tile_n=64, cta_group=1, split_k=1, group_m=8))
    _lib.gemm(operation, dtype, bias_ptr, a.data_ptr(), bt.data_ptr(), outs[1].data_ptr(), batch, m, n, k, cfg,
              workspace.data_ptr(), workspace.numel(), status.data_ptr(), stream)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    # the same products summed in the same order of 16-deep steps; nothing past the output
    assert torch.equal(outs[0][:batch * m], outs[1][:batch * m])
    assert bool(torch.isnan(outs[0][batch * m:]).all())


@pytest.mark.parametrize("batch, m, n, k, piped", [
    (1, 70000, 96, 24, True), (2055, 45, 16, 120, True), (2984, 19, 112, 32, False), (381, 1239, 64, 56, False),
    (1, 36745, 32, 128, False), (5332, 56, 32, 56, False)])
def test_the_packed_kernels_form_is_the_faster_one(batch, m, n, k, piped):
    lead = (batch,) if batch > 1 else ()
    a = torch.zeros((*lead, m, k), device=DEV, dtype=torch.float16)
    bt = torch.zeros((*lead, n, k), device=DEV, dtype=torch.float16)
    out = torch.empty((*lead, m, n), device=DEV, dtype=torch.float16)
    _lib.init(0)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        _lib.gemm_packed("bmm" if batch > 1 else "mm", "float16", 0, a.data_ptr(), bt.data_ptr(), out.data_ptr(), batch, m,
                         n, k, 0, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    names = [event.name for event in profile.events() if "packed" in event.name]
    if not names:
        pytest.skip("no kernel names from the profiler")
    assert len(names) == 1 and ("packed_piped_kernel" in names[0]) == piped, names


# (operation, batch, m, n, k), offset of the results in elements, CTAs on an SM whose share of its shared memory each takes (0: no more
# than it needs)
@pytest.mark.parametrize("operation, batch, m, n, k, offset, ctas", [
    ("mm", 1, 125610, 80, 16, 0, 4), ("addmm", 1, 125610, 80, 16, 8, 4), ("bmm", 2500, 64, 96, 16, 0, 4),
    ("bmm", 2500, 64, 96, 16, 8, 4), ("bmm", 5400, 26, 96, 8, 0, 4),
    ("mm", 1, 75700, 72, 16, 0, 0), ("bmm", 4576, 47, 16, 16, 0, 0)])
def test_packed_ctas_take_their_share_of_an_sm_from_one_and_a_half_rounds_on(operation, batch, m, n, k, offset, ctas, tmp_path):
    _lib.init(0)
    g = torch.Generator(device=DEV).manual_seed(m)
    lead = (batch,) if operation == "bmm" else ()
    a = torch.randn(*lead, m, k, device=DEV, generator=g).half()
    bt = torch.randn(*lead, n, k, device=DEV, generator=g).half()
    bias = torch.randn(n, device=DEV, generator=g).half()
    store = torch.full((batch * m * n + 64 + offset,), 7.0, dtype=torch.float16, device=DEV)
    out = store[offset:-64]
    want = torch.empty(*lead, m, n, dtype=torch.float16, device=DEV)
    status = _lib.StatusWord()
    stream = torch.cuda.current_stream().cuda_stream
    [(name, shared)] = launched_kernels(
        lambda: _lib.gemm_packed(operation, "float16", bias.data_ptr(), a.data_ptr(), bt.data_ptr(), out.data_ptr(), batch, m, n, k,
                                 status.ptr, stream), tmp_path)
    _lib.gemm(operation, "float16", bias.data_ptr(), a.data_ptr(), bt.data_ptr(), want.data_ptr(), batch, m, n, k,
              _lib.Config.from_dict(dict(tile_n=64)), 0, 0, status.ptr, stream)
    torch.cuda.synchronize()
    assert status.peek() == 0
    assert torch.equal(out.view_as(want), want)
    assert bool((store[:offset] == 7.0).all()) and bool((store[-64:] == 7.0).all())
    assert "packed_gemm_kernel" in name, name
    per_sm, reserve = 233472, 1024
    if ctas:
        assert shared >= per_sm // ctas - reserve, (shared, per_sm // ctas - reserve)
    else:
        assert shared < per_sm // 4 - reserve


@pytest.mark.parametrize("batch, m, n, k", [(1097, 19, 96, 128), (151, 301, 80, 88), (1, 124739, 112, 112), (1, 186073, 96, 80)])
def test_results_inside_a_sector_take_the_packed_kernel_only_where_their_staging_rows_fit(batch, m, n, k):
    """Rows written straight from registers make room for a second CTA on an SM; an ``out`` that starts inside a sector
    needs staging rows, which leave room for one, and the general kernel is the faster one."""
    operation = "bmm" if batch > 1 else "mm"
    lead = (batch,) if batch > 1 else ()
    g = torch.Generator(device=DEV).manual_seed(m)
    a = torch.randn(*lead, m, k, device=DEV, generator=g).bfloat16()
    bt = torch.randn(*lead, n, k, device=DEV, generator=g).bfloat16()
    op = gemm_op(operation, "bfloat16")
    store = torch.empty(batch * m * n + 8, dtype=torch.bfloat16, device=DEV)
    results, kernels = [], []
    for offset in (0, 8):
        out = store[offset:offset + batch * m * n].view(*lead, m, n)
        op(a, bt, out)
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
            op(a, bt, out)
            torch.cuda.synchronize()
        kernels += [event.name for event in profile.events() if "packed" in event.name or "gemm_sm100" in event.name]
        results.append(out.clone())
    assert torch.equal(*results)
    if not kernels:
        pytest.skip("no kernel names from the profiler")
    assert len(kernels) == 2 and "packed" in kernels[0] and "gemm_sm100" in kernels[1], kernels
    config = select_gemm_schedule(operation, "bfloat16", m, n, k, batch).builder_config  # not the library's default
    traits = re.search(r"GemmTraits<(\d+), (\d), ", kernels[1]).groups()
    assert traits == (str(config["tile_n"]), str(config["cta_group"])), kernels


@pytest.mark.parametrize("batch, m, n, k", [(1, 70000, 96, 24), (2055, 45, 16, 120), (600, 128, 64, 40)])
def test_piped_packed_kernel_reports_a_timeout_and_keeps_infinities_apart(batch, m, n, k):
    """One B and many, several units per CTA and one."""
    operation = "bmm" if batch > 1 else "mm"
    lead = (batch,) if batch > 1 else ()
    g = torch.Generator(device=DEV).manual_seed(m)
    a = torch.randn((*lead, m, k), device=DEV, generator=g).half()
    bt = (torch.randn((*lead, n, k), device=DEV, generator=g) * k ** -0.5).half()
    out = torch.empty((*lead, m, n), device=DEV, dtype=torch.float16)
    compiler = gemm_jit_compiler(operation, "float16")
    compiler(a, bt, out)
    launcher = next(iter(compiler._cache.values()))
    assert launcher._packed
    want = out.clone()
    a.view(-1, k)[m - 1, 5] = float("inf")
    compiler(a, bt, out)
    bad = ~torch.isfinite(out.view(-1, n))
    assert bool(bad[m - 1].all()) and int(bad.sum()) == n
    a.view(-1, k)[m - 1] = 1.0
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        launcher(a, bt, out)  # no operand arrives: the waits run out
        torch.cuda.synchronize()
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    with pytest.raises(RuntimeError, match="timed out"):
        launcher(a, bt, out)
    out.zero_()
    launcher(a, bt, out)
    launcher.check_status()
    rows = torch.arange(out.numel() // n, device=DEV) != m - 1
    assert torch.equal(out.view(-1, n)[rows], want.view(-1, n)[rows])


def test_packed_kernel_through_the_ops_and_its_limits():
    a = torch.randn(300, 32, 24, device=DEV).half()
    bt = torch.randn(300, 16, 24, device=DEV).half()
    out = torch.empty(300, 32, 16, device=DEV, dtype=torch.float16)
    gemm_op("bmm", "float16")(a, bt, out)
    launcher = gemm_op_compiler("bmm", "float16")._launcher((a, bt, out))
    assert launcher._packed
    assert_parity(out.cpu(), O.bmm_ref32(a.cpu(), bt.cpu()), "packed bmm through the op")
    with pytest.raises(ValueError, match="n <= 128"):
        _lib.gemm_packed("mm", "float16", 0, a.data_ptr(), bt.data_ptr(), out.data_ptr(), 1, 8, 136, 64, 0, 0)
    # Infinities and NaN stay in their own matrix.
    a[7, 3, 5] = float("inf")
    bt[9, 2, 1] = float("nan")
    gemm_op("bmm", "float16")(a, bt, out)
    bad = ~torch.isfinite(out)
    assert bool(bad[7, 3].all()) and bool(bad[9, :, 2].all()) and int(bad.sum()) == 16 + 32
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        launcher(a, bt, out)            # the MMAs are withheld: the wait for them runs out
        torch.cuda.synchronize()
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    with pytest.raises(RuntimeError, match="timed out"):
        launcher(a, bt, out)
    launcher(a, bt, out)
    launcher.check_status()


def test_a_launcher_runs_the_schedule_it_is_given():
    """Also where the ops would take the packed kernel: the schedule's workspace is there, its result right, and the
    record for repeated calls carries it."""
    from ayla_b200.gemm_jit import GemmLauncher, GemmScheduleSeed, _DEFAULTS, packed_serves

    m, n, k = 20000, 32, 128
    assert packed_serves("mm", 1, m, n, k, torch.device(DEV))
    assert not packed_serves("mm", 1, m, n, k, torch.device(DEV), activation="relu")
    captured = {**_DEFAULTS, "tile_n": 64, "cta_group": 1, "split_k": 2}
    seed = GemmScheduleSeed(captured, {key: int(captured[key]) for key in _lib.Config.FIELDS}, (), (m, n, k))
    launcher = GemmLauncher("mm", "bfloat16", 1, m, n, k, seed, torch.device(DEV))
    assert launcher.workspace is not None and launcher.native_call()["config"] != 0
    a = torch.randn(m, k, device=DEV).bfloat16()
    bt = (torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16()
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    launcher(a, bt, out)
    launcher.check_status()
    assert_parity(out.cpu(), O.mm_ref32(a.cpu(), bt.cpu()), "explicit schedule")


def test_gemm_act_mul_op_matches_the_oracle():
    from ayla_b200 import gemm_act_mul_op

    torch.manual_seed(12)
    a = torch.randn(192, 320).to(torch.bfloat16)
    bt = (torch.randn(264, 320) * 320 ** -0.5).to(torch.bfloat16)
    mul = torch.randn(192, 264).to(torch.bfloat16)
    out = torch.empty(192, 264, dtype=torch.bfloat16, device=DEV)
    op = gemm_act_mul_op("mm", "sigmoid", "bfloat16")
    assert op is torch.ops.ayla.jit_mm_sigmoid_mul_bf16.default
    assert op(a.to(DEV), bt.to(DEV), mul.to(DEV), out) is None
    assert_parity(out.cpu(), torch.sigmoid(O.mm_ref32(a, bt)) * mul.float(), "jit_mm_sigmoid_mul_bf16")
    with pytest.raises(ValueError, match="mul must have the shape of out"):
        op(a.to(DEV), bt.to(DEV), mul[:100].contiguous().to(DEV), out)


def test_gemm_act_op_matches_the_oracle():
    from ayla_b200.gemm_jit import gemm_act_op

    torch.manual_seed(11)
    a = torch.randn(192, 320).to(torch.bfloat16)
    bt = (torch.randn(264, 320) * 320 ** -0.5).to(torch.bfloat16)
    bias = torch.randn(264).to(torch.bfloat16)
    out = torch.empty(192, 264, dtype=torch.bfloat16, device=DEV)
    op = gemm_act_op("addmm", "gelu", "bfloat16")
    assert op is gemm_act_op("addmm", "gelu", "bfloat16")
    assert op is torch.ops.ayla.jit_addmm_gelu_bf16.default
    assert gemm_act_op("mm", "none", "bfloat16") is gemm_op("mm", "bfloat16")
    assert op(bias.to(DEV), a.to(DEV), bt.to(DEV), out) is None
    assert_parity(out.cpu(), O.act_ref32("gelu", O.addmm_ref32(bias, a, bt)), "jit_addmm_gelu_bf16")


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_swiglu_variants(cta_group, dtype, device_state):
    torch.manual_seed(cta_group)
    for m, n, k in ((128, 128, 64), (200, 264, 192), (1, 8, 8), (1024, 2048, 1024), (520, 136, 72)):
        x = torch.randn(m, k).to(TD[dtype])
        wg = (torch.randn(n, k) * k ** -0.5).to(TD[dtype])
        wu = (torch.randn(n, k) * k ** -0.5).to(TD[dtype])
        out, status = run_abi("swiglu", dtype, (x, wg, wu), dict(cta_group=cta_group, group_m=2), device_state)
        assert status == 0
        assert_parity(out, O.swiglu_ref32(x, wg, wu), f"swiglu {m}x{n}x{k} cta_group={cta_group}")


# ------------------------------------------------------------- exactness properties

def test_identity_and_power_of_two_scaling_are_exact(device_state):
    torch.manual_seed(5)
    for dtype in ("bfloat16", "float16"):
        td = TD[dtype]
        a = torch.randn(300, 256).to(td)
        eye = torch.eye(256).to(td)
        for cfg in (dict(tile_n=256, cta_group=2), dict(tile_n=64, cta_group=1, split_k=2), None):
            out, _ = run_abi("mm", dtype, (a, eye), cfg, device_state)
            assert torch.equal(out.cpu(), a), cfg                      # a @ I^T == a, bit for bit
        bt = torch.randn(264, 256).to(td)
        base, _ = run_abi("mm", dtype, (a, bt), None, device_state)
        scaled, _ = run_abi("mm", dtype, ((a.float() * 4).to(td), (bt.float() * 0.5).to(td)), None, device_state)
        assert torch.equal(scaled.float().cpu(), base.float().cpu() * 2)  # exact in binary floating point


def test_small_k_results_are_bit_exact(device_state):
    """For K <= 128 every partial sum of 16-bit products fits fp32 exactly often enough
    that the reference pins bit-equality with torch.mm
    (tests/gemm_collection/test_correctness.py:216-234, :302-314); same here against the
    CPU oracle, allowing last-bit flips on at most 0.1 % of elements."""
    for m, n, k, seed in ((128, 256, 128, 7), (3, 256, 64, 3), (128, 256, 64, 128), (256, 256, 64, 256)):
        g = torch.Generator().manual_seed(seed)
        a = torch.randn(m, k, generator=g).bfloat16()
        bt = torch.randn(n, k, generator=g).bfloat16()
        out, _ = run_abi("mm", "bfloat16", (a, bt), None, device_state)
        want = O.gemm_ref("mm", torch.bfloat16, a, bt)
        differing = int((out.cpu().view(torch.int16) != want.view(torch.int16)).sum())
        assert differing <= max(1, out.numel() // 1000), (m, n, k, differing)


def test_repeated_launches_are_deterministic(device_state):
    """Split-K partials are reduced in a fixed order, so results do not depend on
    which CTA finishes last."""
    op, tensors = O.make_inputs("C2b", "bfloat16", scale_down=4)
    cfg = dict(tile_n=64, cta_group=1, split_k=8)
    first, _ = run_abi(op, "bfloat16", tensors, cfg, device_state)
    for _ in range(5):
        again, status = run_abi(op, "bfloat16", tensors, cfg, device_state)
        assert status == 0 and torch.equal(first, again)


# ------------------------------------------------------------ the benchmark configs

def run_op(operation, dtype, tensors):
    dev = [t.to(DEV) for t in tensors]
    if operation == "swiglu":
        out = torch.empty((dev[0].shape[0], dev[1].shape[0]), dtype=dev[0].dtype, device=DEV)
        swiglu_op(dtype)(*dev, out)
        compiler = swiglu_op_compiler(dtype)
    else:
        a, bt = dev[-2:]
        out = torch.empty((*a.shape[:-1], bt.shape[-2]), dtype=a.dtype, device=DEV)
        gemm_op(operation, dtype)(*dev, out)
        compiler = gemm_op_compiler(operation, dtype)
    torch.cuda.synchronize()
    for launcher in compiler._cache.values():
        launcher.check_status()
    return out


@pytest.mark.parametrize("config,dtype", [("C1", "bfloat16"), ("C2a", "bfloat16"), ("C2a", "float16"),
                                          ("C2b", "bfloat16"), ("C2b", "float16"), ("C3a", "bfloat16"),
                                          ("C3b", "bfloat16"), ("C4", "bfloat16")])
def test_benchmark_configs_full_size(config, dtype):
    operation, tensors = O.make_inputs(config, dtype)
    out = run_op(operation, dtype, tensors)
    parity = assert_parity(out, O.gemm_ref32(operation, *tensors), config)
    print(f"\n{config} {dtype}: {parity}")


@pytest.mark.parametrize("index", range(len(O.SWEEP_M) * len(O.SWEEP_NK)))
def test_dynamic_m_sweep(index):
    (m, n, k), (a, bt) = O.make_sweep_inputs(index)
    out = run_op("mm", "bfloat16", (a, bt))
    assert_parity(out, O.mm_ref32(a, bt), f"sweep m={m} n={n} k={k}")


def test_linearity_at_full_size():
    """out(a1 + a2) == out(a1) + out(a2) within rounding, at the 4096^3 size, with
    operands whose sums are exact in bf16 (small integers)."""
    g = torch.Generator().manual_seed(9)
    a1 = torch.randint(-3, 4, (4096, 4096), generator=g).bfloat16()
    a2 = torch.randint(-3, 4, (4096, 4096), generator=g).bfloat16()
    bt = torch.randint(-2, 3, (4096, 4096), generator=g).bfloat16()
    o1 = run_op("mm", "bfloat16", (a1, bt)).float()
    o2 = run_op("mm", "bfloat16", (a2, bt)).float()
    o12 = run_op("mm", "bfloat16", (a1 + a2, bt)).float()
    # integer sums below 2^24 are exact in the fp32 accumulator; only the final rounding differs
    exact = torch.mm((a1 + a2).float(), bt.float().t()).bfloat16().float()
    assert torch.equal(o12.cpu(), exact)
    assert ((o1 + o2) - o12).abs().max().item() <= 2 * float(O._ulp(o12.abs().max().cpu(), torch.bfloat16))


# ------------------------------------------------------------------ error behaviour

def test_op_level_validation():
    a = torch.randn(64, 64, device=DEV, dtype=torch.bfloat16)
    out = torch.empty(64, 64, device=DEV, dtype=torch.bfloat16)
    op = gemm_op("mm", "bfloat16")
    with pytest.raises(ValueError, match="contiguous"):
        op(a.t(), a, out)
    with pytest.raises(ValueError, match="expected dtype"):
        op(a.half(), a, out)
    with pytest.raises(ValueError, match="CUDA tensors"):
        op(a.cpu(), a, out)
    with pytest.raises(ValueError, match="bt must be"):
        op(a, torch.empty(64, 32, device=DEV, dtype=torch.bfloat16), out)
    with pytest.raises(ValueError, match="out must be"):
        op(a, a, torch.empty(64, 32, device=DEV, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="no schedule"):
        op(torch.empty(8, 12, device=DEV, dtype=torch.bfloat16), torch.empty(8, 12, device=DEV, dtype=torch.bfloat16),
           torch.empty(8, 8, device=DEV, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="bias must be"):
        gemm_op("addmm", "bfloat16")(torch.empty(32, device=DEV, dtype=torch.bfloat16), a, a, out)


@pytest.mark.parametrize("m, n, k", [(1024, 1024, 8192), (175, 2304, 8000), (4451, 2240, 7040)])
def test_no_schedule_leaves_a_workspace_alone_that_the_default_does_not_need(m, n, k, device_state):
    """cfg == NULL is the schedule that ayla_b200_default_config reports: where that one asks for no workspace, a lent
    one need not be clean, and two streams may lend the same."""
    status, _ = device_state
    status.zero_()
    assert _lib.workspace_bytes(_lib.default_config("mm", "bfloat16", 1, m, n, k), "mm", 1, m, n, k) == 0
    g = torch.Generator(device=DEV).manual_seed(m)
    a = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    bt = (torch.randn(n, k, device=DEV, generator=g) * k ** -0.5).bfloat16()
    lent = torch.full((64 << 20,), 7, dtype=torch.uint8, device=DEV)
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    _lib.gemm("mm", "bfloat16", 0, a.data_ptr(), bt.data_ptr(), out.data_ptr(), 1, m, n, k, None, lent.data_ptr(),
              lent.numel(), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert bool((lent == 7).all())
    # fp32 sums in another order than the reference's, then one rounding to bfloat16
    torch.testing.assert_close(out.float(), a.float() @ bt.float().T, atol=0.02, rtol=2.0 ** -8)


def test_abi_workspace_and_init_errors(device_state):
    status, workspace = device_state
    a = torch.randn(256, 1024, device=DEV, dtype=torch.bfloat16)
    out = torch.empty(256, 256, device=DEV, dtype=torch.bfloat16)
    cfg = _lib.Config.from_dict(dict(tile_n=64, cta_group=1, split_k=4))
    with pytest.raises(ValueError, match="workspace"):
        _lib.gemm("mm", "bfloat16", 0, a.data_ptr(), a.data_ptr(), out.data_ptr(), 1, 256, 256, 1024, cfg,
                  workspace.data_ptr(), 1024, 0, torch.cuda.current_stream().cuda_stream)
    with pytest.raises(ValueError, match="workspace"):
        _lib.gemm("mm", "bfloat16", 0, a.data_ptr(), a.data_ptr(), out.data_ptr(), 1, 256, 256, 1024, cfg,
                  0, 0, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()


@pytest.mark.parametrize("m", [3, 128, 256])
def test_dynamic_m_matmul(m):
    """tests/gemm_collection/test_correctness.py:302-314 of the reference: m in {3, 128, 256},
    n = 256, k = 64, seed = m; one cached schedule per shape."""
    from ayla_b200.dynamic_m import make_dynamic_m_matmul

    op = make_dynamic_m_matmul(256, 64, namespace=f"ayla_b200_dynamic_m_test_{m}")
    g = torch.Generator().manual_seed(m)
    lhs = torch.randn(m, 64, generator=g).bfloat16()
    rhs = torch.randn(256, 64, generator=g).bfloat16()
    out = op(lhs.to(DEV), rhs.to(DEV))
    assert out.shape == (m, 256)
    want = O.gemm_ref("mm", torch.bfloat16, lhs, rhs)
    differing = int((out.cpu().view(torch.int16) != want.view(torch.int16)).sum())
    assert differing <= max(1, out.numel() // 1000)


# ------------------------------------------------------- failure detection (no GPU fault)

@pytest.mark.parametrize("cfg", [dict(tile_n=128, cta_group=1), dict(tile_n=256, cta_group=2),
                                 dict(tile_n=16, cta_group=1, swap_ab=1, group_m=1)])
def test_bounded_wait_reports_a_stalled_pipeline_and_the_context_survives(cfg, device_state):
    """A launch whose producer never delivers operands must not hang: the MMA warp's wait
    runs out, the kernel finishes, the status word says which wait gave up (code 2 = waiting
    for operands), and the next ordinary launch on the same context is correct."""
    lib = _lib.load()
    g = torch.Generator().manual_seed(3)
    a = torch.randn(300, 264, generator=g).bfloat16()
    bt = torch.randn(264, 264, generator=g).bfloat16()
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        _, status = run_abi("mm", "bfloat16", (a, bt), cfg, device_state)
        assert status & 0xFF in (2, 4), hex(status)   # the MMA wait (2) or, racing it, the epilogue's (4)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    device_state[1].zero_()
    out, status = run_abi("mm", "bfloat16", (a, bt), cfg, device_state)
    assert status == 0
    assert_parity(out, O.mm_ref32(a, bt), "launch after a timed-out one")


def test_launcher_check_status_raises_on_timeout():
    lib = _lib.load()
    compiler = gemm_jit_compiler("mm", "bfloat16")
    a = torch.randn(256, 256, device=DEV, dtype=torch.bfloat16)
    out = torch.empty(256, 256, device=DEV, dtype=torch.bfloat16)
    compiler(a, a, out)
    [launcher] = compiler._cache.values()
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        compiler(a, a, out)
        with pytest.raises(RuntimeError, match="timed out"):
            launcher.check_status()
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    compiler(a, a, out)
    launcher.check_status()
    torch.testing.assert_close(out, a @ a.T, atol=0.125, rtol=0.02)


def test_timed_out_split_k_launch_is_reported_by_the_next_call_without_the_debug_switch(monkeypatch):
    """The status word sits in pinned host memory and is read before every launch: after a k-split
    launch that ran into a bounded wait, the next call of that shape raises (no AYLA_B200_DEBUG, no
    explicit check_status), and the call after it is correct -- the arrival counters a timed-out
    k-split may leave behind are cleared with the report."""
    from ayla_b200.gemm_jit import GemmLauncher, GemmScheduleSeed, _DEFAULTS

    monkeypatch.delenv("AYLA_B200_DEBUG", raising=False)
    lib = _lib.load()
    m, n, k = 256, 256, 2048
    captured = {**_DEFAULTS, "tile_n": 64, "cta_group": 1, "split_k": 4}
    seed = GemmScheduleSeed(captured, {key: int(captured[key]) for key in _lib.Config.FIELDS}, (), (m, n, k))
    launcher = GemmLauncher("mm", "bfloat16", 1, m, n, k, seed, torch.device(DEV))
    assert launcher.workspace is not None and not launcher._debug
    g = torch.Generator().manual_seed(11)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    da, dbt = a.to(DEV), bt.to(DEV)
    out = torch.empty(m, n, device=DEV, dtype=torch.bfloat16)
    launcher(da, dbt, out)
    torch.cuda.synchronize()
    assert launcher.status.peek() == 0
    assert_parity(out, O.mm_ref32(a, bt), "k-split launch before the failure")
    try:
        lib.ayla_b200_set_wait_timeout_ms(30)
        lib.ayla_b200_debug_set_flags(1)
        launcher(da, dbt, out)          # the producer delivers nothing: the waits run out
        torch.cuda.synchronize()
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert launcher.status.peek() & 0xFF in (2, 4)
    with pytest.raises(RuntimeError, match="timed out"):
        launcher(da, dbt, out)
    out.zero_()
    launcher(da, dbt, out)
    torch.cuda.synchronize()
    assert launcher.status.peek() == 0
    assert_parity(out, O.mm_ref32(a, bt), "k-split launch after a reported timeout")


@pytest.mark.parametrize("config", [
    dict(tile_n=128, cta_group=1, split_k=4), dict(tile_n=256, cta_group=2, split_k=3),  # the shared sum
    dict(tile_n=64, cta_group=1, split_k=3, grid_ctas=6)])                               # the last arriver's
def test_timed_out_k_splits_leave_their_counters_at_zero(config, device_state):
    """Nobody can clear the workspace of a captured launch: the launch after one whose waits ran out finds it clean."""
    m, n, k = 500, 520, 2048
    g = torch.Generator().manual_seed(6)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    lib = _lib.load()
    assert _lib.workspace_bytes(_lib.Config.from_dict(config), "mm", 1, m, n, k) > 0
    try:
        lib.ayla_b200_set_wait_timeout_ms(20)
        lib.ayla_b200_debug_set_flags(1)
        _, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert status & 0xFF != 0
    assert not bool(device_state[1][:65536].any())
    out, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    assert status == 0
    assert_parity(out, O.mm_ref32(a, bt), f"after a timed-out k-split {config}")


@pytest.mark.parametrize("config", [
    dict(tile_n=64, cta_group=1, split_k=2), dict(tile_n=128, cta_group=1, split_k=4),
    dict(tile_n=64, cta_group=2, split_k=2), dict(tile_n=16, cta_group=1, swap_ab=1, split_k=4, group_m=1)])
def test_timed_out_cluster_split_leaves_the_context_usable(config, device_state):
    """A cluster k-split whose loads are withheld: every CTA gives up in its own time, and none leaves while
    another may still send partial sums into its shared memory."""
    m, n, k = (8 if config.get("swap_ab") else 512), 1024, 2048
    g = torch.Generator().manual_seed(4)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    config = dict(config, cluster_split=1)
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(20)
        lib.ayla_b200_debug_set_flags(1)
        _, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert status & 0xFF != 0
    out, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    assert status == 0
    assert_parity(out, O.mm_ref32(a, bt), f"after a timed-out cluster split {config}")


@pytest.mark.parametrize("config", [dict(tile_n=128, split_k=1), dict(tile_n=128, split_k=2), dict(tile_n=128, split_k=4),
                                    dict(tile_n=256, split_k=1), dict(tile_n=256, split_k=2), dict(tile_n=256, split_k=4)])
@pytest.mark.parametrize("m", [40, 128])
def test_timed_out_pairs_of_few_rows_leave_the_context_usable(m, config, device_state):
    """Pairs on 128-row tiles with their loads withheld, whole and in clusters of two and four pairs."""
    n, k = 1024, 2048
    g = torch.Generator().manual_seed(m)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    config = dict(config, cta_group=2, cluster_split=int(config["split_k"] > 1))
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(20)
        lib.ayla_b200_debug_set_flags(1)
        _, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert status & 0xFF != 0
    out, status = run_abi("mm", "bfloat16", (a, bt), config, device_state)
    assert status == 0
    assert_parity(out, O.mm_ref32(a, bt), f"after timed-out pairs {config}")


@pytest.mark.parametrize("m, n, k", [(8, 1024, 2048), (100, 1024, 1024), (60, 4096, 512)])
def test_timed_out_swapped_swiglu_leaves_the_context_usable(m, n, k, device_state):
    """The SwiGLU form of few rows, its k split across a cluster or (the last) not split, with its loads withheld."""
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, k, generator=g).bfloat16()
    gate, up = ((torch.randn(n, k, generator=g) * k ** -0.5).bfloat16() for _ in range(2))
    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(20)
        lib.ayla_b200_debug_set_flags(1)
        _, status = run_abi("swiglu", "bfloat16", (x, gate, up), None, device_state)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert status & 0xFF != 0
    out, status = run_abi("swiglu", "bfloat16", (x, gate, up), None, device_state)
    assert status == 0
    assert_parity(out.cpu(), O.swiglu_ref32(x, gate, up), f"after a timed-out launch {m}x{n}x{k}")


@pytest.mark.parametrize("config", [dict(tile_n=64, cta_group=1, grid_ctas=3), dict(tile_n=256, cta_group=1, grid_ctas=2),
                                    dict(tile_n=128, cta_group=2, grid_ctas=4), dict(tile_n=256, cta_group=2, grid_ctas=4)])
def test_timed_out_gated_launch_leaves_the_context_usable(config, device_state):
    """A gated launch whose operands never come, with several units per CTA: its gate boxes do come, and after
    the abort none is asked for again.  The next launch is correct."""
    status, workspace = device_state
    m, n, k = 700, 1024, 256
    g = torch.Generator().manual_seed(8)
    a = torch.randn(m, k, generator=g).bfloat16()
    bt = (torch.randn(n, k, generator=g) * k ** -0.5).bfloat16()
    mul = torch.randn(m, n, generator=g).bfloat16()
    da, dbt, dmul = a.to(DEV), bt.to(DEV), mul.to(DEV)
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)

    def launch():
        status.zero_()
        _lib.gemm_act_mul("mm", "bfloat16", "sigmoid", 0, da.data_ptr(), dbt.data_ptr(), dmul.data_ptr(), out.data_ptr(),
                          1, m, n, k, _lib.Config.from_dict(config), workspace.data_ptr(), workspace.numel(),
                          status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return int(status.item())

    lib = _lib.load()
    try:
        lib.ayla_b200_set_wait_timeout_ms(20)
        lib.ayla_b200_debug_set_flags(1)
        assert launch() & 0xFF in (2, 4)
    finally:
        lib.ayla_b200_debug_set_flags(0)
        lib.ayla_b200_set_wait_timeout_ms(2000)
    assert launch() == 0
    assert_parity(out.cpu(), O.act_ref32("sigmoid", O.gemm_ref32("mm", a, bt)) * mul.float(), f"after a timeout {config}")


def test_random_shapes_through_the_public_ops():
    """Schedule selection on shapes nobody measured: transferred table entries (trimmed tiles, 192-wide
    tiles, cluster k-splits, eviction hints) and the default heuristic must all stay correct on ragged
    extents.  Checked against the GPU's own fp32-accumulating matmul with the reference's test tolerances
    (tests/test_gemm_jit.py:59-63 of the reference)."""
    import random

    rng = random.Random(1234)
    torch.manual_seed(1234)
    picks_m = [1, 3, 8, 17, 33, 64, 100, 128, 200, 256, 384, 512, 777, 1024, 1536, 2048, 3000]
    picks_n = [8, 64, 136, 512, 1000, 2048, 4096, 6144, 7168, 8192, 11008, 14336]
    picks_k = [8, 72, 128, 520, 1024, 2048, 4096, 5120, 8192, 14336]
    for trial in range(120):
        operation = rng.choice(["mm", "mm", "addmm", "bmm"])
        m, n, k = rng.choice(picks_m), rng.choice(picks_n), rng.choice(picks_k)
        batch = rng.choice([2, 3, 5]) if operation == "bmm" else 1
        if batch * (m * k + n * k + m * n) > 160e6:
            k = min(k, 1024)
        dtype = rng.choice(["bfloat16", "float16"])
        td = TD[dtype]
        lead = (batch,) if operation == "bmm" else ()
        a = torch.randn((*lead, m, k), device=DEV).to(td)
        bt = (torch.randn((*lead, n, k), device=DEV) * k ** -0.5).to(td)
        out = torch.full((*lead, m, n), float("nan"), device=DEV, dtype=td)
        if operation == "addmm":
            bias = torch.randn(n, device=DEV).to(td)
            gemm_op(operation, dtype)(bias, a, bt, out)
            want = torch.addmm(bias.float(), a.float(), bt.float().T)
        else:
            gemm_op(operation, dtype)(a, bt, out)
            want = a.float() @ bt.float().transpose(-1, -2)
        torch.testing.assert_close(out.float(), want, atol=0.125, rtol=0.02,
                                   msg=lambda msg: f"{operation} {dtype} {batch}x{m}x{n}x{k}: {msg}")


def test_random_shapes_through_the_fused_ops():
    """SwiGLU, activation and gated epilogues on ragged shapes nobody measured, against fp32 math on
    the GPU rounded once (same tolerances as the plain ops)."""
    import random

    from ayla_b200 import ACTIVATIONS, gemm_act_mul_op, gemm_act_op

    rng = random.Random(4321)
    torch.manual_seed(4321)
    acts = {"relu": torch.relu, "sigmoid": torch.sigmoid, "silu": torch.nn.functional.silu,
            "gelu": torch.nn.functional.gelu,
            "gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}
    assert set(acts) == set(ACTIVATIONS) - {"none"}
    for trial in range(60):
        m = rng.choice([1, 8, 24, 64, 130, 256, 512, 1000, 2048])
        n = rng.choice([8, 72, 512, 1000, 4096, 6144, 14336])
        k = rng.choice([8, 136, 1024, 4096, 5120])
        dtype = rng.choice(["bfloat16", "float16"])
        td = TD[dtype]
        a = torch.randn(m, k, device=DEV).to(td)
        w0 = (torch.randn(n, k, device=DEV) * k ** -0.5).to(td)
        out = torch.full((m, n), float("nan"), device=DEV, dtype=td)
        kind = rng.choice(["swiglu", "act", "gated"])
        if kind == "swiglu":
            w1 = (torch.randn(n, k, device=DEV) * k ** -0.5).to(td)
            swiglu_op(dtype)(a, w0, w1, out)
            want = torch.nn.functional.silu(a.float() @ w0.float().T) * (a.float() @ w1.float().T)
            label = "swiglu"
        else:
            act = rng.choice(sorted(acts))
            with_bias = rng.random() < 0.5
            bias = torch.randn(n, device=DEV).to(td)
            want = a.float() @ w0.float().T
            if with_bias:
                want = want + bias.float()
            want = acts[act](want)
            operation = "addmm" if with_bias else "mm"
            lead = (bias,) if with_bias else ()
            if kind == "act":
                gemm_act_op(operation, act, dtype)(*lead, a, w0, out)
            else:
                mul = torch.randn(m, n, device=DEV).to(td)
                gemm_act_mul_op(operation, act, dtype)(*lead, a, w0, mul, out)
                want = want * mul.float()
            label = f"{kind} {operation} {act}"
        torch.testing.assert_close(out.float(), want, atol=0.125, rtol=0.02,
                                   msg=lambda msg: f"{label} {dtype} {m}x{n}x{k}: {msg}")
