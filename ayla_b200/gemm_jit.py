"""mm, addmm and bmm ops backed by the prebuilt sm_100a kernels.

Drop-in for the reference's JIT GEMM front end (ayla/gemm_jit.py): the same
names, signatures and return types --

    op = gemm_op("mm", "bfloat16")      # op(a, bt, out): out = a @ bt.T
    op(a, bt, out)

``gemm_op(operation, dtype)`` returns the cached ``torch.ops.ayla.jit_{op}_{f16|bf16}``
overload taking ``(a, bt, out)``, ``(bias, a, bt, out)`` or the batched
``(a[B,M,K], bt[B,N,K], out[B,M,N])`` (ayla/gemm_jit.py:396-411);
``measured_gemm_configs`` lists the schedules measured on exactly this shape and
``select_gemm_schedule`` picks the one a launch will use (ayla/gemm_jit.py:168-222).
A schedule here is a tile width / CTA pairing / split-K / raster choice for the
tcgen05 kernel rather than a Hopper pass recipe, and "compiling" a shape only
selects one: the kernels are already built into ``libayla_b200.so``.
"""

from __future__ import annotations

import math
import os
import threading
import weakref
from dataclasses import dataclass, replace
from functools import cache

import torch

from . import _lib
from .gemm_schedule_table import CONFIGS, SCHEDULES
from .jit_compiler import OpTemplate, ShapeSpecializingJITCompiler
from .torch_custom_call import DEFAULT_NAMESPACE, OperandKind, TensorSpec

_SHORT_DTYPES = {"float16": "f16", "bfloat16": "bf16"}
_TORCH_DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}
_OPERATIONS = ("mm", "addmm", "bmm")
ACTIVATIONS = ("none", "relu", "sigmoid", "silu", "gelu", "gelu_tanh")

# Table entries omit default fields.
_DEFAULTS: dict[str, object] = {
    "tile_n": 256,
    "cta_group": 1,
    "swap_ab": 0,
    "split_k": 1,
    "group_m": 8,
    "grid_ctas": 0,
    "l2_hint_a": 0,
    "l2_hint_b": 0,
    "split_tail": 0,
    "l2_prefetch": 0,
    "cluster_split": 0,
    "stream_k": 0,
    "tile_rows": 0,
    "early_prefetch": 0,
}

# A measured schedule is transferred to another shape only when the shapes are
# this close in summed |log2| of (batch, m, n, k); beyond that the shape-aware
# default of the library is the better guess.
_MAX_TRANSFER_DISTANCE = 2.0


@dataclass(frozen=True)
class GemmScheduleSeed:
    captured_config: dict[str, object]
    builder_config: dict[str, object] | None
    adaptations: tuple[str, ...]
    source_shape: tuple[int, int, int] | None
    source_percentage_of_torch: float | None = None
    post_builder_passes: tuple[str, ...] = ()
    unsplit_config: dict[str, object] | None = None  # the schedule before its depth was split further


def _builder_config(captured: dict[str, object]) -> dict[str, object]:
    """The fields the launcher passes to the library (``struct ayla_b200_config``)."""
    return {key: int(captured[key]) for key in _lib.Config.FIELDS}  # type: ignore[arg-type]


def _shape_supported(m: int, n: int, k: int, batch: int) -> bool:
    # 16-byte row pitch for TMA: n and k in multiples of 8 elements.  (The
    # reference needs k % 64 == 0, ayla/gemm_jit.py:134, :234; K tails are
    # zero-filled by TMA here, so multiples of 8 suffice.)
    return min(batch, m, n, k) > 0 and n % 8 == 0 and k % 8 == 0


def _legal(config: dict[str, object], operation: str, dtype: str, m: int, n: int, k: int,
           batch: int) -> bool:
    cfg = _lib.Config.from_dict(config)
    return _lib.config_valid(cfg, operation, dtype, batch, m, n, k)


def _seed(captured: dict[str, object], operation: str, dtype: str, m: int, n: int, k: int,
          batch: int, source: tuple[int, int, int, int], exact: bool) -> GemmScheduleSeed | None:
    if not _shape_supported(m, n, k, batch):
        return None
    if not _legal(captured, operation, dtype, m, n, k, batch):
        return None
    percentage = captured.get("percentage_of_torch")
    return GemmScheduleSeed(
        captured,
        _builder_config(captured),
        () if exact else (f"nearest measured shape {source}",),
        source[1:],
        float(percentage) if isinstance(percentage, (int, float)) else None,
    )


_SM_COUNT = 148
# Clusters of this many CTAs that run at the same time on a B200: each lies within one GPC.
_CLUSTERS_AT_ONCE = {1: 148, 2: 74, 4: 33, 8: 15}


def _waves(config: dict[str, object], batch: int, m: int, n: int) -> int:
    """Passes of the persistent grid a schedule needs on this shape (whole CTAs or clusters at
    a time).  A schedule measured at one wave is a poor guess for a shape where it needs two."""
    pair = int(config["cta_group"])
    rows, cols = (n, m) if config["swap_ab"] else (m, n)
    tile_rows = int(config["tile_rows"]) or 128
    row_tiles = -(-rows // (tile_rows if config["swap_ab"] else 128 * pair))
    tiles = batch * row_tiles * -(-cols // int(config["tile_n"]))
    split = int(config["split_k"])
    if config["cluster_split"]:
        cluster = split * pair
        return -(-tiles // _CLUSTERS_AT_ONCE.get(cluster, max(1, _SM_COUNT // cluster)))
    units = tiles * (1 if config["split_tail"] else split)
    return -(-units // (_SM_COUNT // pair))


def _column_padding(config: dict[str, object], m: int, n: int) -> float:
    """Share of a schedule's tile columns that lie past the matrix on this shape (the swapped form
    tiles the token dimension): a 128-column tile on 64 output columns computes half of itself for
    nothing, however well it did where it was measured on 128."""
    cols = m if config["swap_ab"] else n
    tile = int(config["tile_n"])
    padded = -(-cols // tile) * tile
    return (padded - cols) / padded


def measured_gemm_configs(operation: str, dtype: str, m: int, n: int, k: int,
                          batch: int = 1) -> tuple[dict[str, object], ...]:
    """All schedules measured on exactly this shape, winner first, as fresh copies."""
    indices = SCHEDULES.get((operation, dtype), {}).get((batch, m, n, k), ())
    return tuple({**_DEFAULTS, **CONFIGS[index]} for index in indices)


def _fit_labels(before: dict[str, object], after: dict[str, object], m: int) -> tuple[str, ...]:
    """What ``ayla_b200_fit_depth`` made of a schedule, in words."""
    if m <= 128 and after["cta_group"] == 2 and not (before["cta_group"] == 2 and before["tile_n"] == after["tile_n"]):
        return ("pairs on 128 rows",)
    labels = []
    if (after["tile_n"], after["cta_group"]) != (before["tile_n"], before["cta_group"]):
        labels.append("tiles of another width or pairing")
    if int(after["split_k"]) > 1:
        if any(after[key] != before[key] for key in ("split_k", "split_tail", "cluster_split")):
            labels.append("depth split where SMs would idle")
    else:
        if int(before["split_k"]) > 1:
            labels.append("depth whole")
        if after["split_tail"] != before["split_tail"]:
            labels.append("last wave in halves" if after["split_tail"] else "last wave of whole tiles")
    return tuple(labels) or ("fitted to the shape",)


def _fitted(seed: GemmScheduleSeed | None, operation: str, dtype: str, m: int, n: int, k: int, batch: int,
            activation: str) -> GemmScheduleSeed | None:
    """The schedule as ``ayla_b200_fit_depth_act`` fits it to the shape: its depth split where SMs would idle, its last wave
    whole, in halves or split, tiles that all run at once, pairs on 128 rows."""
    if seed is None or seed.builder_config is None:
        return seed
    fitted = _lib.fit_depth(_lib.Config.from_dict(seed.builder_config), operation, dtype, batch, m, n, k, activation).to_dict()
    if fitted == seed.builder_config:
        return seed
    captured = {**seed.captured_config, **fitted}
    return replace(seed, captured_config=captured, builder_config=_builder_config(captured),
                   unsplit_config=seed.builder_config,
                   adaptations=(*seed.adaptations, *_fit_labels(seed.builder_config, fitted, m)))


def _streams_weights(operation: str, batch: int, m: int, n: int, k: int) -> bool:
    """A few rows against a large weight."""
    return operation != "bmm" and batch == 1 and m <= 64 and n >= 1024 and k >= 1024


def _ctas(config: dict[str, object], m: int, n: int) -> int:
    """CTAs that a schedule puts to work, cluster members included."""
    pair = int(config["cta_group"])
    rows, cols = (n, m) if config["swap_ab"] else (m, n)
    height = (int(config["tile_rows"]) or 128) if config["swap_ab"] else 128 * pair
    return -(-rows // height) * -(-cols // int(config["tile_n"])) * int(config["split_k"]) * pair


def _rule_streams_better(neighbour: dict[str, object], rule: dict[str, object], activation: str, m: int, n: int,
                         k: int) -> bool:
    """Whether the library's rule for a stream of weights is the better guess than a neighbour's schedule.

    Over 483 shapes of up to 64 rows timed with both, the rule is taken for 297: the geometric mean of the times is 0.938
    of the neighbours', two are slower by 2 to 3 %; with the rule always it is 0.948 and 58 are slower, up to 1.66 times.
    It is better (us, neighbour -> rule)
     * where it puts more SMs to work, a short product against whole rows of the weight aside (32x8192x1856 20.4 -> 10.4,
       30x4928x4608 18.6 -> 13.0; but of 20 k-blocks or fewer 45x2752x1088 7.2 -> 7.6);
     * against clusters that tile the rows, from 24 k-blocks on and with nothing fused (58x1152x2816 8.7 -> 6.9; with a
       gate 41x9216x3840 18.1 -> 23.3, of 18 k-blocks 53x1560x1112 6.0 -> 6.6);
     * against the same tiles without a hint that the weight leaves L2 first (4x2752x1280 5.9 -> 5.3).
    Not against whole rows of the weight on as many SMs (63x7232x1280 8.4 -> 10.7, gated 41x4416x1728 9.2 -> 15.3), and not
    with clusters of four against eight that run at once (2x1408x7680 7.6 -> 8.7)."""
    waves, rule_waves = _waves(neighbour, 1, m, n), _waves(rule, 1, m, n)
    if waves != rule_waves:
        return rule_waves < waves
    k_blocks = -(-k // 64)
    share = _ctas(rule, m, n) / _ctas(neighbour, m, n)
    if not neighbour["swap_ab"]:
        if int(neighbour["split_k"]) == 1:
            return share > 1.05 and k_blocks > 20
        return share > 1.1 or (activation == "none" and k_blocks >= 24)
    unhinted = not neighbour["l2_hint_b"] and neighbour["tile_n"] == rule["tile_n"] and int(neighbour["split_k"]) < 8
    return share > 1.05 or unhinted


def select_gemm_schedule(operation: str, dtype: str, m: int, n: int, k: int,
                         batch: int = 1, activation: str = "none", share_depth: bool = True,
                         row_factors: bool = False) -> GemmScheduleSeed | None:
    """The schedule a launch of this shape uses, or ``None`` if the shape is unsupported.

    An exact table hit has empty ``adaptations``; a schedule transferred from a
    nearby measured shape names that shape; otherwise the library's shape-aware
    default, which takes the fused ``activation`` into account, is returned with
    ``source_shape`` ``None``.  Any of them is fitted to the shape where that is faster (``_fitted``), exact hits too, which
    its adaptations then say, unless ``share_depth`` is false (for a gate shaped like the output, whose kernels do not
    split, and for launches that leave SMs to others), by what their epilogue costs: ``activation`` and ``row_factors``.  It is a schedule of the general
    kernel: plain products that ``packed_serves`` run on the packed kernel, which takes none.
    """
    if min(batch, m, n, k) <= 0 or operation not in _OPERATIONS:
        return None
    if dtype not in _SHORT_DTYPES:
        return None
    # fp16 and bf16 run the same kernels at the same speed: a shape measured only in one serves the other
    other = "float16" if dtype == "bfloat16" else "bfloat16"
    table = {**SCHEDULES.get((operation, other), {}), **SCHEDULES.get((operation, dtype), {})}
    if not _shape_supported(m, n, k, batch):
        return None
    query = (batch, m, n, k)

    def distance(shape: tuple[int, int, int, int]) -> float:
        return sum(abs(math.log2(a) - math.log2(b)) for a, b in zip(shape, query, strict=True))

    def finished(seed: GemmScheduleSeed | None) -> GemmScheduleSeed | None:
        epilogue = "relu" if row_factors and activation == "none" else activation
        return _fitted(seed, operation, dtype, m, n, k, batch, epilogue) if share_depth else seed

    rule = None
    if query not in table and _streams_weights(operation, batch, m, n, k):
        rule = _fallback_schedule(operation, dtype, m, n, k, batch, activation)
    for shape in sorted(table, key=distance):
        if distance(shape) > _MAX_TRANSFER_DISTANCE:
            break
        for index in table[shape]:
            captured = {**_DEFAULTS, **CONFIGS[index]}
            if shape != query and _waves(captured, batch, m, n) > _waves(captured, shape[0], shape[1], shape[2]):
                continue  # it would no longer fit the number of waves it was measured at
            if shape != query:
                waste = _column_padding(captured, m, n)
                if waste >= 0.34 and waste > _column_padding(captured, shape[1], shape[2]) + 0.2:
                    continue  # its tiles would be a third or more padding here and were not where it was measured
            seed = _seed(captured, operation, dtype, m, n, k, batch, shape, exact=shape == query)
            if seed is not None:
                if rule is not None and _rule_streams_better(captured, rule.captured_config, activation, m, n, k):
                    return finished(rule)
                if shape not in SCHEDULES.get((operation, dtype), {}):
                    seed = GemmScheduleSeed(seed.captured_config, seed.builder_config,
                                            (*seed.adaptations, f"measured in {other}"), seed.source_shape,
                                            seed.source_percentage_of_torch)
                return finished(seed)
    return finished(_fallback_schedule(operation, dtype, m, n, k, batch, activation))


def _fallback_schedule(operation: str, dtype: str, m: int, n: int, k: int,
                       batch: int = 1, activation: str = "none") -> GemmScheduleSeed | None:
    """Unmeasured schedule from the library's heuristic (ayla_b200_default_config_act)."""
    if not _shape_supported(m, n, k, batch) or dtype not in _SHORT_DTYPES:
        return None
    if operation not in _OPERATIONS or (operation != "bmm" and batch != 1):
        return None
    captured = {**_DEFAULTS, **_lib.default_config(operation, dtype, batch, m, n, k, activation).to_dict()}
    return GemmScheduleSeed(
        captured,
        _builder_config(captured),
        ("unmeasured shape-aware default schedule",),
        None,
        None,
    )


def packed_serves(operation: str, batch: int, m: int, n: int, k: int, device: torch.device,
                  activation: str = "none", gated: bool | str = False) -> bool:
    """Whether the ops run a product of these extents on the packed kernel (few columns, a shallow depth, rows
    enough to fill the GPU) instead of the general one with ``select_gemm_schedule``'s schedule."""
    if activation != "none" or gated:
        return False
    index = device.index if device.index is not None else torch.cuda.current_device()
    with torch.cuda.device(index):
        _lib.init(index)  # the rule goes by the device's SM count
        return _lib.packed_preferred(operation, batch, m, n, k)


class _StreamWorkspace:
    """Memory that the k-split launches of one stream take in turn: each leaves its arrival counters at zero, wherever
    the next one's partial sums lie."""

    def __init__(self, size: int, device: torch.device):
        self.size = size
        self.tensor = torch.zeros(size, dtype=torch.uint8, device=device)


_WORKSPACES: weakref.WeakValueDictionary[tuple[int, int], _StreamWorkspace] = weakref.WeakValueDictionary()
_WORKSPACES_LOCK = threading.Lock()


def _stream_workspace(index: int, stream: int, size: int, device: torch.device) -> _StreamWorkspace:
    """The workspace of ``stream``, the current one, with at least ``size`` bytes.  All shapes share it (one each, for a
    thousand token counts through one layer, had taken ten gigabytes).  It grows by a factor of two or more; a launcher
    keeps what it was given, so a stream holds less than four times its largest need, and the memory goes with the last
    launcher that has it."""
    with _WORKSPACES_LOCK:
        workspace = _WORKSPACES.get((index, stream))
        if workspace is None or workspace.size < size:
            workspace = _StreamWorkspace(size if workspace is None else max(size, 2 * workspace.size), device)
            _WORKSPACES[index, stream] = workspace
        return workspace


class GemmLauncher:
    """One specialised ``(operation, dtype, shape, device)`` launch.

    Owns the status word of its shape and holds the split-K workspace of every stream it is used on
    (``_stream_workspace``; two launches that overlap on different streams would otherwise sum into
    each other's partial tiles): that of the stream which is current at specialisation time from then on,
    so that a launch there allocates nothing, another stream's from its first use.  A captured launch gets the workspace of its graph
    (``ayla_b200_capture_workspace``), since the graph may be replayed beside eager launches and
    other graphs; without memory for one it runs a schedule that needs none.  Where a k-split was
    measured for the shape itself, its first call on a stream must happen outside capture:
    inside it raises ``RuntimeError`` as a first call of a new shape does.

    The status word lives in pinned host memory (``_lib.StatusWord``): every call reads it
    before launching, without synchronising, and raises ``RuntimeError`` if an earlier
    launch of this shape ran into one of the kernel's bounded waits; the split-K arrival
    counters that launch may have left dirty are cleared first, so the call after the
    error is correct again.  ``check_status()`` does the same after a synchronise, and
    ``AYLA_B200_DEBUG=1`` calls it after every launch.

    It runs the schedule it is given.  With ``packed`` (for what ``packed_serves`` says) the launch goes to the
    packed kernel instead, and ``seed`` and ``config`` are used for an ``out`` on 16 bytes alone where the general
    kernel is then the faster one.
    """

    _captured_only_where_run = True  # a capture on a stream where this launcher has not run is refused
    _unsplit_config: _lib.Config | None = None
    _unsplit_tail: tuple | None = None
    _inside_tail: tuple | None = None  # for results that start inside a 32-byte sector

    def __init__(self, operation: str, dtype: str, batch: int, m: int, n: int, k: int,
                 seed: GemmScheduleSeed, device: torch.device, activation: str = "none",
                 gated: bool | str = False, packed: bool = False):
        assert seed.builder_config is not None
        self.operation, self.dtype, self.activation, self.gated = operation, dtype, activation, gated
        self.batch, self.m, self.n, self.k = batch, m, n, k
        self.seed = seed
        self.device = device
        self.config = _lib.Config.from_dict(seed.builder_config)
        index = device.index if device.index is not None else torch.cuda.current_device()
        with torch.cuda.device(index):
            _lib.init(index)
        self._packed = packed  # the library takes that kernel where it is given no schedule
        need = 0 if self._packed else _lib.workspace_bytes(self.config, operation, batch, m, n, k)
        self._ws_bytes = need
        self.workspace = None
        self._home_stream = None
        self._held: list[_StreamWorkspace] = []
        if need:
            with torch.cuda.device(index):
                self._home_stream = torch.cuda.current_stream().cuda_stream
                self._held.append(_stream_workspace(index, self._home_stream, need, device))
            self.workspace = self._held[0].tensor
        self.status = _lib.StatusWord()
        self._ws_ptr = self.workspace.data_ptr() if self.workspace is not None else 0
        self._status_ptr = self.status.ptr
        # stream handle -> (workspace tensor, argument tail), other than the stream current now
        self._per_stream: dict[int, tuple[torch.Tensor, tuple]] = {}
        self._debug = bool(os.environ.get("AYLA_B200_DEBUG"))
        # Everything that does not change from call to call, converted for the C call once.
        import ctypes

        lib = _lib.load()
        self._entry = lib.ayla_b200_gemm_act_rowmul if gated == "row" else lib.ayla_b200_gemm_act_mul
        self._head = (_lib.OP_CODES[operation], _lib.DTYPE_CODES[dtype], _lib.ACT_CODES[activation])
        self._tail = (batch, m, n, k, None if self._packed else ctypes.byref(self.config), self._ws_ptr or None,
                      self._ws_bytes, self._status_ptr)
        if self._packed and not _lib.workspace_bytes(self.config, operation, batch, m, n, k):
            with torch.cuda.device(index):
                if not _lib.packed_preferred(operation, batch, m, n, k, 16):
                    self._inside_tail = (batch, m, n, k, ctypes.byref(self.config), None, 0, self._status_ptr)
        self._has_bias = operation == "addmm"
        self._device_index = index
        self._captured_only_where_run = not seed.adaptations
        if need and seed.adaptations:
            # What a capture without memory for a workspace records, unless this schedule was measured for the shape: the
            # one before its depth was split, the library's, or this one with its depth whole.
            whole = {**seed.builder_config, "split_k": 1, "split_tail": 0, "cluster_split": 0}
            library = _lib.default_config(operation, dtype, batch, m, n, k, activation).to_dict()
            for candidate in (seed.unsplit_config, library, whole):
                if candidate is None or not _legal(candidate, operation, dtype, m, n, k, batch):
                    continue
                unsplit = _lib.Config.from_dict(candidate)
                if not _lib.workspace_bytes(unsplit, operation, batch, m, n, k):
                    self._unsplit_config = unsplit
                    self._unsplit_tail = (batch, m, n, k, ctypes.byref(unsplit), None, 0, self._status_ptr)
                    break

    def __call__(self, *tensors: torch.Tensor) -> None:
        bias_ptr = mul_ptr = None
        if self._has_bias:
            bias_ptr = tensors[0].data_ptr()
            tensors = tensors[1:]
        if self.gated:
            a, bt, mul, out = tensors
            mul_ptr = mul.data_ptr()
        else:
            a, bt, out = tensors
        if self.status.peek():
            self._report_timeout()
        stream = torch.cuda.current_stream(self._device_index).cuda_stream
        tail = self._tail
        if self._ws_bytes:
            tail = self._tail_for_stream(stream)
        elif self._inside_tail is not None and out.data_ptr() & 31:
            tail = self._inside_tail
        # The library launches on the current device (the reference's launcher guards the device
        # the same way, ayla/ptx_runtime.py:268-275).
        if torch.cuda.current_device() != self._device_index:
            with torch.cuda.device(self._device_index):
                code = self._entry(*self._head, bias_ptr, a.data_ptr(), bt.data_ptr(), mul_ptr, out.data_ptr(),
                                   *tail, stream)
        else:
            code = self._entry(*self._head, bias_ptr, a.data_ptr(), bt.data_ptr(), mul_ptr, out.data_ptr(),
                               *tail, stream)
        if code:
            _lib.check(code)
        if self._debug:
            self.check_status()

    def native_call(self) -> dict[str, object] | None:
        """What the compiled dispatcher needs to repeat this launch on its home stream; ``None`` where every launch
        is to be checked (``AYLA_B200_DEBUG``)."""
        if self._debug:
            return None
        import ctypes

        op, dtype, activation = self._head
        return {
            "entry": ctypes.cast(self._entry, ctypes.c_void_p).value, "swiglu": False,
            "op": op, "dtype": dtype, "activation": activation,
            "has_bias": self._has_bias, "gated": bool(self.gated),
            "batch": self.batch, "m": self.m, "n": self.n, "k": self.k,
            "config": 0 if self._packed else ctypes.addressof(self.config),
            "inside_config": 0 if self._inside_tail is None else ctypes.addressof(self.config),
            "workspace": self._ws_ptr, "workspace_bytes": self._ws_bytes,
            "status": self._status_ptr, "home_stream": self._home_stream or 0, "device": self._device_index,
        }

    def _tail_for_stream(self, stream: int) -> tuple:
        """The call arguments with the workspace that belongs to ``stream`` (allocated on first use), or to the graph
        under capture there."""
        entry = self._per_stream.get(stream)
        with torch.cuda.device(self._device_index):
            capturing = torch.cuda.is_current_stream_capturing()
            if capturing:
                if self._captured_only_where_run and entry is None and stream != self._home_stream:
                    raise RuntimeError(
                        f"jit_{self.operation}: the first launch of this k-split shape on a stream cannot happen during "
                        "CUDA graph capture; run it once on that stream before capturing")
                return self._captured_tail(stream)
        if stream == self._home_stream:
            return self._tail
        if entry is None:
            with torch.cuda.device(self._device_index):
                space = _stream_workspace(self._device_index, stream, self._ws_bytes, self.device)
            self.__dict__.setdefault("_held", []).append(space)
            entry = (space.tensor, self._tail_with(space.tensor.data_ptr()))
            self._per_stream[stream] = entry
        return entry[1]

    def _tail_with(self, workspace: int) -> tuple:
        batch, m, n, k, cfg, _, _, status = self._tail
        return (batch, m, n, k, cfg, workspace, self._ws_bytes, status)

    def _captured_tail(self, stream: int) -> tuple:
        workspace = _lib.capture_workspace(stream, self._ws_bytes)
        if workspace is not None:
            return self._tail_with(workspace)
        if self._unsplit_tail is None:
            raise RuntimeError(f"jit_{self.operation}: no memory for the workspace of a captured launch")
        return self._unsplit_tail

    def _report_timeout(self) -> None:
        code = self.status.peek()
        with torch.cuda.device(self._device_index):
            torch.cuda.current_stream().synchronize()  # nothing of the failed launch is still running
            # Arrival counters a timed-out k-split leaves behind: behind the launches of the stream that uses them.
            here = torch.cuda.current_stream().cuda_stream
            spaces = [(stream, workspace) for stream, (workspace, _) in self._per_stream.items()]
            for stream, workspace in [(self._home_stream, self.workspace), *spaces]:
                if workspace is None:
                    continue
                if stream is None or stream == here:
                    workspace.zero_()
                else:
                    with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
                        workspace.zero_()
        self.status.clear()
        raise RuntimeError(
            f"jit_{self.operation}: device wait timed out (code {code & 0xFF}, CTA {code >> 8})"
        )

    def check_status(self) -> None:
        """Synchronise and raise if one of the kernel's bounded waits gave up."""
        torch.cuda.synchronize(self._device_index)
        if self.status.peek():
            self._report_timeout()


def _op_name(operation: str, dtype: str, activation: str = "none", gated: bool | str = False) -> str:
    middle = ("" if activation == "none" else f"_{activation}") + {False: "", True: "_mul", "row": "_rowmul"}[gated]
    return f"jit_{operation}{middle}_{_SHORT_DTYPES[dtype]}"


def _template(operation: str, dtype: str, activation: str = "none", gated: bool | str = False) -> OpTemplate:
    torch_dtype = _TORCH_DTYPES[dtype]
    rank = 3 if operation == "bmm" else 2
    tensor = TensorSpec(torch_dtype, (None,) * rank)
    signature = (tensor,) * (4 if gated else 3)  # a, bt, [mul,] out
    if operation == "addmm":
        signature = (TensorSpec(torch_dtype, (None,)), *signature)
    return OpTemplate(_op_name(operation, dtype, activation, gated), signature)


def gemm_jit_compiler(operation: str, dtype: str, activation: str = "none",
                      gated: bool | str = False) -> ShapeSpecializingJITCompiler:
    """Per-shape dispatcher for one op: validates operands, picks the schedule once
    per ``(device, shapes)`` and launches (ayla/gemm_jit.py:339-393).  ``activation``
    (one of ``ACTIVATIONS``) is fused into the epilogue; with ``gated`` the op takes one more
    operand ``mul`` (shaped like ``out``, before it) and writes ``activation(...) * mul``; with
    ``gated="row"`` that operand is one factor per output row, shaped ``(..., m, 1)``."""
    if gated not in (False, True, "row"):
        raise ValueError(f"unsupported gate {gated!r}")
    if operation not in _OPERATIONS:
        raise ValueError(f"unsupported GEMM operation {operation}")
    if dtype not in _SHORT_DTYPES:
        raise ValueError(f"unsupported GEMM dtype {dtype}")
    if activation not in ACTIVATIONS:
        raise ValueError(f"unsupported GEMM activation {activation}")
    template = _template(operation, dtype, activation, gated)

    def compile_specialization(bound: OpTemplate, device: torch.device) -> GemmLauncher:
        sizes = [spec.sizes for spec in bound.signature]
        mul = sizes.pop(-2) if gated else None
        *bias, a, bt, out = sizes
        *batch, m, k = a
        n = bt[-2]
        lead = tuple(batch)
        if tuple(bt) != (*lead, n, k):
            raise ValueError(
                f"{bound.name}: bt must be {(*lead, n, k)} for a of shape {tuple(a)} "
                f"(out = a @ bt.T), got {tuple(bt)}"
            )
        if tuple(out) != (*lead, m, n):
            raise ValueError(f"{bound.name}: out must be {(*lead, m, n)}, got {tuple(out)}")
        if bias and tuple(bias[0]) != (n,):
            raise ValueError(f"{bound.name}: bias must be ({n},), got {tuple(bias[0])}")
        if gated == "row" and tuple(mul) != (*lead, m, 1):
            raise ValueError(f"{bound.name}: the row factors must be {(*lead, m, 1)}, got {tuple(mul)}")
        if gated is True and tuple(mul) != tuple(out):
            raise ValueError(f"{bound.name}: mul must have the shape of out {tuple(out)}, got {tuple(mul)}")
        count = batch[0] if batch else 1
        schedule = select_gemm_schedule(operation, dtype, m, n, k, count, activation, gated is not True, gated == "row")
        if schedule is None:
            raise ValueError(f"{bound.name}: no schedule for {operation} {lead}x{m}x{n}x{k}")
        return GemmLauncher(operation, dtype, count, m, n, k, schedule, device, activation, gated,
                            packed_serves(operation, count, m, n, k, device, activation, gated))

    return ShapeSpecializingJITCompiler(template, compile_specialization)


_COMPILERS: dict[tuple[str, str, str], ShapeSpecializingJITCompiler] = {}


def gemm_op(operation: str, dtype: str, namespace: str = DEFAULT_NAMESPACE) -> torch._ops.OpOverload:
    """Torch op ``(bias?, a, bt, out) -> ()`` writing ``out = [bias +] a @ bt^T``.

    Cached: the same overload object is returned for the same arguments."""
    return _gemm_op(operation, dtype, namespace)


@cache
def _gemm_op(operation: str, dtype: str, namespace: str) -> torch._ops.OpOverload:
    from .torch_custom_call import make_torch_custom_call

    compiler = gemm_jit_compiler(operation, dtype)
    _COMPILERS[(operation, dtype, namespace)] = compiler
    inputs = 3 if operation == "addmm" else 2
    return make_torch_custom_call(compiler, [OperandKind.R] * inputs + [OperandKind.RW],
                                  namespace=namespace)


def gemm_op_compiler(operation: str, dtype: str,
                     namespace: str = DEFAULT_NAMESPACE) -> ShapeSpecializingJITCompiler:
    """The dispatcher behind ``gemm_op(operation, dtype, namespace)`` (for its cache
    size and the launchers' status words)."""
    gemm_op(operation, dtype, namespace)
    return _COMPILERS[(operation, dtype, namespace)]


def gemm_act_mul_op(operation: str, activation: str, dtype: str,
                    namespace: str = DEFAULT_NAMESPACE) -> torch._ops.OpOverload:
    """Torch op ``(bias?, a, bt, mul, out) -> ()`` writing ``out = activation([bias +] a @ bt^T) * mul``
    with ``mul`` shaped like ``out``, named ``jit_{operation}[_{activation}]_mul_{f16|bf16}``: a gated
    projection (``sigmoid(x @ Wg^T) * v``) in one kernel, the product taken in fp32 before the single
    rounding.  The reference recognises this producer region in compiled graphs
    (ayla/torch_compile.py:288-504) but has no kernel for it."""
    return _gemm_act_mul_op(operation, activation, dtype, namespace)


@cache
def _gemm_act_mul_op(operation: str, activation: str, dtype: str, namespace: str) -> torch._ops.OpOverload:
    from .torch_custom_call import make_torch_custom_call

    compiler = gemm_jit_compiler(operation, dtype, activation, gated=True)
    _COMPILERS[(f"{operation}_{activation}_mul", dtype, namespace)] = compiler
    inputs = 4 if operation == "addmm" else 3
    return make_torch_custom_call(compiler, [OperandKind.R] * inputs + [OperandKind.RW],
                                  namespace=namespace)


def gemm_act_rowmul_op(operation: str, activation: str, dtype: str,
                       namespace: str = DEFAULT_NAMESPACE) -> torch._ops.OpOverload:
    """Torch op ``(bias?, a, bt, row_mul, out) -> ()`` writing
    ``out = activation([bias +] a @ bt^T) * row_mul`` with ``row_mul`` shaped ``(..., m, 1)`` (one factor
    per output row, as a ``keepdim`` reduction over the rows of ``a`` leaves it), named
    ``jit_{operation}[_{activation}]_rowmul_{f16|bf16}``.  With no activation and no bias it is a GEMM
    whose left operand carries a per-row scale: an RMSNorm followed by a projection becomes one row
    reduction and this op once the norm's weight vector is folded into ``bt``, because
    ``(x * r[:, None] * g) @ W.T == r[:, None] * (x @ (W * g).T)``.  The reference lists epilogue
    fusion as an aim (README.md:6-7) and has no kernel of this form."""
    return _gemm_act_rowmul_op(operation, activation, dtype, namespace)


@cache
def _gemm_act_rowmul_op(operation: str, activation: str, dtype: str, namespace: str) -> torch._ops.OpOverload:
    from .torch_custom_call import make_torch_custom_call

    compiler = gemm_jit_compiler(operation, dtype, activation, gated="row")
    _COMPILERS[(f"{operation}+{activation}+rowmul", dtype, namespace)] = compiler
    inputs = 4 if operation == "addmm" else 3
    return make_torch_custom_call(compiler, [OperandKind.R] * inputs + [OperandKind.RW], namespace=namespace)


def gemm_act_op(operation: str, activation: str, dtype: str,
                namespace: str = DEFAULT_NAMESPACE) -> torch._ops.OpOverload:
    """Torch op ``(bias?, a, bt, out) -> ()`` writing ``out = activation([bias +] a @ bt^T)``,
    named ``jit_{operation}_{activation}_{f16|bf16}``; the activation is evaluated on the fp32
    accumulator before the single rounding.  The reference has one such kernel, a fixed
    4096-cube matmul + sigmoid (ayla/gemm_collection/auto_matmul_4096_wgmma256_wg_sigmoid.py:22-142);
    this is the same fusion for every shape, operation and activation in ``ACTIVATIONS``.
    ``activation="none"`` returns ``gemm_op(operation, dtype)``."""
    if activation == "none":
        return gemm_op(operation, dtype, namespace)
    return _gemm_act_op(operation, activation, dtype, namespace)


@cache
def _gemm_act_op(operation: str, activation: str, dtype: str, namespace: str) -> torch._ops.OpOverload:
    from .torch_custom_call import make_torch_custom_call

    compiler = gemm_jit_compiler(operation, dtype, activation)
    _COMPILERS[(f"{operation}_{activation}", dtype, namespace)] = compiler
    inputs = 3 if operation == "addmm" else 2
    return make_torch_custom_call(compiler, [OperandKind.R] * inputs + [OperandKind.RW],
                                  namespace=namespace)
