"""The C-ABI library on a machine without a GPU: it loads, exports everything the
header declares, and its host-side logic (validation, schedule choice, workspace
sizing) behaves.  No kernel is launched here."""

import ctypes
import re
from pathlib import Path

import pytest

from ayla_b200 import _lib

HEADER = Path(__file__).resolve().parent.parent / "include" / "ayla_b200.h"


def declared_symbols() -> list[str]:
    return re.findall(r"AYLA_B200_API[^;(]*?\b(ayla_b200_\w+)\s*\(", HEADER.read_text())


def test_library_exports_every_declared_symbol():
    names = declared_symbols()
    assert len(names) >= 12
    lib = _lib.load()
    for name in names:
        assert hasattr(lib, name), name
    assert set(names) == set(_lib.EXPORTS)


def test_version_and_variants():
    assert "sm_100a" in _lib.version()
    variants = _lib.kernel_variants()
    keys = {(v["tile_n"], v["cta_group"], v["epilogue"], v["transposed_out"]) for v in variants}
    assert len(keys) == len(variants)
    for tile_n in (64, 128, 192, 256):
        for cta_group in (1, 2):
            for epilogue in (0, 1):
                assert (tile_n, cta_group, epilogue, 0) in keys
    for tile_n in (16, 32, 64, 128):
        assert (tile_n, 1, 0, 1) in keys and (tile_n, 1, 1, 1) in keys
    assert (256, 1, 2, 0) in keys and (256, 2, 2, 0) in keys
    for v in variants:
        assert v["smem_bytes"] <= 232448 and v["stages"] >= 3


def test_struct_layout_matches_header():
    fields = re.search(r"typedef struct ayla_b200_config \{(.*?)\} ayla_b200_config;", HEADER.read_text(), re.S)
    names = re.findall(r"int32_t\s+(\w+);", fields.group(1))
    assert tuple(names) == _lib.Config.FIELDS
    assert ctypes.sizeof(_lib.Config) == 4 * len(names)


@pytest.mark.parametrize(
    "args, code",
    [
        ((0, 1, 1, 64, 64, 64), 0),
        ((7, 1, 1, 64, 64, 64), _lib.E_INVALID),      # unknown op
        ((0, 5, 1, 64, 64, 64), _lib.E_INVALID),      # unknown dtype
        ((0, 1, 1, 0, 64, 64), _lib.E_INVALID),       # non-positive extent
        ((0, 1, 2, 64, 64, 64), _lib.E_INVALID),      # batch on mm
        ((2, 1, 2, 64, 64, 64), 0),                   # batch on bmm
        ((0, 1, 1, 64, 65, 64), _lib.E_UNSUPPORTED),  # n % 8
        ((0, 1, 1, 64, 64, 36), _lib.E_UNSUPPORTED),  # k % 8
        ((0, 1, 1, 64, 64, 40), 0),                   # k % 8 == 0 is enough (TMA zero-fills the tail)
    ],
)
def test_default_config_validates_shapes(args, code):
    cfg = _lib.Config()
    assert _lib.load().ayla_b200_default_config(*args, ctypes.byref(cfg)) == code
    if code:
        assert _lib.last_error()


def test_default_schedules_for_the_benchmark_shapes():
    big = _lib.default_config("mm", "bfloat16", 1, 4096, 4096, 4096)
    # 256 paired tiles on 74 SM pairs = 3.46 waves: the 34 tiles of the last wave run at half width
    assert (big.tile_n, big.cta_group, big.swap_ab, big.split_k, big.split_tail) == (256, 2, 0, 1, 2)
    assert _lib.workspace_bytes(big, "mm", 1, 4096, 4096, 4096) == 0
    ksplit = _lib.Config.from_dict(dict(tile_n=256, cta_group=2, split_k=2, split_tail=1))
    assert _lib.workspace_bytes(ksplit, "mm", 1, 4096, 4096, 4096) == 65536 + 34 * 2 * 2 * 128 * 256 * 4
    whole = _lib.default_config("mm", "bfloat16", 1, 8192, 8192, 8192)  # 13.8 waves: no split
    assert (whole.split_k, whole.split_tail) == (1, 0)
    decode = _lib.default_config("mm", "bfloat16", 1, 1, 4096, 4096)
    assert decode.swap_ab == 1 and decode.tile_n == 16 and decode.split_k >= 2
    # 112 tiles of bt leave no room to split K: a few dozen rows of `a` go through the plain 128-wide
    # tile (its `a` box trimmed), a handful stay on the swapped form
    m64 = _lib.default_config("mm", "bfloat16", 1, 64, 14336, 4096)
    assert (m64.swap_ab, m64.tile_n, m64.split_k) == (0, 128, 1)
    m8 = _lib.default_config("mm", "bfloat16", 1, 8, 14336, 4096)
    assert (m8.swap_ab, m8.tile_n) == (1, 16)
    m64_k = _lib.default_config("mm", "bfloat16", 1, 64, 4096, 4096)  # 32 tiles: K split over a cluster of 4
    assert (m64_k.swap_ab, m64_k.tile_n, m64_k.split_k, m64_k.cluster_split) == (1, 64, 4, 1)
    m256 = _lib.default_config("mm", "bfloat16", 1, 256, 4096, 4096)  # pairs, K split over two pairs
    assert (m256.tile_n, m256.cta_group, m256.split_k, m256.cluster_split) == (128, 2, 2, 1)
    deep = _lib.default_config("addmm", "bfloat16", 1, 256, 1024, 16384)
    assert deep.swap_ab == 0 and deep.split_k > 1
    for cfg, shape in ((big, (1, 4096, 4096, 4096)), (decode, (1, 1, 4096, 4096)),
                       (deep, (1, 256, 1024, 16384))):
        assert _lib.config_valid(cfg, "mm", "bfloat16", *shape)


@pytest.mark.parametrize("activation, m, n, k, swapped", [
    ("sigmoid", 38, 11512, 2952, False), ("silu", 40, 10752, 8704, False), ("sigmoid", 20, 11136, 5312, True),
    ("none", 38, 13376, 3136, True), ("none", 44, 12216, 4760, True), ("sigmoid", 8, 14336, 4096, True)])
def test_long_streams_behind_an_activation_are_row_major_from_33_rows_on(activation, m, n, k, swapped):
    cfg = _lib.default_config("mm", "bfloat16", 1, m, n, k, activation)
    assert cfg.swap_ab == int(swapped) and cfg.split_k == 1
    assert swapped or (cfg.tile_n, cfg.tile_rows, cfg.split_tail) == (128, 0, 2)


def test_config_validation():
    ok = _lib.Config.from_dict(dict(tile_n=128, cta_group=2))
    assert _lib.config_valid(ok, "mm", "bfloat16", 1, 512, 512, 512)
    for bad in (dict(tile_n=48), dict(tile_n=16), dict(cta_group=3), dict(split_k=0), dict(group_m=0),
                dict(tile_n=256, swap_ab=1), dict(tile_n=64, swap_ab=1, cta_group=2), dict(l2_hint_a=3)):
        cfg = _lib.Config.from_dict({**dict(tile_n=128, cta_group=1), **bad})
        assert not _lib.config_valid(cfg, "mm", "bfloat16", 1, 512, 512, 512), bad
    assert _lib.config_valid(_lib.Config.from_dict(dict(tile_n=16, swap_ab=1)), "mm", "float16", 1, 8, 512, 512)
    # cluster split-K: cluster of at most 8 CTAs, tile columns divisible among the k-splits
    csk = dict(tile_n=64, cta_group=1, split_k=4, cluster_split=1)
    assert _lib.config_valid(_lib.Config.from_dict(csk), "mm", "bfloat16", 1, 64, 512, 4096)
    assert _lib.workspace_bytes(_lib.Config.from_dict(csk), "mm", 1, 64, 512, 4096) == 0
    assert _lib.config_valid(_lib.Config.from_dict({**csk, "cta_group": 2}), "mm", "bfloat16", 1, 64, 512, 4096)
    for bad in (dict(split_k=3), dict(cta_group=2, split_k=8), dict(tile_n=16, swap_ab=1, split_k=8), dict(stream_k=1)):
        assert not _lib.config_valid(_lib.Config.from_dict({**csk, **bad}), "mm", "bfloat16", 1, 64, 512, 4096), bad
    assert not _lib.config_valid(_lib.Config.from_dict(csk), "mm", "bfloat16", 1, 64, 512, 128)  # 2 k-blocks, 4 CTAs
    # trimmed tiles exist only in the swapped form
    trimmed = dict(tile_n=16, swap_ab=1, tile_rows=97)
    assert _lib.config_valid(_lib.Config.from_dict(trimmed), "mm", "bfloat16", 1, 8, 14336, 4096)
    for bad in (dict(tile_rows=4), dict(tile_rows=129), dict(swap_ab=0, tile_n=64)):
        assert not _lib.config_valid(_lib.Config.from_dict({**trimmed, **bad}), "mm", "bfloat16", 1, 8, 14336, 4096), bad


def test_workspace_sizing():
    none = _lib.Config.from_dict(dict(tile_n=256, cta_group=1, split_k=1))
    assert _lib.workspace_bytes(none, "mm", 1, 256, 1024, 16384) == 0
    cfg = _lib.Config.from_dict(dict(tile_n=64, cta_group=1, split_k=4))
    # 2 row tiles x 16 column tiles, 4 splits, 128 x 64 fp32 slabs, + the fixed 64 KiB counter header
    counters = _lib.workspace_counter_bytes(cfg, "mm", 1, 256, 1024, 16384)
    assert counters == 65536
    assert _lib.workspace_bytes(cfg, "mm", 1, 256, 1024, 16384) == counters + 32 * 4 * 128 * 64 * 4
    # more splits than 64-wide k blocks are clamped
    deep = _lib.Config.from_dict(dict(tile_n=64, cta_group=1, split_k=64))
    assert _lib.workspace_bytes(deep, "mm", 1, 128, 64, 128) == 65536 + 1 * 2 * 128 * 64 * 4
    huge = _lib.Config.from_dict(dict(tile_n=64, cta_group=1, split_k=2))
    assert not _lib.config_valid(huge, "mm", "bfloat16", 1, 128 * 200, 64 * 100, 256)  # 20000 tiles
    pair = _lib.Config.from_dict(dict(tile_n=128, cta_group=2, split_k=2))
    assert _lib.workspace_bytes(pair, "mm", 1, 256, 128, 1024) == 65536 + 2 * 2 * 128 * 128 * 4


def test_gemm_rejects_bad_arguments_before_touching_the_device():
    lib = _lib.load()
    one = ctypes.c_void_p(16)
    assert lib.ayla_b200_gemm(0, 1, None, None, one, one, 1, 64, 64, 64, None, None, 0, None, None) == _lib.E_INVALID
    assert "non-null" in _lib.last_error()
    assert lib.ayla_b200_gemm(1, 1, None, one, one, one, 1, 64, 64, 64, None, None, 0, None, None) == _lib.E_INVALID
    assert "bias" in _lib.last_error()
    odd = ctypes.c_void_p(24)
    assert lib.ayla_b200_gemm(0, 1, None, odd, one, one, 1, 64, 64, 64, None, None, 0, None, None) == _lib.E_UNSUPPORTED
    assert "16-byte" in _lib.last_error()
    assert lib.ayla_b200_swiglu(1, one, one, None, one, 64, 64, 64, None, None, None) == _lib.E_INVALID
    with pytest.raises(ValueError, match="multiple of 8"):
        _lib.check(lib.ayla_b200_gemm(0, 1, None, one, one, one, 1, 64, 65, 64, None, None, 0, None, None))


@pytest.mark.parametrize("op, batch, m, n, k, tile_n, plain, gelu", [
    # Tiles of a shallow product: the width that the cost model picks for single CTAs, paired where that measured
    # faster -- wide tiles of two waves and more, rows that start inside a sector; with padding only without a GELU ...
    ("mm", 1, 12095, 5824, 256, 256, 2, 2), ("addmm", 1, 10351, 3728, 224, 256, 2, 2), ("mm", 1, 8216, 4976, 104, 256, 2, 2),
    ("mm", 1, 11696, 520, 88, 128, 2, 2), ("bmm", 26, 830, 1264, 256, 256, 2, 1),
    # ... not 128-wide tiles of two k-blocks, a single wave, or rows that pairs would pad ...
    ("addmm", 1, 10600, 520, 64, 128, 1, 1), ("mm", 1, 1667, 3912, 96, 128, 1, 1), ("bmm", 28, 1873, 1576, 128, 256, 1, 1),
    ("bmm", 53, 310, 528, 128, 128, 1, 1), ("mm", 1, 3755, 816, 192, 128, 1, 1),
    # ... and never another width than single CTAs would take (22.5 us as 256 wide, 26.2 as 128-wide pairs; 6.5 and 7.9).
    ("addmm", 1, 12751, 3104, 64, 256, 2, 2), ("addmm", 1, 824, 4232, 88, 128, 2, 1),
])
def test_shallow_products_are_paired_where_it_measured_faster(op, batch, m, n, k, tile_n, plain, gelu):
    for activation, pairing in (("none", plain), ("gelu", gelu)):
        cfg = _lib.default_config(op, "bfloat16", batch, m, n, k, activation)
        assert (cfg.tile_n, cfg.cta_group) == (tile_n, pairing), (activation, cfg.to_dict())
        assert _lib.config_valid(cfg, op, "bfloat16", batch, m, n, k)


@pytest.mark.parametrize("m, n, k, tile_n, split", [
    (8, 1024, 4096, 16, 4), (8, 4096, 4096, 16, 2), (128, 4096, 4096, 128, 2), (512, 1024, 4096, 128, 2),
    # Unshared 128-wide accumulators: deep products only.
    (1024, 1024, 4096, 128, 1), (337, 2672, 4288, 128, 1), (68, 5232, 11720, 128, 1),
    (374, 2944, 3200, 128, 1), (150, 3304, 1664, 128, 1),
    (740, 1504, 896, 0, 0), (595, 1024, 2112, 0, 0), (381, 3136, 3208, 0, 0), (142, 3632, 656, 0, 0),
    (64, 14336, 4096, 0, 0), (8192, 14336, 4096, 0, 0),
])
def test_swiglu_of_few_rows_is_swapped_where_it_measured_faster(m, n, k, tile_n, split):
    cfg = _lib.swiglu_default_config("bfloat16", m, n, k)
    if tile_n == 0:
        assert (cfg.swap_ab, cfg.tile_n, cfg.split_k, cfg.cta_group) == (0, 256, 1, 2 if m >= 256 else 1)
    else:
        assert (cfg.swap_ab, cfg.tile_n, cfg.split_k, cfg.cluster_split) == (1, tile_n, split, int(split > 1))


# (m, n, k), tile width, the schedule's last wave -> width, splits and last wave that are fitted
@pytest.mark.parametrize("shape, tile_n, tail, expected", [
    ((4156, 1088, 3712), 256, 0, (256, 6, 1)),  # 1 + 11/74 waves of 58 k-blocks
    ((2229, 4864, 1792), 256, 0, (256, 1, 2)),  # 2 + 23/74 of 28: halves
    ((1128, 7488, 7928), 256, 0, (256, 11, 1)),  # rows inside a sector
    ((2920, 2568, 3832), 256, 2, (256, 1, 0)),  # 1 + 58/74: two halves of a tile do not fit
    ((9874, 640, 832), 256, 2, (256, 1, 0)),
    ((1260, 4480, 768), 256, 2, (256, 1, 2)),
    ((7328, 640, 5168), 192, 0, (256, 5, 1)),  # a thinner last wave of wider tiles
    ((6690, 1408, 3200), 192, 0, (192, 1, 0)),
    ((4096, 4096, 4096), 256, 2, (256, 1, 2)),
])
def test_last_waves_are_fitted_by_their_length(shape, tile_n, tail, expected):
    m, n, k = shape
    cfg = _lib.Config.from_dict(dict(group_m=8, tile_n=tile_n, cta_group=2, split_k=1, split_tail=tail))
    out = _lib.fit_depth(cfg, "mm", "bfloat16", 1, m, n, k)
    assert _lib.config_valid(out, "mm", "bfloat16", 1, m, n, k)
    assert (out.tile_n, out.split_k, out.split_tail) == expected


# (m, n, k), the schedule measured elsewhere -> tiles that all run at once here
@pytest.mark.parametrize("shape, config, expected", [
    ((5539, 384, 4096), dict(tile_n=256, cta_group=2, split_tail=2), (128, 2, 1, 0, 0)),
    ((1240, 2176, 28672), dict(tile_n=256, cta_group=2), (192, 2, 1, 0, 0)),
    ((620, 7232, 1664), dict(tile_n=256, cta_group=2, split_tail=2), (256, 1, 1, 0, 0)),
    ((119, 5312, 832), dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1), (64, 1, 1, 0, 0)),
    # as they are: the shallowest, clusters whose rows start inside a sector, few rows, what the model finds no faster
    ((1759, 1344, 640), dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 1, 2, 0)),
    ((200, 3208, 2456), dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1), (128, 1, 2, 0, 1)),
    ((64, 3208, 2048), dict(tile_n=64, cta_group=1), (64, 1, 1, 0, 0)),
    ((1056, 2048, 28288), dict(tile_n=256, cta_group=1), (256, 1, 2, 0, 0)),
])
def test_schedules_from_other_shapes_are_fitted_to_one_wave(shape, config, expected):
    m, n, k = shape
    out = _lib.fit_depth(_lib.Config.from_dict(dict(group_m=8, **config)), "mm", "bfloat16", 1, m, n, k)
    assert _lib.config_valid(out, "mm", "bfloat16", 1, m, n, k)
    assert (out.tile_n, out.cta_group, out.split_k, out.split_tail, out.cluster_split) == expected


# (m, n, k), activation, a schedule -> the one that measured faster of it and whole tiles in one wave
@pytest.mark.parametrize("shape, activation, config, expected", [
    # 128-wide pairs in more than one wave: by the activation, the k-blocks and the tiles left over
    ((9457, 384, 1280), "none", dict(tile_n=128, cta_group=2, split_tail=2), (192, 2, 1, 0)),
    ((9457, 384, 1280), "relu", dict(tile_n=128, cta_group=2, split_tail=2), (192, 2, 1, 0)),
    ((9457, 384, 1280), "silu", dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 1, 2)),
    ((990, 2368, 768), "none", dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 1, 2)),
    ((990, 2368, 960), "none", dict(tile_n=128, cta_group=2, split_tail=2), (192, 2, 1, 0)),
    ((990, 2368, 1088), "relu", dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 1, 2)),
    ((1147, 1920, 1408), "gelu", dict(tile_n=128, cta_group=2, split_tail=2), (128, 1, 1, 0)),
    ((1072, 2240, 1856), "gelu", dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 1, 2)),
    ((1072, 2240, 2112), "gelu", dict(tile_n=128, cta_group=2, split_tail=2), (192, 2, 1, 0)),
    # ... many k-blocks, with a split last wave there
    ((2200, 1216, 35136), "none", dict(tile_n=128, cta_group=2, split_tail=2), (128, 2, 4, 1)),
    ((1304, 1808, 33888), "none", dict(tile_n=128, cta_group=2), (128, 2, 4, 1)),
    ((1752, 1912, 26640), "none", dict(tile_n=128, cta_group=2), (192, 2, 1, 0)),
    # single CTAs of the same width (whole lines, and others), and clusters
    ((1722, 2560, 768), "none", dict(tile_n=256, cta_group=1), (256, 1, 1, 0)),
    ((2188, 1992, 1040), "relu", dict(tile_n=256, cta_group=1), (256, 2, 1, 0)),
    ((1581, 1712, 760), "none", dict(tile_n=256, cta_group=1), (192, 2, 1, 0)),
    ((179, 768, 1296), "relu", dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1), (64, 1, 2, 0)),
    ((192, 1664, 1152), "none", dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1), (64, 2, 1, 0)),
    ((282, 5440, 3776), "none", dict(tile_n=256, cta_group=1, split_k=2, cluster_split=1), (256, 1, 2, 0)),
])
def test_one_wave_only_where_it_measured_faster(shape, activation, config, expected):
    m, n, k = shape
    out = _lib.fit_depth(_lib.Config.from_dict(dict(group_m=8, **config)), "addmm", "bfloat16", 1, m, n, k, activation)
    assert _lib.config_valid(out, "addmm", "bfloat16", 1, m, n, k)
    assert (out.tile_n, out.cta_group, out.split_k, out.split_tail) == expected


# (m, n, k), a schedule -> pairs on tiles of 128 rows
@pytest.mark.parametrize("shape, config, expected", [
    ((128, 4096, 4096), dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1), (128, 2, 2, 0, 1)),
    ((65, 8192, 2048), dict(tile_n=128, cta_group=1, split_k=2, cluster_split=1), (128, 2, 1, 0, 0)),
    ((128, 14336, 4096), dict(tile_n=128, cta_group=1, split_tail=2), (256, 2, 1, 0, 0)),
    ((74, 960, 3136), dict(tile_n=64, cta_group=1, split_k=5), (128, 2, 4, 0, 1)),
    ((64, 8832, 2816), dict(tile_n=64, cta_group=1, swap_ab=1, split_k=2, cluster_split=1), (128, 2, 1, 0, 0)),
    ((33, 1344, 8448), dict(tile_n=64, cta_group=1, swap_ab=1, split_k=4, cluster_split=1), (128, 2, 4, 0, 1)),
    # as they are: other numbers of rows, whole tiles of few rows, few k-blocks, clusters of eight on the fewest tiles, more
    # than one wave of pairs, the swapped form of more rows, a given grid
    ((32, 1408, 8448), dict(tile_n=64, cta_group=1, swap_ab=1, split_k=4, cluster_split=1), (64, 1, 4, 0, 1)),
    ((64, 5120, 3328), dict(tile_n=64, cta_group=1), (64, 1, 1, 0, 0)),
    ((64, 128, 9728), dict(tile_n=64, cta_group=1, swap_ab=1, split_k=8, cluster_split=1), (64, 1, 8, 0, 1)),
    ((129, 4096, 4096), dict(tile_n=128, cta_group=2, split_k=2), (128, 2, 2, 0, 0)),
    ((128, 4096, 704), dict(tile_n=64, cta_group=1), (64, 1, 1, 0, 0)),
    ((128, 256, 9728), dict(tile_n=64, cta_group=1, split_k=8, cluster_split=1), (64, 1, 8, 0, 1)),
    ((128, 19200, 1024), dict(tile_n=256, cta_group=1), (256, 1, 1, 0, 0)),
    ((128, 4096, 4096), dict(tile_n=128, cta_group=1, swap_ab=1, split_k=4, cluster_split=1), (128, 1, 4, 0, 1)),
    ((128, 4096, 4096), dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1, grid_ctas=140), (64, 1, 2, 0, 1)),
])
def test_few_rows_are_given_to_pairs(shape, config, expected):
    m, n, k = shape
    out = _lib.fit_depth(_lib.Config.from_dict(dict(group_m=8, **config)), "mm", "bfloat16", 1, m, n, k)
    assert _lib.config_valid(out, "mm", "bfloat16", 1, m, n, k)
    assert (out.tile_n, out.cta_group, out.split_k, out.split_tail, out.cluster_split) == expected
    if out.cta_group == 2 and m <= 128:
        assert out.swap_ab == 0 and out.tile_rows == 0
        assert _lib.workspace_bytes(out, "mm", 1, m, n, k) == 0


# (batch, m, n, k), a schedule that stays one of single CTAs
@pytest.mark.parametrize("batch, shape, config", [
    # rows inside a sector: split depths of narrow tiles, whole tiles of a batch, neither rows nor columns for a second CTA
    (1, (64, 104, 13320), dict(tile_n=64, cta_group=1, split_k=16)),
    (1, (64, 104, 10520), dict(tile_n=64, cta_group=1, split_k=8)),
    (17, (78, 944, 392), dict(tile_n=128, cta_group=1)),
    (11, (37, 64, 3576), dict(tile_n=64, cta_group=1, split_k=4, cluster_split=1)),
    # mostly padding, in place of 16-way splits or with nearly as many clusters as run at once
    (1, (65, 32, 15984), dict(tile_n=64, cta_group=1, split_k=16)),
    (33, (72, 72, 1512), dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1)),
    (24, (64, 64, 1024), dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1)),
])
def test_few_rows_stay_with_single_ctas_where_those_measured_faster(batch, shape, config):
    m, n, k = shape
    operation = "bmm" if batch > 1 else "mm"
    cfg = _lib.Config.from_dict(dict(group_m=8, l2_hint_a=2, l2_hint_b=1, **config))
    out = _lib.fit_depth(cfg, operation, "bfloat16", batch, m, n, k)
    assert _lib.config_valid(out, operation, "bfloat16", batch, m, n, k)
    assert out.cta_group == 1


# (batch, m, n, k), a schedule of single CTAs that measured slower than pairs beside the ones above
@pytest.mark.parametrize("batch, shape, config, expected", [
    (37, (61, 72, 2240), dict(tile_n=128, cta_group=1, split_k=4, cluster_split=1), (128, 1)),
    (17, (66, 256, 3136), dict(tile_n=128, cta_group=1, split_k=4), (128, 1)),
    (33, (89, 56, 1088), dict(tile_n=64, cta_group=1, split_k=2, cluster_split=1), (128, 1)),
    (1, (128, 192, 760), dict(tile_n=64, cta_group=1, split_k=4, cluster_split=1), (128, 2)),
    (1, (128, 544, 3464), dict(tile_n=64, cta_group=1, split_k=4, cluster_split=1), (128, 4)),
])
def test_few_rows_of_the_same_kinds_go_to_pairs_where_those_measured_faster(batch, shape, config, expected):
    m, n, k = shape
    operation = "bmm" if batch > 1 else "mm"
    out = _lib.fit_depth(_lib.Config.from_dict(dict(group_m=8, **config)), operation, "bfloat16", batch, m, n, k)
    assert _lib.config_valid(out, operation, "bfloat16", batch, m, n, k)
    assert out.cta_group == 2 and (out.tile_n, out.split_k) == expected


def test_whole_narrow_tiles_of_few_rows_are_not_given_a_split_depth():
    out = _lib.fit_depth(_lib.Config.from_dict(dict(group_m=8, tile_n=64, cta_group=1)), "mm", "float16", 1, 94, 3456, 1024)
    assert out.split_k == 1


def test_depth_is_shared_where_sms_would_idle():
    def shared(m, n, k, **config):
        cfg = _lib.Config.from_dict(dict(group_m=8, **config))
        out = _lib.share_depth(cfg, "mm", "bfloat16", 1, m, n, k)
        assert _lib.config_valid(out, "mm", "bfloat16", 1, m, n, k)
        return (out.tile_n, out.cta_group, out.split_k, out.split_tail, out.cluster_split), out.to_dict() == cfg.to_dict()

    pairs = dict(tile_n=256, cta_group=2, split_k=1)
    # a thin last wave: split where a tile is long, run at half width where it is not, left alone where it is full
    assert shared(2744, 2112, 29248, **pairs)[0] == (256, 2, 2, 1, 0)
    assert shared(4451, 2240, 7040, **pairs)[0] == (256, 2, 5, 1, 0)
    assert shared(1260, 4480, 768, **pairs)[0] == (256, 2, 1, 2, 0)
    assert shared(8192, 1024, 8192, **pairs)[1]
    assert shared(3266, 1600, 512, **pairs)[0] == (256, 2, 1, 2, 0)
    assert shared(4546, 1408, 256, **pairs)[1] and shared(2348, 1408, 448, tile_n=128, cta_group=2)[1]
    # rows that start inside a sector: behind one wave, two with little left, or instead of halves
    halves = dict(pairs, split_tail=2)
    assert shared(785, 5056, 8456, **pairs)[0] == (256, 2, 2, 1, 0)
    assert shared(4096, 2560, 8008, **pairs)[0] == (256, 2, 2, 1, 0)
    assert shared(4527, 3200, 10792, **halves)[0] == (256, 2, 2, 1, 0)
    for m, n, k in ((4846, 3968, 12696), (6658, 2304, 12136), (4619, 4992, 11400), (3790, 5568, 7608), (3296, 3136, 8488)):
        assert shared(m, n, k, **pairs)[1]
    # a deep product on a few SMs, and clusters that do not all run at once
    assert shared(536, 896, 59968, tile_n=128, cta_group=1, split_k=4, cluster_split=1)[0][1:] == (2, 6, 0, 0)
    assert shared(175, 2304, 8000, tile_n=128, cta_group=1, split_k=4, cluster_split=1)[0] == (128, 2, 4, 0, 0)
    # not for a little in the model where pairs pad, or where rows start inside a sector; no single CTAs for pairs there
    assert shared(296, 1088, 14016, tile_n=128, cta_group=1, split_k=4, cluster_split=1)[1]
    assert shared(332, 960, 2568, tile_n=64, cta_group=1, split_k=2, cluster_split=1)[1]
    assert shared(524, 3200, 13656, **pairs)[0][1] == 2
    # neither: shallow, few rows, swapped, or a grid of its own
    assert shared(256, 1024, 1024, tile_n=64, cta_group=2, split_k=1)[1]
    assert shared(128, 4096, 4096, tile_n=64, cta_group=1, split_k=2, cluster_split=1)[1]
    assert shared(8, 4096, 4096, tile_n=16, cta_group=1, split_k=4, cluster_split=1, swap_ab=1)[1]
    assert shared(4451, 2240, 7040, grid_ctas=140, **pairs)[1]
