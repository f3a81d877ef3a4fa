"""How rects are cut into tiles (csrc/wg_tiling.h), compiled for the host."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SLOTS = 444   # 148 SMs, three CTAs each


class Tiling(C.Structure):
    _fields_ = [("tw", C.c_uint32), ("th", C.c_uint32), ("ntx", C.c_uint32), ("n_win", C.c_uint64)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiling")
    src = d / "tiling.cpp"
    src.write_text('#include "wg_tiling.h"\nusing namespace wg;\n'
                   'extern "C" Tiling wave(uint64_t w, uint64_t h, uint64_t n, uint64_t s) { return wave_tiles(w, h, n, s); }\n'
                   'extern "C" Tiling rect(uint64_t w, uint64_t h, uint64_t t, uint64_t m) { return tile_rect(w, h, t, m); }\n')
    out = str(d / "tiling.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wno-return-type-c-linkage", "-I",
                    os.path.join(ROOT, "low-witch-finder_b200", "csrc"), str(src), "-o", out], check=True)
    lib = C.CDLL(out)
    for f in (lib.wave, lib.rect):
        f.argtypes, f.restype = [C.c_uint64] * 4, Tiling
    return lib


def covers(t, w, h):
    """The tiles cover the rect, and none is empty."""
    rows = t.n_win // t.ntx
    return t.n_win == t.ntx * rows and (t.ntx - 1) * t.tw < w <= t.ntx * t.tw and (rows - 1) * t.th < h <= rows * t.th


RECTS = [(1, 1), (2, 1), (1, 31), (9, 9), (33, 32), (158, 158), (400, 400), (1023, 1), (1024, 1), (10000, 1), (20000, 4),
         (40000, 8), (40000, 20), (2046, 64), (2047, 65), (6000, 5999), (100000, 40), (117188, 117188), (1 << 24, 3)]


@pytest.mark.parametrize("w,h", RECTS)
@pytest.mark.parametrize("n", [1, 4, 100, 444, 1777, 100000])
def test_a_rect_and_its_transpose_get_the_same_tiles(lib, w, h, n):
    a, b = lib.wave(w, h, n, SLOTS), lib.wave(h, w, n, SLOTS)
    for t, x, z in ((a, w, h), (b, h, w)):
        assert covers(t, x, z)
        assert max(t.tw, t.th) <= 1023 and t.tw * t.th <= 65536
    assert abs(a.n_win - b.n_win) <= 0.02 * a.n_win + 1
    # room for a wave of tiles and regions for it: most of a wave's CTAs have one
    if n * w * h >= 64 * SLOTS and n <= SLOTS:
        assert n * a.n_win >= 0.9 * SLOTS or (a.tw, a.th) == (w, h)


@pytest.mark.parametrize("w,h", RECTS)
@pytest.mark.parametrize("target,side", [(1, 1023), (2048, 1023), (4096, 4096), (16384, 1023), (65536, 1023)])
def test_rect_tiles_cover_the_rect(lib, w, h, target, side):
    t = lib.rect(w, h, target, side)
    assert covers(t, w, h)
    assert max(t.tw, t.th) <= side and t.tw * t.th <= target
