"""The fixed-point lattice coordinates of the FP32 core's samplers (csrc/wg_fixed.h), compiled for the host."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src = d / "fixed.cpp"
    src.write_text('#include "wg_fixed.h"\nusing namespace wg;\n'
                   'extern "C" void at(uint64_t b, uint64_t s, uint32_t d, uint32_t *cell, float *frac) '
                   '{ const uint64_t v = fixed_at(b, s, d); *cell = fixed_cell(v); *frac = fixed_frac(v); }\n'
                   'extern "C" uint64_t fixed(double v) { return to_fixed(v); }\n')
    out = str(d / "fixed.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "low-witch-finder_b200", "csrc"), str(src), "-o", out], check=True)
    lib = C.CDLL(out)
    lib.at.argtypes = [C.c_uint64, C.c_uint64, C.c_uint32, C.POINTER(C.c_uint32), C.POINTER(C.c_float)]
    lib.fixed.argtypes, lib.fixed.restype = [C.c_double], C.c_uint64
    return lib


def test_fractions_have_all_bits_of_fp32(lib):
    """The cell is exact and the fraction the coordinate's, rounded to FP32: within 2^-25 (the conversion) and
    2^-32 (the bits below the word that is converted)."""
    rng = np.random.default_rng(3)
    cell, frac = C.c_uint32(), C.c_float()
    edge = [0, 1, (1 << 56) - 1, (1 << 64) - 1, 255 << 56]
    bases = edge + [int(v) for v in rng.integers(0, 1 << 64, 4000, dtype=np.uint64)]
    for n, b in enumerate(bases):
        step = int(4.0 * (337.0 / 331.0 if n & 1 else 1.0) * 2.0 ** -(n % 12) * 2.0 ** 56)
        d = int(rng.integers(0, 1 << 15))
        lib.at(b, step, d, C.byref(cell), C.byref(frac))
        v = (b + d * step) % (1 << 64)
        assert cell.value == v >> 56
        assert abs(frac.value - (v % (1 << 56)) / 2.0 ** 56) <= 2.0 ** -25 + 2.0 ** -32


def test_coordinates_are_taken_mod_256(lib):
    rng = np.random.default_rng(4)
    for v in [0.0, 256.0, -256.0, -1e-30, 255.99999999999997] + list(rng.uniform(-1e6, 1e6, 2000)):
        got = lib.fixed(v) / 2.0 ** 56
        want = v % 256.0
        assert min(abs(got - want), 256.0 - abs(got - want)) <= 2.0 ** -44   # an ulp below 256
