"""GPU: the solver's lift over every valuation class of the offsets.

The lift settles v2(rho) bits a step and has its own instances for m = 0 and m > 0 and for either
axis as the odd one; tasks with a planted solution reach each of them (offsets whose 2-adic
valuations differ by 1 to 4 and more, both ways round, the smaller 0 to 3), in near and far regions.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFFSETS = [(1, 2), (2, 1), (3, 4), (4, 3), (5, 8), (8, 5), (7, 16), (16, 7), (9, 0), (0, 9), (2, 4), (4, 2), (6, 8),
           (8, 6), (10, 16), (16, 10), (2, 0), (0, 2), (4, 8), (8, 4), (4, 16), (16, 12), (8, 16), (16, 8), (8, 0), (0, 16)]


def planted_at(port, rng, ox, oz, reach):
    """(S, rx, rz, X): a structure seed whose hut lies at (ox, oz) in a region within reach, its carver state."""
    cx, cz = C.c_int(), C.c_int()
    while True:
        S = int(rng.integers(0, 1 << 48))
        rx, rz = (int(v) for v in rng.integers(-reach, reach + 1, 2))
        port.lib.wo_hut_in_region(S, rx, rz, 14357620, C.byref(cx), C.byref(cz))
        if (cx.value - 32 * rx, cz.value - 32 * rz) == (ox, oz):
            return S, rx, rz, port.mineshaft_start(S, cx.value, cz.value)[1]


@pytest.mark.parametrize("ox,oz", OFFSETS)
def test_planted_solutions_are_found(engine, port, ox, oz):
    rng = np.random.default_rng(1000 * ox + oz)
    for reach in (40, 58593):
        S, rx, rz, X = planted_at(port, rng, ox, oz, reach)
        hits = sorted(int(h["s48"]) for h in engine.deep_solve_tasks(X, [rx], [rz], [ox], [oz]))
        assert S in hits
        assert hits == port.solve_task(X, rx, rz, ox, oz)
