"""The largest value a Perlin sample can take: the unit kernel's first entrance test skips noises on
the strength of |sample| <= 1.0625 (kPerlinMax, wg_unit.cuh)."""
from __future__ import annotations

import os
import re

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_perlin_samples_stay_below_the_bound():
    text = open(os.path.join(ROOT, "low-witch-finder_b200", "csrc", "wg_unit.cuh")).read()
    bound = float(re.search(r"kPerlinMax = ([0-9.]+);", text).group(1))
    # A gradient has two components of +-1, so a corner's product is at most the sum of the two
    # largest offsets from it; the sample blends the corners with weights that sum to 1.  The largest
    # blend on a grid of cell centres of side h (one octant, by symmetry), plus what it can grow by to a
    # corner of a grid cell: per axis a slope of at most 1.875 (the fade's) times the difference of two
    # averages in [0, 2], plus 1 (the products' own slope).
    n = 200
    h = 0.5 / n
    c = (np.arange(n) + 0.5) * h
    fade = lambda d: d * d * d * (d * (d * 6 - 15) + 10)
    y, z = np.meshgrid(c, c, indexing="ij")
    top = 0.0
    for x in c:
        v = np.zeros_like(y)
        for i in (0, 1):
            for j in (0, 1):
                for k in (0, 1):
                    d = np.stack([np.full_like(y, abs(x - i)), np.abs(y - j), np.abs(z - k)])
                    w = (fade(x) if i else 1 - fade(x)) * (fade(y) if j else 1 - fade(y)) * (fade(z) if k else 1 - fade(z))
                    v += w * (d.sum(0) - d.min(0))
        top = max(top, float(v.max()))
    slope = 2 * 1.875 + 1
    assert top + 3 * slope * h / 2 <= bound
