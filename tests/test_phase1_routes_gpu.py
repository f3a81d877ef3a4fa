"""GPU: phase 1's list kernels against the unit kernel and against themselves after a full list, and results
larger than the staging buffer.  Each test asserts which kernels ran."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lists_ran(st):
    """Six list kernels in front of each entrance kernel, for every batch."""
    return st["kernel_launches"][0] == 6 * st["kernel_launches"][1] > 0


@pytest.mark.parametrize("preset", ["NORMAL", "LARGE_BIOMES"])
def test_list_and_unit_kernels_agree(engine, wg, preset):
    """400 seeds x 100 x 100 regions (the unit kernel) and the same regions as 40,000 units of 10 x 10 (the list
    kernels), at a relaxed floor so that there are survivors."""
    seeds = wg.splitmix64_array(77, 400)
    whole = engine.seed_check(seeds=seeds, rect=(-50, 50, -50, 50), max_height=40, preset=preset)
    assert whole.stats["kernel_launches"][1] == 0 and len(whole.candidates)
    jobs = [{"seeds": seeds, "rect": (x, x + 10, z, z + 10), "max_height": 40, "preset": preset}
            for x in range(-50, 50, 10) for z in range(-50, 50, 10)]
    per, st = engine.seed_check_jobs(jobs)
    assert lists_ran(st)
    assert np.array_equal(np.sort(np.concatenate(per), order=["seed_index", "rz", "rx"]), whole.candidates)
    assert st["reject_hist"] == whole.stats["reject_hist"]
    assert st["tier_hist"] == whole.stats["tier_hist"]


def test_longest_strip_of_the_list_kernels(engine):
    kw = {"gen": (3, 24576), "rect": (0, 500, 0, 1), "max_height": 0}
    a = engine.seed_check(**kw)
    engine.set_noise_core("fp64")
    try:
        b = engine.seed_check(**kw)
    finally:
        engine.set_noise_core("fp32")
    assert lists_ran(a.stats) and not lists_ran(b.stats)
    assert np.array_equal(a.candidates, b.candidates)
    assert a.stats["reject_hist"] == b.stats["reject_hist"] and a.stats["tier_hist"] == b.stats["tier_hist"]


def test_full_lists_halve_the_batch(engine):
    """2^19 times the same seed over a rect where it has at least 20 erosion survivors: more than the 2^23
    regions a list holds, so the batch is run again in halves, and every count is 2^19 times one seed's."""
    n, preset, best = 1 << 19, "LARGE_BIOMES", (0,)
    for seed in range(1, 9):
        codes, _ = engine.phase1_codes(seeds=[seed], rect=(-64, 64, -64, 64), max_height=-50, preset=preset)
        kept = (codes[0].reshape(16, 8, 16, 8) != 0).sum((1, 3))   # per 8 x 8 block [z][x]
        z, x = np.unravel_index(kept.argmax(), kept.shape)
        best = max(best, (int(kept[z, x]), seed, -64 + 8 * int(x), -64 + 8 * int(z)))
    kept, seed, x, z = best
    assert kept >= 20
    kw = {"rect": (x, x + 8, z, z + 8), "max_height": -50, "preset": preset}
    one = engine.seed_check(seeds=[seed], **kw)
    many = engine.seed_check(seeds=np.full(n, seed, np.int64), **kw)
    st = many.stats
    assert lists_ran(st) and st["retries"] > 0
    assert st["reject_hist"] == [n * v for v in one.stats["reject_hist"]]
    assert st["tier_hist"] == [n * v for v in one.stats["tier_hist"]]
    assert len(many.candidates) == n * len(one.candidates)


def test_results_larger_than_the_staging_buffer(engine):
    """Start chunks of 8 structure seeds x 4,000 x 4,000 regions, more than 16 MiB, against one seed at a time and, for
    the first, quarters of less than 1 MiB (no staging)."""
    rect = (-2000, 2000, -2000, 2000)
    whole = engine.deep_starts(base=11, count=8, rect=rect)
    assert whole.nbytes > (16 << 20)
    for i in range(8):
        got = engine.deep_starts(base=11 + i, count=1, rect=rect)
        mine = whole[whole["seed_index"] == i]
        assert len(got) == len(mine) > (1 << 20) // got.itemsize
        for f in got.dtype.names:
            if f != "seed_index":
                assert np.array_equal(got[f], mine[f])
    rows = np.concatenate([engine.deep_starts(base=11, count=1, rect=(-2000, 2000, q, q + 500)) for q in range(-2000, 2000, 500)])
    assert rows.tobytes() == whole[whole["seed_index"] == 0].tobytes()
