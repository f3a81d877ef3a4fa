"""GPU: the one-CTA-per-unit phase-1 kernel (few seeds or many regions per seed), verdict by verdict
against the C restatement.

The sizes are where its tiles and blocks can go wrong: one region, blocks of 32 regions a side exactly
full and one over, rects one region wide and longer than a tile's largest side (1,023), a tile cut off
at the rect's edge, the world border, and coordinates beyond the FP32 core's range.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RECTS = [(0, 1, 0, 1), (-16, 16, -16, 16), (5, 38, -7, 26), (0, 1, -530, 570), (-40, 61, 3, 5), (-70, 70, -1, 30),
         (58540, 58594, -58594, -58550), (3_000_000, 3_000_040, -3_000_033, -3_000_000)]


@pytest.mark.parametrize("core", ["fp32", "fp64", "fp32_recheck_all"])
@pytest.mark.parametrize("version,preset", [("1.19.x~26.1", "NORMAL"), ("26.2", "LARGE_BIOMES"), ("1.18.2", "NORMAL")])
@pytest.mark.parametrize("rect", RECTS)
def test_codes_equal_the_oracle(engine, port, bind_mod, core, version, preset, rect):
    rules = bind_mod.rules(version, preset)
    seeds = [1473884015873122059, -7, 3]
    engine.set_noise_core(core)
    try:
        codes, tiers = engine.phase1_codes(seeds=seeds, rect=rect, max_height=-50, version=version, preset=preset)
    finally:
        engine.set_noise_core("fp32")
    for i, s in enumerate(seeds):
        c, t, _, _ = port.phase1_rect(s, rules, -50, rect)
        assert np.array_equal(codes[i], c)
        assert np.array_equal(tiers[i], t)


def test_survivors_equal_the_list_kernels(engine, wg):
    """A rect of many regions per seed (one CTA per tile) against the same regions in strips of few per
    seed run as jobs (the list kernels), at a relaxed floor so that there are survivors."""
    seeds = wg.splitmix64_array(77, 6)
    whole = engine.seed_check(seeds=seeds, rect=(-100, 100, -100, 100), max_height=40)
    assert len(whole.candidates)
    jobs = [{"seeds": seeds, "rect": (x, x + 20, z, z + 20), "max_height": 40} for x in range(-100, 100, 20)
            for z in range(-100, 100, 20)]
    per, st = engine.seed_check_jobs(jobs)
    parts = np.sort(np.concatenate(per), order=["seed_index", "rz", "rx"])
    assert np.array_equal(parts, whole.candidates)
    assert st["reject_hist"] == whole.stats["reject_hist"]
    assert st["tier_hist"] == whole.stats["tier_hist"]


@pytest.mark.parametrize("preset", ["NORMAL", "LARGE_BIOMES"])
@pytest.mark.parametrize("rect", [(0, 3, -160, 161), (-111, 110, 9, 13), (0, 8, 5, 92), (-60, 57, -40, -9)])
def test_thin_tiles_equal_the_oracle(engine, port, bind_mod, preset, rect):
    """Rects less than a block of 32 across, whose blocks are longer: one more region than a block's length."""
    codes, tiers = engine.phase1_codes(seeds=[41, -8], rect=rect, max_height=-50, preset=preset)
    for i, s in enumerate([41, -8]):
        c, t, _, _ = port.phase1_rect(s, bind_mod.rules("1.19.x~26.1", preset), -50, rect)
        assert np.array_equal(codes[i], c)
        assert np.array_equal(tiers[i], t)


@pytest.mark.parametrize("version,preset", [("1.19.x~26.1", "NORMAL"), ("26.2", "LARGE_BIOMES"), ("1.18.2", "NORMAL")])
@pytest.mark.parametrize("n,rect", [(24576, (-4, 5, -4, 5)), (24579, (0, 1, 0, 3)), (25001, (7, 17, -30, -21)),
                                    (24577, (58585, 58594, -58594, -58574)), (24576, (-30, 17, 0, 1)),
                                    (24577, (4, 6, -12, 12)), (24580, (0, 16, 3, 10)), (24576, (0, 501, 0, 1))])
def test_list_kernels_codes_equal_the_fp64_core(engine, version, preset, n, rect):
    """From 24,576 units of few regions on, the FP32 core takes the list kernels and the FP64 core the
    fused ones: every verdict equal, at unit counts that leave groups of units and records part full."""
    a = engine.phase1_codes(gen=(n, n), rect=rect, max_height=-50, version=version, preset=preset)
    engine.set_noise_core("fp64")
    try:
        b = engine.phase1_codes(gen=(n, n), rect=rect, max_height=-50, version=version, preset=preset)
    finally:
        engine.set_noise_core("fp32")
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])


@pytest.mark.parametrize("core", ["fp64", "fp32"])
@pytest.mark.parametrize("x0,z0", [(-128, -127), (2_999_900, -3_000_000)])
def test_pools_drained_many_times_equal_the_oracle(engine, port, bind_mod, core, x0, z0):
    """One tile of 65,536 regions a seed (64 blocks of 32 x 32): its pool fills and drains about ten times, in the
    FP64 instance too (the FP64 core, and the FP32 core beyond its small coordinates)."""
    rect, seeds = (x0, x0 + 256, z0, z0 + 256), [1473884015873122059, 11, -5]
    engine.set_noise_core(core)
    engine.set_tuning([0, 0, 0, 65536])
    try:
        per, st = engine.seed_check_jobs([{"seeds": seeds, "rect": rect, "max_height": 40}])
    finally:
        engine.set_tuning()
        engine.set_noise_core("fp32")
    assert st["kernel_launches"][1] == 0   # the unit kernel: no entrance kernel beside it
    hist, tier, rows = np.zeros(len(st["reject_hist"]), np.int64), np.zeros(len(st["tier_hist"]), np.int64), []
    for i, s in enumerate(seeds):
        c, t, _, _ = port.phase1_rect(s, bind_mod.rules("1.19.x~26.1", "NORMAL"), 40, rect)
        hist += np.bincount(c, minlength=len(hist))
        tier += np.bincount(t[t >= 0], minlength=len(tier))
        rows += [(i, x0 + int(r) % 256, z0 + int(r) // 256) for r in np.flatnonzero(c == len(hist) - 1)]
    assert st["reject_hist"] == list(hist)
    assert st["tier_hist"] == list(tier)
    assert [(int(r["seed_index"]), int(r["rx"]), int(r["rz"])) for r in per[0]] == rows


@pytest.mark.parametrize("rect", [(-16, 16, -16, 16), (-150, 150, -150, 150)])
def test_check_mode_takes_every_gate_again(engine, rect):
    """fp32_recheck_all: one FP64 decision for each region at tier 0, for each that reaches one of the six
    erosion steps after it, temperature and ridge, and for each climate survivor at the entrance gate."""
    engine.set_noise_core("fp32_recheck_all")
    try:
        st = engine.seed_check(seeds=[1473884015873122059], rect=rect, max_height=-50).stats
    finally:
        engine.set_noise_core("fp32")
    assert st["kernel_launches"][1] == 0 and st["climate_survivors"] > 0
    tier, left = st["tier_hist"], st["scanned"]
    want = left
    for t in tier[:-1]:
        left -= t
        want += left
    left -= tier[-1]
    want += left + (left - st["reject_hist"][1]) + st["climate_survivors"]
    assert st["rechecks"] == want


@pytest.mark.parametrize("n,rect,unit", [(400, (0, 56, 0, 56), True), (12000, (0, 56, 0, 56), False),
                                         (5000, (-30, 30, -30, 30), True), (200, (-2000, 2000, 0, 4), True),
                                         (1500, (-2000, 2000, 0, 4), False), (600, (-80, 80, -80, 80), True)])
def test_fp64_routes_equal_the_fp32_core(engine, n, rect, unit):
    """The FP64 core on both sides of its rules for the unit kernel (regions of a seed or of a tile, few units)
    against the FP32 core, whose unit kernel takes all of these."""
    a = engine.seed_check(gen=(n, n), rect=rect, max_height=40)
    engine.set_noise_core("fp64")
    try:
        b = engine.seed_check(gen=(n, n), rect=rect, max_height=40)
    finally:
        engine.set_noise_core("fp32")
    assert a.stats["kernel_launches"][1] == 0
    assert (b.stats["kernel_launches"][1] == 0) == unit
    assert len(a.candidates) and np.array_equal(a.candidates, b.candidates)
    assert a.stats["reject_hist"] == b.stats["reject_hist"]
    assert a.stats["tier_hist"] == b.stats["tier_hist"]


def test_no_memory_for_the_lists(wg, engine):
    """A call that would take the list kernels, with less device memory free than their lists need (228 MB):
    the fused kernels serve it, with the same survivors and funnel."""
    import torch
    want = engine.seed_check(gen=(5, 24576), rect=(-4, 5, -4, 5), max_height=40)
    assert want.stats["kernel_launches"][0] == 6 * want.stats["batches"]
    with wg.Engine(0) as e:
        e.seed_check(gen=(1, 20000), rect=(-4, 5, -4, 5), max_height=40)   # its kernels are loaded
        torch.cuda.synchronize()
        full = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (160 << 20)), dtype=torch.uint8, device="cuda")
        try:
            got = e.seed_check(gen=(5, 24576), rect=(-4, 5, -4, 5), max_height=40)
        finally:
            del full
            torch.cuda.empty_cache()
        assert got.stats["kernel_launches"][0] == got.stats["batches"]
        assert len(want.candidates) and np.array_equal(got.candidates, want.candidates)
        assert got.stats["reject_hist"] == want.stats["reject_hist"]
        again = e.seed_check(gen=(5, 24576), rect=(-4, 5, -4, 5), max_height=40)
        assert again.stats["kernel_launches"][0] == 6 * again.stats["batches"]


@pytest.mark.parametrize("queue", [True, False])
@pytest.mark.parametrize("window,unit", [(0, True), (512, False), (2048, False), (4096, False), (8192, True)])
def test_tuned_windows_choose_the_kernel(engine, queue, window, unit):
    """Jobs of more than 4,096 regions in tuned windows: small ones take the fused kernels, with the same results."""
    jobs = [{"gen": (7, 900), "rect": (-64, 65, -64, 65), "max_height": 40}]
    want, st0 = engine.seed_check_jobs(jobs)
    engine.set_tuning([0, 0, 0, window])
    engine.set_job_queue(queue)
    try:
        got, st = engine.seed_check_jobs(jobs)
    finally:
        engine.set_job_queue(True)
        engine.set_tuning()
    assert (st["kernel_launches"][1] == 0) == unit
    assert len(want[0]) and np.array_equal(got[0], want[0])
    assert st["reject_hist"] == st0["reject_hist"] and st["tier_hist"] == st0["tier_hist"]
