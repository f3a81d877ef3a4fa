"""The workloads this engine is timed on, through the Python binding of libwitchgpu.so.

Every kind is a call that hunt.py or an in-process caller makes:

  check   Engine.seed_check / seed_check_device: world seeds x a rect of hut regions, phase 1
  codes   Engine.phase1_codes: the verdict of every (seed, region)
  jobs    Engine.seed_check_jobs: many uneven Seed Check jobs in one call
  serve   Server.submit / wait / take: requests that are all in the queue at once
  walk    Engine.deep_starts: huts on mineshaft start chunks, structure seeds x a rect
  sweep   Engine.deep_sweep: the forward sweep with a catalogue of layouts
  spots   Engine.deep_spots: the 65,536 upper-bit variants of each start chunk, phase 1
  solve   Engine.deep_solve: structure seeds of a plan line's layout, group by group

All outputs are whole numbers: survivors, verdicts and the funnel's counts.  The calls that need
the game's data tables (phase 2, the finisher, the biome map) are not among them: a library built
without those tables serves every case here.
"""
from __future__ import annotations

import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
M64 = (1 << 64) - 1
WORLD = 58594      # half the +-30M world's width in hut regions
# Layouts of the catalogued -58 and -59 hunts, probed by the sweep and solved by the solver.
LAYOUTS = (231564844655014, 156186219368766, 270840896143627)

# Start chunks of found huts, (structure seed, chunk x, chunk z): one world seed of each passes phase 1 at -54.
FINDS = ((15346771344729, -1549312, 1202688), (65715769224899, 84992, 981504), (10390828338972, 1509888, 1081344),
         (131406940487925, 197632, 1145344), (63222906094649, 673473, -123702), (22628496036936, -1169337, -1731564),
         (219520057933190, -1327150, -1672953), (51412493502282, -1216053, -1381130),
         (776291107475, -1079060, 1091893), (152794059197724, 1255908, 1087153), (49646657190359, -1520221, -1306360),
         (70208971750217, 1408500, -1815593))


def package():
    name = "low_witch_finder_b200"
    if name not in sys.modules:
        path = os.path.join(ROOT, "low-witch-finder_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path)
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


@functools.lru_cache(maxsize=None)
def engine(core: str):
    """A program opens one engine and makes all its calls through it."""
    return package().Engine(0, noise_core=core)


@functools.lru_cache(maxsize=None)
def server():
    return package().Server(0)


def listed():
    check = {"kind": "check", "source": "host", "version": "1.19.x~26.1", "preset": "NORMAL", "core": "fp32", "floor": -50}
    return [
        # one world seed, the hut regions within 5,000 blocks of spawn: a player's single look-up
        dict(check, name="check_one_seed_5k", seeds=1, x0=-10, x1=10, z0=-10, z1=10),
        # a few thousand listed seeds, 9 x 9 regions: one worker request of the per-area hunt
        dict(check, name="check_4k_seeds", seeds=4096, x0=-4, x1=5, z0=-4, z1=5),
        # the newest rules with LARGE_BIOMES, a deeper floor and an off-centre rect
        dict(check, name="check_256k_large", seeds=262144, x0=-6, x1=11, z0=-9, z1=6, version="26.2",
             preset="LARGE_BIOMES", floor=-54),
        # the headline: 2^24 seeds resident on the device x 9 x 9 regions
        dict(check, name="check_16m_device", seeds=1 << 24, source="device", x0=-4, x1=5, z0=-4, z1=5),
        # one seed within 40,000 blocks: hunt.py's default area
        dict(check, name="check_area_40k", seeds=1, x0=-79, x1=79, z0=-79, z1=79),
        # one seed over the whole +-30M world: hunt.py's per-seed workload
        dict(check, name="check_world", seeds=1, x0=-WORLD, x1=WORLD, z0=-WORLD, z1=WORLD),
        # uneven batched jobs: 1..4,096 seeds and radius 1..64 each, floors -50..-54
        {"name": "jobs_2k", "kind": "jobs", "jobs": 2048, "max_seeds": 4096, "max_radius": 64},
        # a job server with a backlog of requests of 1..65,536 seeds
        {"name": "serve_32", "kind": "serve", "requests": 32, "max_seeds": 65536, "max_radius": 32},
        # the region walk around spawn, every start chunk returned
        {"name": "walk_4", "kind": "walk", "seeds": 4, "x0": -2048, "x1": 2048, "z0": -2048, "z1": 2048},
        # the forward sweep of one structure seed over the whole world
        {"name": "sweep_world", "kind": "sweep", "seeds": 1, "layouts": 64, "x0": -58593, "x1": 58594, "z0": -58593,
         "z1": 58594},
        # the terrain stage of a batch of start chunks at -54
        {"name": "spots_256", "kind": "spots", "spots": 256, "version": "1.19.x~26.1", "floor": -54},
        # the solver on the -58 plan line (regime 22, offset class odd)
        {"name": "solve_odd", "kind": "solve", "layout": LAYOUTS[0], "regime": "22", "tier": "odd", "groups": 32},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(lo * (hi / lo + 1.0 / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["check"] * 5 + ["codes", "jobs", "serve", "walk", "sweep", "spots", "solve"])
    if kind in ("check", "codes"):
        w, h = _log(rng, 1, 200), _log(rng, 1, 200)
        if kind == "check" and rng.random() < 0.25:      # far from spawn, up to a large part of the world
            w, h = _log(rng, 200, 40000), _log(rng, 200, 40000)
        most = 4.0e6 if kind == "codes" else 1.0e9       # (seed, region) checks of one call
        n = _log(rng, -(-64 // (w * h)), int(max(64, min(1 << 22, most // (w * h)))))
        lim = WORLD - max(w, h)
        x0, z0 = (-(w // 2), -(h // 2)) if rng.random() < 0.6 else (rng.randint(-lim, lim), rng.randint(-lim, lim))
        c = {"kind": kind, "seeds": n, "source": "host", "x0": x0, "x1": x0 + w, "z0": z0, "z1": z0 + h,
             "version": rng.choice(["1.19.x~26.1", "1.19.x~26.1", "26.2", "1.18.2"]),
             "preset": rng.choice(["NORMAL", "NORMAL", "NORMAL", "LARGE_BIOMES"]),
             "core": rng.choice(["fp32", "fp32", "fp32", "fp64"]), "floor": -50 - rng.randrange(5)}
        if kind == "check":
            c["source"] = rng.choice(["host", "gen", "device"])
        return c
    if kind == "jobs":
        return {"kind": kind, "jobs": _log(rng, 1, 2048), "max_seeds": _log(rng, 16, 4096), "max_radius": _log(rng, 2, 64)}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 1, 32), "max_seeds": _log(rng, 16, 65536),
                "max_radius": _log(rng, 2, 32)}
    if kind in ("walk", "sweep"):
        top = 4096 if kind == "walk" else 100000
        w, h = _log(rng, 16, top), _log(rng, 16, top)
        n = _log(rng, 1, int(max(1, min(4096, (6.7e7 if kind == "walk" else 1.0e10) // (w * h)))))
        lim = WORLD - 1 - max(w, h) // 2
        x0, z0 = rng.randint(-lim, lim) - w // 2, rng.randint(-lim, lim) - h // 2
        c = {"kind": kind, "seeds": n, "x0": x0, "x1": x0 + w, "z0": z0, "z1": z0 + h}
        if kind == "sweep":
            c["layouts"] = _log(rng, 3, 4096)
        return c
    if kind == "spots":
        return {"kind": kind, "spots": _log(rng, 1, 256), "version": rng.choice(["1.19.x~26.1", "26.2", "1.18.2"]),
                "floor": rng.choice([-50, -54])}
    tier = rng.choice(["odd", "odd", "u2", "eq"])
    return {"kind": kind, "layout": rng.choice(LAYOUTS), "regime": rng.choice(["22", "00", "21"]), "tier": tier,
            "groups": _log(rng, 1, 4 if tier == "eq" else 32)}


def _regions(case):
    return (case["x1"] - case["x0"]) * (case["z1"] - case["z0"])


def _mean_log(top):
    """Mean of floor((top + 1) ** U), about."""
    return max(1.0, top / math.log(top + 1.0))


# Operations of the path, each counted once: a Perlin table (its generator, draws and swaps), one
# sample of it, the placement of one hut, the start test of one chunk, one lifted list entry.
OPS_TABLE, OPS_SAMPLE, OPS_HUT, OPS_START, OPS_LIFT = 7160, 244, 40, 60, 150


def _check_ops(seeds, regions):
    # nearly every seed with a few dozen regions reads all 18 climate tables; a region takes the two
    # samples of tier 0, and 43 % of them about 2.5 more; 1.7 % reach the caves
    tables = min(18.0, 2.0 + 1.2 * regions) + min(18.0, 0.3 * regions)
    return seeds * (tables * OPS_TABLE + regions * (OPS_HUT + (2 + 0.43 * 2.5 + 0.017 * 46) * OPS_SAMPLE))


def work(case):
    k = case["kind"]
    if k in ("check", "codes"):
        n, r = case["seeds"], _regions(case)
        return {"bytes": 8 * n + (2 * n * r if k == "codes" else 0), "flops": _check_ops(n, r)}
    if k in ("jobs", "serve"):
        n = case["jobs" if k == "jobs" else "requests"] * _mean_log(case["max_seeds"])
        return {"bytes": 8 * n if k == "jobs" else 8 * case["requests"],
                "flops": _check_ops(n, 2.0 * case["max_radius"] * _mean_log(case["max_radius"]))}
    if k in ("walk", "sweep"):
        r = case["seeds"] * _regions(case)
        return {"bytes": 8 * case["seeds"] + (40 * 0.004 * r if k == "walk" else 8 * case["seeds"]),
                "flops": r * (OPS_HUT + OPS_START)}
    if k == "spots":
        n = case["spots"] * 65536
        return {"bytes": 16 * case["spots"], "flops": n * (3.2 * (OPS_TABLE + OPS_SAMPLE) + OPS_HUT)}
    # a group holds about one region in 2^20 of its regime's; an odd or u2 class takes up to 288
    # offsets with 1,024 list entries each, and half that many for eq
    side = {"0": 32767, "1": 32768, "2": 51648}
    regions = case["groups"] * side[case["regime"][0]] * side[case["regime"][1]] / 1048576.0
    tasks = regions * {"odd": 288, "u2": 90, "eq": 191}[case["tier"]]
    return {"bytes": 32 * case["groups"], "flops": tasks * 1024 * OPS_LIFT}


def _seeds(case, seed):
    """World seeds of the whole 64-bit range."""
    return package().splitmix64_array((seed * 0x9E3779B97F4A7C15 + 0x5EED) & M64, case["seeds"])


def _structure_seeds(seed, n):
    return np.array([int(v) & 0xFFFFFFFFFFFF for v in package().splitmix64_array(seed * 7919 + 11, n)], np.int64)


def _room(case):
    """Rows a program holds ready for a call's results: far more than a call at these floors gives."""
    k = case["kind"]
    if k == "walk":
        return 4096 + int(0.006 * case["seeds"] * _regions(case))   # 0.4 % of the regions
    if k == "solve":
        return 4096 + 2048 * case["groups"]
    if k == "check":
        return 4096 + ((case["seeds"] * _regions(case)) >> 18)
    return 1 << 16


def prepare(case, seed):
    wg, k = package(), case["kind"]
    s = {"kind": k}
    if k != "codes":
        dtype = {"walk": wg.DEEP_START_DTYPE, "sweep": wg.SWEEP_MATCH_DTYPE, "solve": wg.SOLVE_HIT_DTYPE}.get(
            k, wg.CANDIDATE_DTYPE)
        s["rows"] = np.zeros((_room(case), dtype.itemsize // 4), np.int32)
    if k in ("check", "codes"):
        s["engine"] = engine(case["core"])
        s["rect"] = (case["x0"], case["x1"], case["z0"], case["z1"])
        s["floor"] = case["floor"]
        s["opts"] = wg.make_opts(case["version"], case["preset"])
        s["source"], s["n"] = case["source"], case["seeds"]
        if case["source"] == "gen":
            s["gen"] = ((seed << 32) & M64, case["seeds"])
        elif case["source"] == "device":
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["seeds"] = torch.randint(-(1 << 63), (1 << 63) - 1, (case["seeds"],), generator=g, device="cuda",
                                       dtype=torch.int64)
            s["out"] = torch.zeros(s["rows"].shape, dtype=torch.int32, device="cuda")
        else:
            s["seeds"] = _seeds(case, seed)
    elif k == "jobs":
        s["engine"] = engine("fp32")
        s["jobs"] = wg.uneven_jobs(case["jobs"], base=(seed << 32) & M64, max_seeds=case["max_seeds"],
                                   max_radius=case["max_radius"])
    elif k == "serve":
        s["server"] = server()
        s["requests"] = wg.serving_requests(case["requests"], 1.0, base=(seed << 32) & M64, max_seeds=case["max_seeds"],
                                            max_radius=case["max_radius"])
    elif k in ("walk", "sweep"):
        s["engine"] = engine("fp32")
        s["s48"] = _structure_seeds(seed, case["seeds"])
        s["rect"] = (case["x0"], case["x1"], case["z0"], case["z1"])
        if k == "sweep":
            # the catalogue: the hunts' layouts and others of real start chunks, some of them in the rect
            x, z = case["x0"], case["z0"]
            near = s["engine"].deep_starts(s48=s["s48"][:4], rect=(x, min(x + 512, case["x1"]), z, min(z + 512, case["z1"])))
            far = s["engine"].deep_starts(base=seed, count=2, rect=(-512, 512, -512, 512))
            rest = case["layouts"] - len(LAYOUTS)
            pool = np.concatenate([near["carver"][:rest // 2], far["carver"]])[:rest]
            s["layouts"] = list(LAYOUTS) + [int(v) for v in pool]
            s["values"] = list(range(len(s["layouts"])))
    elif k == "spots":
        s["engine"] = engine("fp32")
        # start chunks of the region walk and, one in sixteen, of a hut that was found
        near = s["engine"].deep_starts(base=seed * 1000003, count=3, rect=(-128, 128, -128, 128))
        near = near[np.linspace(0, len(near) - 1, case["spots"]).astype(np.int64)]
        s["s48"], s["cx"], s["cz"] = (np.array(near[f]) for f in ("s48", "chunk_x", "chunk_z"))
        for i in range(0, case["spots"], 16):
            s["s48"][i], s["cx"][i], s["cz"][i] = FINDS[(seed + i // 16) % len(FINDS)]
        s["floor"] = case["floor"]
        s["opts"] = wg.make_opts(case["version"], "NORMAL")
    else:
        s["engine"] = engine("fp32")
        s["plan"] = [(case["layout"], (int(case["regime"][0]), int(case["regime"][1])), case["tier"])]
        s["first"] = (seed * 2654435761) % ((1 << 20) - case["groups"])
        s["groups"] = case["groups"]
    return s


def _collect(s, rows):
    """The rows of a result, gathered in the program's own array."""
    n = min(len(rows), len(s["rows"]))
    s["rows"][:n] = np.ascontiguousarray(rows[:n]).view(np.int32).reshape(n, s["rows"].shape[1])
    return {"rows": s["rows"], "found": len(rows)}


def _funnel(st):
    return np.array([st["scanned"], st["accepted"], st["climate_survivors"], st["deep_candidates"]] +
                    st["reject_hist"] + st["tier_hist"], np.int64)


def run(s):
    k = s["kind"]
    if k == "check" and s["source"] == "device":
        found, st = s["engine"].seed_check_device(s["seeds"].data_ptr(), 0, s["n"], s["rect"], s["floor"], s["opts"],
                                                  s["out"].data_ptr(), len(s["out"]),
                                                  torch.cuda.current_stream().cuda_stream)
        # the survivors come home and are put in order (the device writes them as they are found)
        rows = s["out"][:min(found, len(s["out"]))].cpu().numpy()
        return dict(_collect(s, rows[np.lexsort((rows[:, 4], rows[:, 5], rows[:, 0], rows[:, 1]))]), funnel=_funnel(st))
    if k == "check":
        r = s["engine"].seed_check(seeds=s.get("seeds"), gen=s.get("gen"), rect=s["rect"], max_height=s["floor"],
                                   opts=s["opts"])
        return dict(_collect(s, r.candidates), funnel=_funnel(r.stats))
    if k == "codes":
        codes, tiers = s["engine"].phase1_codes(seeds=s["seeds"], rect=s["rect"], max_height=s["floor"], opts=s["opts"])
        return {"codes": codes, "tiers": tiers}
    if k == "jobs":
        per, st = s["engine"].seed_check_jobs(s["jobs"])
        return dict(_collect(s, np.concatenate(per)), per_job=np.array([len(p) for p in per]), funnel=_funnel(st))
    if k == "serve":
        before = _funnel(s["server"].stats())
        ids = [s["server"].submit(gen=q["gen"], rect=q["rect"], max_height=q["max_height"]) for q in s["requests"]]
        per = []
        for i in ids:
            s["server"].wait(i)
            per.append(s["server"].take(i))
        return dict(_collect(s, np.concatenate(per)), per_job=np.array([len(p) for p in per]),
                    funnel=_funnel(s["server"].stats()) - before)
    if k == "walk":
        return _collect(s, s["engine"].deep_starts(s48=s["s48"], rect=s["rect"]))
    if k == "sweep":
        matches, starts = s["engine"].deep_sweep(s["layouts"], s["values"], s48=s["s48"], rect=s["rect"])
        return dict(_collect(s, matches), starts=starts)
    if k == "spots":
        surv, bad = s["engine"].deep_spots(s["s48"], s["cx"], s["cz"], max_height=s["floor"], opts=s["opts"])
        return dict(_collect(s, surv), not_start=bad)
    hits, st = s["engine"].deep_solve(s["plan"], s["first"], s["groups"])
    return dict(_collect(s, hits), counts=np.array([st["groups"], st["regions"], st["tasks"], st["hits"]], np.int64))
