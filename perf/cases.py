"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values.  ``prepare`` makes what a user's program holds before the call
(resident handles, terrain and vents on the host, page-locked result buffers), ``run`` is one pass
through the public entry points and returns whole results, ``work`` is what a pass cannot do without,
``exact`` gives independent values where a short plain computation can.

Kinds of case (field ``kind``):
  ca      one lava or classic job on a resident handle: reset, terrain, vents, run to the stop rule,
          counters and history, the five planes into page-locked memory
  steps   the same job driven step by step, as the engine does when it reports progress or snapshots
  batch   several jobs at once in one CaBatch, as the job server steps them
  basalt  the crystallisation stage on a finished lava job: domain and mobility from the CA handle,
          sweeps with statistics in between, the orientations into page-locked memory
  space   the crystallisation stage on a whole space (mc.domain = full)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from volcano_ca_mc_b200 import capi, workloads

# cooling of the defaults (a flow stays liquid for over a thousand steps) and of the small test
# configurations (it solidifies within the run)
COOLING = {
    "slow": {"cooling_ambient": 0.3, "cooling_lateral": 1.5, "cooling_fall": 0.1, "eruption_steps": 300},
    "fast": {"cooling_ambient": 3.0, "cooling_lateral": 12.0, "cooling_fall": 8.0, "eruption_steps": 150},
}


def _ca(name, nx, ny, nz, neighborhood, boundary, steps, cones, vents, cooling="slow", sweep="active", kind="ca"):
    return {"name": name, "kind": kind, "mode": "lava", "nx": nx, "ny": ny, "nz": nz, "neighborhood": neighborhood,
            "boundary": boundary, "steps": steps, "cones": cones, "vents": vents, "cooling": cooling, "sweep": sweep}


def listed():
    return [
        # A 2D cross-section of one cone: the quick look before a 3D run (the 512 x 1 x 256 workload).
        _ca("section", 512, 1, 256, "moore", "absorbing", 300, 1, 2),
        # The smallest calls: a ragged 2D section with hexagonal cells, one call per step with its
        # counters, as the engine drives a run that reports progress or writes snapshots.
        _ca("step_by_step", 333, 1, 121, "hexagonal", "periodic", 120, 1, 1, "fast", kind="steps"),
        # A run at the size of the digital-elevation-model configurations (160 x 160 x 70), odd sizes,
        # von Neumann cells, cooling fast enough to end by solidifying.
        _ca("dem_size", 163, 157, 71, "von_neumann", "absorbing", 2000, 2, 3, "fast"),
        # The mid-size 3D workload: 256 x 256 x 128, two cones, Moore, periodic.
        _ca("mid_3d", 256, 256, 128, "moore", "periodic", 400, 2, 3),
        # The largest single-GPU workload: 1024 x 1024 x 256, six cones, pentagonal, absorbing.
        _ca("large_3d", 1024, 1024, 256, "pentagonal", "absorbing", 800, 6, 8),
        # ca.sweep = full: every cell read and written every step.
        _ca("full_sweep", 512, 512, 128, "moore", "absorbing", 60, 3, 4, sweep="dense"),
        # ca.mode = classic at the size of its reference configuration: grains grow until the space is full.
        {"name": "classic", "kind": "ca", "mode": "classic", "nx": 100, "ny": 100, "nz": 100, "neighborhood": "von_neumann",
         "boundary": "periodic", "steps": 65535, "cones": 0, "vents": 10, "cooling": "slow", "sweep": "active"},
        # Ten jobs of mixed sizes stepped together, as the job server does.
        {"name": "job_batch", "kind": "batch", "members": 10, "side": 192, "steps": 300},
        # Crystallisation of the mid-size job's basalt, statistics every 25 MCS.
        {**_ca("basalt_mid", 256, 256, 128, "moore", "periodic", 400, 2, 3, kind="basalt"), "Q": 128, "kT": 0.6, "mcs": 100,
         "stats": 25},
        # Crystallisation of a large job's basalt, statistics at both ends.
        {**_ca("basalt_large", 512, 512, 256, "pentagonal", "absorbing", 800, 6, 8, kind="basalt"), "Q": 256, "kT": 0.5,
         "mcs": 200, "stats": 200},
        # Whole-space crystallisation at the size of its reference configuration, statistics every 5 MCS.
        {"name": "space_small", "kind": "space", "nx": 50, "ny": 50, "nz": 50, "neighborhood": "moore", "boundary": "periodic",
         "Q": 50, "kT": 0.0, "mcs": 50, "stats": 5},
        # Whole-space crystallisation at the benchmark's size (67 M cells), no statistics.
        {"name": "space_large", "kind": "space", "nx": 512, "ny": 512, "nz": 256, "neighborhood": "moore",
         "boundary": "periodic", "Q": 64, "kT": 0.5, "mcs": 10, "stats": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _space(rng, three, lo, hi):
    """Sides of a 2D x-z section or a 3D space (z about half a side) of lo..hi cells, odd ones among them."""
    cells = _log(rng, lo, hi)
    if not three:
        nx = max(24, int(math.sqrt(cells) * rng.uniform(1.0, 2.0)))
        return nx, 1, max(24, cells // nx)
    side = max(20, int((2 * cells) ** (1 / 3) * rng.uniform(0.9, 1.2)))
    ny = max(16, int(side * rng.uniform(0.7, 1.2)))
    return side, ny, max(16, cells // (side * ny))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, every neighbourhood, both boundaries."""
    kind = rng.choice(["ca", "ca", "ca", "steps", "batch", "basalt", "basalt", "space"])
    boundary = rng.choice(["absorbing", "periodic"])
    if kind == "batch":
        return {"kind": "batch", "members": rng.randint(3, 10), "side": rng.randint(96, 200), "steps": rng.randint(150, 400)}
    if kind == "space":
        three = rng.random() < 0.6
        if three:
            nx, ny, nz = _space(rng, True, 30_000, 30_000_000)
        else:
            n = _log(rng, 60, 2000)
            nx, ny, nz = n, max(40, int(n * rng.uniform(0.5, 1.1))), 1
        nb = rng.choice(["moore", "von_neumann", "pentagonal"] + ([] if three else ["hexagonal"]))
        cells = nx * ny * nz
        mcs = max(4, min(60, 200_000_000 // cells))
        return {"kind": "space", "nx": nx, "ny": ny, "nz": nz, "neighborhood": nb, "boundary": boundary,
                "Q": rng.choice([32, 50, 64, 128, 300]), "kT": rng.choice([0.0, 0.5, 0.8]), "mcs": mcs,
                "stats": 0 if cells > 2_000_000 else max(1, mcs // rng.randint(1, 5))}
    if kind == "ca" and rng.random() < 0.15:
        three = rng.random() < 0.7
        nx, ny, nz = _space(rng, True, 30_000, 3_000_000) if three else (rng.randint(80, 700), rng.randint(80, 700), 1)
        nb = rng.choice(["moore", "von_neumann", "pentagonal"] + ([] if three else ["hexagonal"]))
        return {"kind": "ca", "mode": "classic", "nx": nx, "ny": ny, "nz": nz, "neighborhood": nb, "boundary": boundary,
                "steps": 65535, "cones": 0, "vents": rng.randint(4, 60), "cooling": "slow", "sweep": "active"}
    three = rng.random() < 0.7
    if kind == "ca":
        nx, ny, nz = _space(rng, three, 20_000, 60_000_000 if three else 1_000_000)
        steps, sweep = rng.randint(150, 800), "active"
        if rng.random() < 0.15:
            sweep, steps = "dense", max(20, min(200, 2_000_000_000 // (nx * ny * nz)))
    elif kind == "steps":
        nx, ny, nz = _space(rng, three, 10_000, 3_000_000 if three else 300_000)
        steps, sweep = rng.randint(40, 200), "active"
    else:
        nx, ny, nz = _space(rng, three, 60_000, 40_000_000 if three else 1_000_000)
        steps, sweep = rng.randint(200, 800), "active"
    nb = rng.choice(["moore", "von_neumann", "pentagonal"] + ([] if three else ["hexagonal"]))
    case = _ca("", nx, ny, nz, nb, boundary, steps, rng.randint(1, 6), rng.randint(1, 8), rng.choice(["slow", "slow", "fast"]),
               sweep, kind)
    del case["name"]
    if kind == "basalt":
        case.update(Q=rng.choice([32, 64, 128, 256]), kT=rng.choice([0.0, 0.5, 0.6]), mcs=rng.randint(20, 200))
        case["stats"] = max(5, case["mcs"] // rng.randint(1, 6))
    return case


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _terrain(nx, ny, nz, cones, vents, seed):
    """Gaussian cones with value noise and one vent near each summit: (heights, [(x, y, z, flowId)])."""
    rng = np.random.default_rng(seed)
    x, y = np.arange(nx)[None, :], np.arange(ny)[:, None]
    h = np.zeros((ny, nx))
    tops = []
    wide = max(nx, ny)
    for _ in range(cones):
        cx = rng.uniform(0.2, 0.8) * nx
        cy = rng.uniform(0.2, 0.8) * ny if ny > 1 else 0.0
        peak, sigma = rng.uniform(0.3, 0.75) * nz, rng.uniform(0.08, 0.22) * wide
        h = np.maximum(h, peak * np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * sigma * sigma)))
        tops.append((int(cx), int(cy)))
    h = h + 0.015 * nz * workloads.value_noise(nx, ny, seed)
    heights = np.clip(np.ceil(h), 0, nz - 1).astype(np.int32)
    cells = []
    for k in range(vents):
        cx, cy = tops[k % cones]
        vx = min(nx - 1, cx + 3 * (k // cones))
        cells.append((vx, cy, int(heights[cy, vx]), k + 1))
    return heights.reshape(-1), cells


def _pinned(n, dtype):
    size = np.dtype(dtype).itemsize
    return torch.empty(n * size, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)


def _planes(n):
    return tuple(_pinned(n, t) for t in (np.uint8, np.int32, np.float32, np.uint16, np.uint16))


def _job(case, seed):
    """A resident handle, its terrain and vents, and page-locked planes for its result."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    params = capi.CaParams(nx, ny, nz, neighborhood=case["neighborhood"], boundary=case["boundary"], mode=case["mode"],
                           seed=seed, max_steps=case["steps"],
                           sweep=capi.SWEEP_DENSE if case["sweep"] == "dense" else capi.SWEEP_ACTIVE, **COOLING[case["cooling"]])
    if case["mode"] == "classic":
        rng = np.random.default_rng(seed)
        at = rng.choice(nx * ny * nz, size=case["vents"], replace=False)
        heights = None
        vents = [(int(c % nx), int(c // nx % ny), int(c // (nx * ny)), k + 1) for k, c in enumerate(at)]
    else:
        heights, vents = _terrain(nx, ny, nz, case["cones"], case["vents"], seed)
    return {"ca": capi.LavaCA(params), "heights": heights, "vents": vents, "out": _planes(nx * ny * nz),
            "history": np.zeros((3, case["steps"]), np.int64)}


def _batch_cases(case):
    """The member jobs of a batch: 2D sections and 3D spaces, every neighbourhood, both boundaries."""
    rng = np.random.default_rng(case["members"] * 1000 + case["side"])
    for k in range(case["members"]):
        side = int(rng.uniform(0.35, 1.0) * case["side"])
        three = k % 3 != 0
        nb = str(rng.choice(["moore", "von_neumann", "pentagonal"] + ([] if three else ["hexagonal"])))
        nx, ny, nz = (side, side, max(16, side // 2)) if three else (4 * side, 1, 2 * side)
        yield _ca("", nx, ny, nz, nb, ["absorbing", "periodic"][k % 2], int(case["steps"] * rng.uniform(0.7, 1.0)),
                  int(rng.integers(1, 4)), int(rng.integers(1, 6)), ["slow", "fast"][(k // 2) % 2])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ca", "steps"):
        return {"case": case, **_job(case, seed)}
    if kind == "batch":
        return {"case": case, "jobs": [_job(c, seed + k) for k, c in enumerate(_batch_cases(case))],
                "batch": capi.CaBatch(0, max_members=16)}
    n = case["nx"] * case["ny"] * case["nz"]
    mc = capi.PottsMC(capi.McParams(case["nx"], case["ny"], case["nz"], neighborhood=case["neighborhood"],
                                    boundary=case["boundary"], domain_full=kind == "space", seed=seed, Q=case["Q"],
                                    kT=case["kT"]))
    state = {"case": case, "mc": mc, "out": _pinned(n, np.int32)}
    if kind == "basalt":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        heights, vents = _terrain(nx, ny, nz, case["cones"], case["vents"], seed)
        ca = capi.LavaCA(capi.CaParams(nx, ny, nz, neighborhood=case["neighborhood"], boundary=case["boundary"], seed=seed,
                                       max_steps=case["steps"], **COOLING[case["cooling"]]))
        ca.apply_terrain(heights)
        ca.place_seeds(vents)
        ca.run()
        state["ca"] = ca
    return state


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def _set_up(job):
    ca = job["ca"]
    ca.reset()
    if job["heights"] is not None:
        ca.apply_terrain(job["heights"])
    ca.place_seeds(job["vents"])


def _result(job):
    ca = job["ca"]
    info = ca.info()
    active, changed = ca.history()
    job["history"][:2, :info.steps] = active, changed  # zero past the stop
    planes = ca.download(job["out"])
    return [*planes, job["history"], np.array([info.steps, info.stop_reason, info.lava_cells, info.air_cells], np.int64)]


def _stats(mc):
    g = mc.grains(True, 0.5)
    return mc.energy(), [int(getattr(g, name)) for name, _ in capi.GrainStats._fields_]


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "ca":
        _set_up(state)
        state["ca"].run()
        return _result(state)
    if kind == "steps":
        _set_up(state)
        ca, k = state["ca"], 0
        while ca.step():
            state["history"][2, k] = ca.info().lava_cells
            k += 1
        return _result(state)
    if kind == "batch":
        for job in state["jobs"]:
            _set_up(job)
            state["batch"].add(job["ca"])
        state["batch"].run()
        got = [_result(job) for job in state["jobs"]]
        return {"planes": [r[:5] for r in got],
                "history": np.concatenate([r[5].reshape(-1) for r in got]), "info": np.stack([r[6] for r in got])}
    mc = state["mc"]
    if kind == "basalt":
        mc.set_domain_from_ca(state["ca"])
        mc.set_mobility_from_ca(state["ca"], 0.05, True)
    else:
        mc.set_domain(None)
    mc.initialize()
    every = case["stats"] or case["mcs"]
    energies, grains, accepted, done = [], [], [], 0
    if case["stats"]:
        e, g = _stats(mc)
        energies.append(e)
        grains.append(g)
    while done < case["mcs"]:
        n = min(every, case["mcs"] - done)
        accepted.append(mc.sweep(n))
        done += n
        if case["stats"]:
            e, g = _stats(mc)
            energies.append(e)
            grains.append(g)
    info = mc.info()
    out = {"crystals": mc.crystals(state["out"]),
           "counts": np.array(accepted + [info.domain_cells, info.attempts, info.accepted, info.uphill], np.int64)}
    if case["stats"]:
        out["energy"] = np.array(energies)
        out["grains"] = np.array(grains, np.int64)
    return out


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def work(case):
    """Bytes: host inputs read once and results written once; a full sweep by its definition reads and
    writes the 13 bytes of every cell every step; a lava stage reads the 5 bytes per cell that give
    domain and mobility."""
    kind = case["kind"]
    if kind == "batch":
        return {"bytes": sum(work(c)["bytes"] for c in _batch_cases(case)), "flops": 0}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind in ("ca", "steps"):
        b = 13 * n + (4 * case["nx"] * case["ny"] if case["mode"] == "lava" else 0)
        if case["sweep"] == "dense":
            b += 26 * n * case["steps"]
        return {"bytes": b, "flops": 0}
    return {"bytes": 4 * n + (5 * n if kind == "basalt" else 0), "flops": 0}


# ------------------------------------------------------------------------------------------
# independent values
# ------------------------------------------------------------------------------------------
def _mix(x):
    """splitmix64 on uint64 arrays."""
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _prefix(seed, step):
    return _mix(_mix(np.array([seed], np.uint64) ^ np.uint64(0xA0761D6478BD642F)) ^ np.uint64(step))[0]


def exact(case, seed):
    """The orientations and energies of a small whole-space Moore run, in plain numpy.  The other cases
    have none: a lava run's temperatures are defined by their 32-bit roundings (the solidification test
    turns on them, and with it every later step), and a larger run takes too long."""
    if case["kind"] != "space" or case["neighborhood"] != "moore" or not case["stats"]:
        return None
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if n * case["mcs"] > 8_000_000 or n * case["mcs"] // case["stats"] > 1_500_000:
        return None
    periodic, Q, kT = case["boundary"] == "periodic", case["Q"], case["kT"]
    with np.errstate(over="ignore"):
        g = np.arange(n, dtype=np.uint64)
        base = _mix(_prefix(seed, 0) ^ g)
        spin = 1 + (_mix(base ^ np.uint64(0x4D43494E49544F52)) % np.uint64(Q)).astype(np.int64)
        gi = g.astype(np.int64)
        pos = [gi % nx, gi // nx % ny, gi // (nx * ny)]
        dims = [nx, ny, nz]
        rng3 = [(-1, 0, 1) if d > 1 else (0,) for d in dims]
        offs = [(a, b, c) for c in rng3[2] for b in rng3[1] for a in rng3[0] if (a, b, c) != (0, 0, 0)]
        nbs = []  # n is the index of the frame: orientation 0
        for o in offs:
            q, ok = [], np.ones(n, bool)
            for p, d, s in zip(pos, dims, o):
                v = p + s
                inside = (v >= 0) & (v < d)
                if not (periodic and d > 1):
                    ok &= inside
                q.append(v % d)
            nbs.append(np.where(ok, q[0] + nx * (q[1] + ny * q[2]), n))
        nbs = np.stack(nbs)

        def cls(p, d):
            c = p % 2 if d > 1 else np.zeros_like(p)
            return np.where(p == d - 1, 2, c) if periodic and d > 1 and d % 2 == 1 else c

        k = [1 if d == 1 else (3 if periodic and d % 2 == 1 else 2) for d in dims]
        color = cls(pos[0], nx) + k[0] * (cls(pos[1], ny) + k[1] * cls(pos[2], nz))
        lists = [np.nonzero(color == c)[0] for c in range(k[0] * k[1] * k[2])]
        fwd = np.array([o[2] > 0 or (o[2] == 0 and (o[1] > 0 or (o[1] == 0 and o[0] > 0))) for o in offs])
        spin = np.append(spin, 0)

        def energy():
            s = spin[nbs[fwd]]
            return float(((s != 0) & (s != spin[:n][None, :])).sum())

        energies = [energy()]
        for t in range(case["mcs"]):
            pre = _prefix(seed, t)
            for cells in lists:
                h = _mix(pre ^ cells.astype(np.uint64))
                cur = spin[cells]
                prop = 1 + (_mix(h ^ np.uint64(0x4D434F5249454E54)) % np.uint64(Q - 1)).astype(np.int64)
                prop += prop >= cur
                s = spin[nbs[:, cells]]
                dE = (s == cur).sum(0) - (s == prop).sum(0)
                take = dE <= 0
                if kT > 0.0:
                    u = (_mix(h ^ np.uint64(0x4D43414343455054)) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
                    take |= u < np.exp(-dE / kT)
                spin[cells] = np.where(take, prop, cur)
            if (t + 1) % case["stats"] == 0 or t + 1 == case["mcs"]:
                energies.append(energy())
    return {"crystals": spin[:n].astype(np.int32), "counts": None, "energy": np.array(energies), "grains": None}
