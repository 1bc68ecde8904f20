"""The calls whose speed matters to a user of this package.

Three ways in, each through the public classes:

  pipeline   physim's own step on host arrays: zeroed accelerations, the element's
             transform, the verlet integrator (`Pipeline.step`), one step per pass;
  sim        a device-resident `Simulation`: `step(k)`, then `download()`, as a
             program that renders or writes every k-th state does;
  ensemble   many uneven direct-sum members advanced together: `step(k)`, then every
             member's state.

A pass hands on the whole new state.  Bodies are the repository's synthetic
workloads (a Plummer sphere; a spinning cube with four heavy stars) with the total
mass near 1, so that a state stays close to its start however many passes are made.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import physim_gb300 as pg
from physim_gb300 import ics

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "radius", "mass", "id", "fixed")

_DEFAULTS = dict(gravity="simple_astro", n=0, steps=1, ic="plummer", fixed=0, e=0.01, dt=1e-5,
                 theta=1.0, leaf=1, traversal="exact", quadrupole=False, com_theta=0.0,
                 integrator="verlet", members=0, lo=0, hi=0)


def _case(path: str, name: str | None = None, **kw) -> dict:
    c = dict(_DEFAULTS, path=path, **kw)
    if name:
        c["name"] = name
    return c


def listed() -> list[dict]:
    return [
        # the smallest host-array step: a few launches and synchronisations, no arithmetic
        _case("pipeline", "pipeline_direct_1k", n=1002, ic="cube"),
        # an ordinary exact-gravity pipeline, odd size, a few bodies held fixed
        _case("pipeline", "pipeline_direct_30k", n=30011, fixed=7),
        # the drop-in default of `astro2`: one body per leaf, each body's own list
        _case("pipeline", "pipeline_astro2_250k", gravity="astro2", n=250007, theta=1.0),
        # the quadtree element at the tighter opening angle
        _case("pipeline", "pipeline_astro_50k", gravity="astro", n=50021, theta=0.5, ic="cube"),
        # the small direct-sum + verlet configuration: 100 short steps per frame
        _case("sim", "sim_direct_4k", n=4098, steps=100, ic="cube"),
        # four force evaluations per step, between the small and the large kernels
        _case("sim", "sim_direct_rk4_16k", n=16387, steps=5, integrator="rk4"),
        # the precision study's size: a Plummer sphere of 262,144 bodies, made odd
        _case("sim", "sim_direct_262k", n=262147, steps=1),
        # the headline direct sum
        _case("sim", "sim_direct_1m", n=1048580, steps=1, ic="cube"),
        # a small served job: the tree build is all launches and latency
        _case("sim", "sim_bh_8k", gravity="astro2", n=8195, steps=50, theta=0.5, leaf=16,
              traversal="warp"),
        # the large Barnes-Hut configuration
        _case("sim", "sim_bh_1m", gravity="astro2", n=1048580, steps=40, theta=0.5, leaf=16,
              traversal="warp", ic="cube"),
        # the accuracy options: quadrupoles and the centre-of-mass guard
        _case("sim", "sim_bh_quad_100k", gravity="astro2", n=100003, steps=10, theta=0.5, leaf=16,
              traversal="warp", quadrupole=True, com_theta=0.6),
        # a batch of uneven members, sizes log-uniform
        _case("ensemble", "ensemble_30", members=30, lo=256, hi=16384, steps=10),
    ]


def _size(rng, lo: int, hi: int) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng) -> dict:
    """One more case: a way in, an element, its options, and a size log-uniform over
    the range in which the element is used that way."""
    ic = rng.choice(("plummer", "cube"))
    e = rng.choice((0.01, 0.001, 1.0))
    path = rng.choice(("pipeline", "pipeline", "sim", "sim", "sim", "ensemble"))
    if path == "ensemble":
        lo = _size(rng, 100, 2000)
        return _case(path, members=rng.randint(6, 32), lo=lo, hi=lo * rng.randint(2, 16), e=e,
                     steps=rng.randint(3, 20), ic=ic)
    tree = rng.random() < 0.55
    if path == "pipeline":
        fixed = rng.choice((0, 0, 3))
        if not tree:
            return _case(path, n=_size(rng, 300, 200000), ic=ic, e=e, fixed=fixed)
        return _case(path, gravity=rng.choice(("astro2", "astro2", "astro")),
                     n=_size(rng, 1000, 1000000), theta=rng.choice((0.3, 0.5, 1.0, 1.5)), ic=ic,
                     e=e, fixed=fixed)
    if not tree:
        n = _size(rng, 500, 400000)
        integrator = rng.choice(("verlet", "verlet", "euler", "rk4"))
        evals = 4 if integrator == "rk4" else 1
        steps = max(1, min(100, int(2e11 / (evals * float(n) * n))))
        return _case(path, n=n, steps=steps, integrator=integrator, ic=ic, e=e)
    n = _size(rng, 2000, 1000000)
    steps = max(5, min(100, int(2e7 / n)))
    warp = rng.random() < 0.7
    quad = warp and rng.random() < 0.3
    return _case(path, gravity=rng.choice(("astro2", "astro2", "astro2", "astro")), n=n,
                 steps=steps, theta=rng.choice((0.5, 0.7, 1.0, 1.5)),
                 leaf=rng.choice((8, 16, 16, 32)) if warp else 1,
                 traversal="warp" if warp else "exact", quadrupole=quad,
                 com_theta=0.6 if quad else 0.0, ic=ic, e=e)


def _bodies(ic: str, n: int, seed: int, fixed: int = 0) -> np.ndarray:
    if ic == "cube":
        s = ics.cube_with_stars(n - 4, seed=seed, stars=ics.STARS_4, star_mass=0.1 * n)
        s["mass"] /= n
        # a velocity dispersion, as bodies have after a few steps
        rng = np.random.Generator(np.random.PCG64(seed + 1))
        for f in ("vx", "vy", "vz"):
            s[f] += rng.normal(0.0, 0.3, size=n)
    else:
        s = ics.plummer(n, seed=seed)
    if fixed:
        s["fixed"][np.random.Generator(np.random.PCG64(seed)).choice(n, fixed, replace=False)] = 1
    return s


def _states(case: dict, seed: int) -> list[np.ndarray]:
    if case["path"] != "ensemble":
        return [_bodies(case["ic"], case["n"], seed, case["fixed"])]
    # the members' sizes are the case's, so that every seed does the same work
    sizes = ics.ensemble_sizes(case["members"], seed=3, lo=case["lo"], hi=case["hi"])
    return [_bodies(case["ic"], int(n), seed + 1000 * k) for k, n in enumerate(sizes)]


def _config(case: dict) -> pg.SimConfig:
    return pg.SimConfig(gravity=case["gravity"], theta=case["theta"], e=case["e"], dt=case["dt"],
                        leaf_size=case["leaf"], traversal=case["traversal"],
                        integrator=case["integrator"], quadrupole=case["quadrupole"],
                        com_theta=case["com_theta"])


def prepare(case: dict, seed: int) -> dict:
    states = _states(case, seed)
    out = {"path": case["path"], "steps": case["steps"]}
    if case["path"] == "pipeline":
        props = {"e": case["e"]}
        if case["gravity"] != "simple_astro":
            props["theta"] = case["theta"]
        element = pg.TransformElementHandler(case["gravity"], props)
        out["pipeline"] = pg.Pipeline([element], pg.GpuVerlet(), case["dt"])
        out["state"] = states[0]
    elif case["path"] == "sim":
        out["sim"] = pg.Simulation(states[0], _config(case))
    else:
        out["ensemble"] = pg.Ensemble(states, _config(case))
    return out


def _fields(state: np.ndarray) -> dict:
    return {f: state[f] for f in FIELDS}


def _columns(state: np.ndarray) -> list:
    """A member's state as two arrays without a copy: x .. mass, and (id, fixed)."""
    words = state.view(np.uint64).reshape(-1, 10)
    return [words[:, :8].view(np.float64), words[:, 8:]]


def run(state: dict):
    if state["path"] == "pipeline":
        state["state"] = state["pipeline"].step(state["state"])
        return _fields(state["state"])
    if state["path"] == "sim":
        state["sim"].step(state["steps"])
        return _fields(state["sim"].download())
    ens = state["ensemble"]
    ens.step(state["steps"])
    return [_columns(ens.download(k)) for k in range(len(ens.sizes))]


def _evaluations(case: dict) -> int:
    return case["steps"] * (4 if case["integrator"] == "rk4" else 1)


def work(case: dict) -> dict:
    """Bytes: the state (80 bytes a body) in and out.  Operations: 27 per unordered
    pair (17 FP32 lane operations, ten of them multiply-adds) for direct sums; for trees
    20 per interaction at about 60 log2(n) / (1 + theta)^3 interactions a body."""
    if case["path"] == "ensemble":
        sizes = [int(v) for v in ics.ensemble_sizes(case["members"], seed=3, lo=case["lo"],
                                                    hi=case["hi"])]
    else:
        sizes = [case["n"]]
    flops = 0.0
    for n in sizes:
        if case["gravity"] == "simple_astro":
            flops += 27.0 * n * (n - 1) / 2
        else:
            flops += 20.0 * n * 60.0 * math.log2(n) / (1.0 + case["theta"]) ** 3
    return {"bytes": 160.0 * sum(sizes), "flops": flops * _evaluations(case)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _acc64(pos: torch.Tensor, mass: torch.Tensor, fixed: torch.Tensor, e: float) -> torch.Tensor:
    """sum_j m_j (x_j - x_i) / (r (r^2 + e)) over bodies at other positions; 0 where fixed."""
    n = pos.shape[0]
    out = torch.empty_like(pos)
    step = max(1, min(n, 24_000_000 // n))
    for a in range(0, n, step):
        p = pos[a:a + step]
        d = [pos[None, :, c] - p[:, None, c] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        w = mass[None, :] / (torch.sqrt(r2) * (r2 + e))
        w = torch.where(r2 > 0, w, torch.zeros_like(w))
        for c in range(3):
            out[a:a + step, c] = (w * d[c]).sum(1)
    out[fixed] = 0.0
    return out


def _advance64(s: np.ndarray, case: dict) -> np.ndarray:
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def col(names):
        return torch.tensor(np.stack([s[f] for f in names], 1), dtype=torch.float64, device=dev)

    x, v = col(("x", "y", "z")), col(("vx", "vy", "vz"))
    mass = torch.tensor(s["mass"].copy(), dtype=torch.float64, device=dev)
    fixed = torch.tensor(s["fixed"].astype(bool), device=dev)
    dt, prev = case["dt"], None

    def acc(p):
        return _acc64(p, mass, fixed, case["e"])

    for _ in range(case["steps"]):
        if case["integrator"] == "rk4":
            k = [(dt * v, dt * acc(x))]
            for half in (0.5, 0.5, 1.0):
                kx, kv = k[-1]
                k.append((dt * (v + half * kv), dt * acc(x + half * kx)))
            x = x + (k[0][0] + 2 * k[1][0] + 2 * k[2][0] + k[3][0]) / 6
            v = v + (k[0][1] + 2 * k[1][1] + 2 * k[2][1] + k[3][1]) / 6
        elif case["integrator"] == "euler" or prev is None:
            a = acc(x)
            prev, x, v = x, x + v * dt + 0.5 * a * dt * dt, v + a * dt
        else:
            a = acc(x)
            new = 2 * x - prev + a * dt * dt
            prev, x, v = x, new, (new - x) / dt
    x, v = x.cpu().numpy(), v.cpu().numpy()
    out = s.copy()
    for c, f in enumerate("xyz"):
        out[f], out["v" + f] = x[:, c], v[:, c]
    return out


def exact(case: dict, seed: int):
    """The direct sum in 64 bits and the same integrator; for the tree elements, what
    they approximate.  None where that takes too long."""
    states = _states(case, seed)
    pairs = sum(float(len(s)) ** 2 for s in states) * _evaluations(case)
    if pairs > 1.5e11:
        return None
    parts = [_advance64(s, case) for s in states]
    return [_columns(p) for p in parts] if case["path"] == "ensemble" else _fields(parts[0])
