"""The line between the blocks that own their bodies and the each-pair-once plan
(7,400 bodies) and the sizes at which the former fill every SM (16 bodies per
block on 152 SMs): steps of the heuristic plan against those of an explicit
one-pair plan.  Both sum in FP32 with compensation, so positions and velocities
after five steps agree to relative L2 1e-6, as plans of the direct sum do."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["verlet", "euler", "rk4"])
@pytest.mark.parametrize("n", [2415, 2416, 2417, 2432, 2433, 7399, 7400, 7401, 8193])
def test_heuristic_against_one_pair(n, integrator):
    import physim_gb300 as pg
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n % 89)
    s["mass"] *= np.random.default_rng(n).uniform(0.5, 1.5, size=n)
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4, integrator=integrator)
    with pg.Simulation(s, cfg) as a, pg.Simulation(s, cfg) as b:
        b.set_plan(block=128, ipt=4, splits=4)
        a.step(5)
        b.step(5)
        x, y = a.download(), b.download()
    for f in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.linalg.norm(x[f] - y[f]) <= 1e-6 * np.linalg.norm(y[f]), f
