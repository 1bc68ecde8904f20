"""Several steps in one call (csrc/sim.cu: pairs of steps replayed as one graph)
against the same steps one call each: the same bits, for every integrator and
gravity, for odd and even counts, across a second upload (which changes the half
of the pair-law maxima that the graphs were captured with), a new plan and
profiling switched on between."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "vx", "vy", "vz")


def _state(n, seed):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=seed)
    s["fixed"][n // 2] = 1
    return s


def _same(a, b):
    for f in FIELDS:
        assert a[f].tobytes() == b[f].tobytes(), f


@pytest.mark.parametrize("integrator", ["verlet", "euler", "rk4"])
@pytest.mark.parametrize("gravity,n", [("simple_astro", 13001), ("simple_astro", 700),
                                       ("astro2", 3001), ("astro", 20011)])
def test_steps_together_and_apart(gravity, n, integrator):
    import physim_gb300 as pg
    cfg = pg.SimConfig(gravity=gravity, theta=0.8, e=0.01, dt=1e-4, integrator=integrator)
    with pg.Simulation(_state(n, 1), cfg) as a, pg.Simulation(_state(n, 1), cfg) as b:
        for count in (1, 2, 3, 6, 5):
            a.step(count)
            for _ in range(count):
                b.step(1)
            _same(a.download(), b.download())
        a.upload(_state(n, 2))
        b.upload(_state(n, 2))
        a.step(8)
        for _ in range(8):
            b.step(1)
        _same(a.download(), b.download())


def test_plan_and_profiling_between():
    import physim_gb300 as pg
    n = 13001
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)
    with pg.Simulation(_state(n, 1), cfg) as a, pg.Simulation(_state(n, 1), cfg) as b:
        plan = dict(block=128, ipt=4, splits=8)
        for s, counts in ((a, (7, 5, 4, 6)), (b, (1,) * 22)):
            done = 0
            for c in counts:
                if done == 7:
                    s.set_plan(**plan)
                if done == 12:
                    s.set_profiling(True)
                if done == 16:
                    s.set_profiling(False)
                s.step(c)
                done += c
        _same(a.download(), b.download())
