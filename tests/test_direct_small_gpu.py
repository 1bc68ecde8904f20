"""Small direct sums (csrc/direct_small.cu): blocks that own their bodies, as one
force pass and as whole verlet steps in one launch.

  * accelerations against the f64 oracle, 1e-5 relative per body (the FP32 pair
    law's tolerance, as for the other pair kernels), at the edges of a unit of 64
    bodies, of a block's 16 bodies, of the units the warps hold at a time (64 and
    72) and of the largest state;
  * whole steps against the separate launches (profiling on), which use the same
    force kernel and the same f64 update: bit for bit, for any division into
    calls;
  * a wait between two steps that gives up is reported and leaves the state
    alone;
  * a captured step may be launched any number of times."""
from __future__ import annotations

import numpy as np
import pytest

from test_direct_gpu import RTOL, _vec, rel_err

pytestmark = pytest.mark.gpu

LARGEST = 12500


def _state(n, seed=3):
    from physim_gb300 import ics
    s = ics.cube_with_stars(max(n - 2, 0), seed=seed, stars=ics.STARS_2[: min(n, 2)])
    if n > 9:
        s["fixed"][n // 3] = 1
        s["mass"][n // 7] = 0.0  # massless: the reference's 0/0
        for k in range(n // 2, n // 2 + 3):  # coincident bodies skip each other
            s[k]["x"], s[k]["y"], s[k]["z"] = 0.125, -0.25, 0.375
    return s


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 127, 511, 513, 2431, 2433, 4095, 4097,
                               4607, 4608, 4609, 8193, LARGEST - 1, LARGEST, LARGEST + 1])
def test_accelerations(oracle_mod, n):
    import physim_gb300 as pg
    s = _state(n)
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01)) as sim:
        got = sim.accelerations()
    want = oracle_mod.simple_astro(s, 0.01)
    bad = np.isnan(_vec(want)).any(axis=1)
    assert np.array_equal(np.isnan(_vec(got)).any(axis=1), bad)
    assert np.all(rel_err(got[~bad], want[~bad]) < RTOL)


@pytest.mark.parametrize("calls", [[1], [2], [5], [1, 4], [3, 2, 1]])
@pytest.mark.parametrize("n", [1, 40, 700, 4098, LARGEST])
def test_whole_steps_are_the_separate_launches(n, calls):
    import physim_gb300 as pg
    s = _state(n, seed=n + 1)
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)
    out = []
    for profiling in (False, True):
        with pg.Simulation(s, cfg) as sim:
            sim.set_profiling(profiling)
            for k in calls:
                sim.step(k)
            out.append((sim.download().tobytes(), _vec(sim.accelerations()).tobytes()))
    assert out[0] == out[1]


def test_a_wait_that_gives_up_is_reported():
    import physim_gb300 as pg
    s = _state(4098)
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)) as sim:
        before = sim.download()
        pg.lib.physim_gpu_set_wait_limit(1)
        try:
            sim.step(50)
            with pytest.raises(pg.PhysimError) as err:
                sim.synchronize()
            assert err.value.code == 5  # PHYSIM_ERR_TIMEOUT
        finally:
            pg.lib.physim_gpu_set_wait_limit(0)
        sim.upload(before)
        sim.step(3)
        got = sim.download()
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)) as sim:
        sim.step(3)
        assert sim.download().tobytes() == got.tobytes()


@pytest.mark.parametrize("n", [3000, 20000])
def test_a_captured_step_can_be_repeated(n):
    """Steps captured by the caller, launched three times: also the larger state's
    maxima, which change halves from step to step outside a capture, must be
    found where the launch before left them."""
    torch = pytest.importorskip("torch")
    import physim_gb300 as pg
    s = _state(n)
    stream = torch.cuda.Stream()
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4, stream=stream.cuda_stream)
    with pg.Simulation(s, cfg) as sim:
        sim.step(1)  # the Taylor step
        sim.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sim.step(1)
        with torch.cuda.stream(stream):
            for _ in range(3):
                graph.replay()
        got = sim.download()
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)) as sim:
        sim.step(4)
        assert sim.download().tobytes() == got.tobytes()
