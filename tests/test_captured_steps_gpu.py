"""Steps that a caller captures."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, scale, seed):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=seed)
    for f in "xyz":
        s[f] *= scale
    for f in ("vx", "vy", "vz"):
        s[f] = 0.0
    s["mass"] *= np.random.default_rng(seed).uniform(0.5, 1.5, size=n)
    s["fixed"][n // 2] = 1
    return s


@pytest.mark.parametrize("integrator", ["verlet", "euler", "rk4"])
@pytest.mark.parametrize("gravity,n", [("simple_astro", 3000), ("simple_astro", 9001),
                                       ("astro2", 3000)])
def test_captured_after_any_number_of_steps(gravity, n, integrator):
    """The simulation's own graphs are there by then, or not, for the current half of
    the maxima: a step and a run of steps are captured all the same, and leave the
    bits of steps that were never captured."""
    torch = pytest.importorskip("torch")
    import physim_gb300 as pg
    stream = torch.cuda.Stream()
    kw = dict(gravity=gravity, theta=0.8, e=0.01, dt=1e-4, integrator=integrator)
    first = _state(n, 1.0, 1)
    with pg.Simulation(first, pg.SimConfig(stream=stream.cuda_stream, **kw)) as sim, \
            pg.Simulation(first, pg.SimConfig(**kw)) as ref:
        for before, captured in ((1, 1), (1, 1), (2, 2), (5, 4)):
            sim.step(before)
            sim.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                sim.step(captured)
            with torch.cuda.stream(stream):
                graph.replay()
            ref.step(before + captured)
            assert sim.download().tobytes() == ref.download().tobytes(), (before, captured)


@pytest.mark.parametrize("integrator", ["verlet", "euler", "rk4"])
@pytest.mark.parametrize("n", [3000, 9001])
@pytest.mark.parametrize("scale,e,dt", [(1e7, 0.01, 1e4), (1e-7, 0.0, 1e-13)])
def test_between_other_steps_and_uploads(n, scale, e, dt, integrator):
    """A captured step launched between steps and uploads outside its graph
    (csrc/integrate.cu: swap_halves): every state and its accelerations are, bit for
    bit, those of a simulation that was never captured.  At these coordinates
    accelerations are lost without the pair law's scale, so a graph or a later step
    that misses the current maxima shows."""
    torch = pytest.importorskip("torch")
    import physim_gb300 as pg
    stream = torch.cuda.Stream()
    kw = dict(gravity="simple_astro", e=e, dt=dt, integrator=integrator)
    first, second = _state(n, scale, 1), _state(n, 3.0 * scale, 2)
    second["mass"] *= 1e6
    with pg.Simulation(first, pg.SimConfig(stream=stream.cuda_stream, **kw)) as sim, \
            pg.Simulation(first, pg.SimConfig(**kw)) as ref:
        sim.step(1)
        sim.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sim.step(1)
        ref.step(1)

        def check(what):
            got, want = sim.accelerations(), ref.accelerations()
            assert np.count_nonzero(want["x"]) == n - 1, what  # one body is fixed
            assert got.tobytes() == want.tobytes(), what
            assert sim.download().tobytes() == ref.download().tobytes(), what

        def replay():
            with torch.cuda.stream(stream):
                graph.replay()
            ref.step(1)

        check("capture")
        replay()
        check("graph")
        sim.step(1)
        ref.step(1)
        check("step")
        replay()
        check("graph after a step")
        sim.step(5)
        ref.step(5)
        check("steps")
        replay()
        replay()
        check("graph twice")
        for s in (sim, ref):
            s.upload(second)
        if integrator == "verlet":  # the graph's step is not the first of a state
            sim.step(1)
            ref.step(1)
        check("upload")
        replay()
        check("graph after an upload")
        sim.step(1)
        ref.step(1)
        replay()
        check("step and graph after an upload")


def test_every_launch_that_gives_up_is_reported():
    """Whole steps of a small direct sum, captured with a wait limit of one poll:
    each launch of the graph is reported by the next synchronising call, not only the
    one that the capture itself announced.  (The state is invalid from the first on,
    until the next upload.)"""
    torch = pytest.importorskip("torch")
    import physim_gb300 as pg
    stream = torch.cuda.Stream()
    s = _state(4098, 1.0, 3)
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4, stream=stream.cuda_stream)
    with pg.Simulation(s, cfg) as sim:
        sim.step(1)
        sim.synchronize()
        graph = torch.cuda.CUDAGraph()
        pg.lib.physim_gpu_set_wait_limit(1)
        try:
            with torch.cuda.graph(graph, stream=stream):
                sim.step(50)
        finally:
            pg.lib.physim_gpu_set_wait_limit(0)
        for call in (sim.synchronize, sim.download, sim.accelerations):
            with torch.cuda.stream(stream):
                graph.replay()
            with pytest.raises(pg.PhysimError) as err:
                call()
            assert err.value.code == 5  # PHYSIM_ERR_TIMEOUT
        sim.synchronize()  # reported once each
        sim.upload(s)
        sim.step(3)
        got = sim.download()
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)) as sim:
        sim.step(3)
        assert sim.download().tobytes() == got.tobytes()
