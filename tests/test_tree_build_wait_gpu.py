"""A wait between the stages of the one-launch tree build (csrc/bh.cu:
tree_build_kernel) that gives up, here because one block waits for a count that
nothing reaches: it is reported by the next synchronising call, and the next state
builds as ever."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 20011, 77824])
def test_a_build_that_gives_up_is_reported(n):
    import physim_gb300 as pg
    from physim_gb300 import ics
    s = ics.plummer(n, seed=4)
    cfg = pg.SimConfig(gravity="astro2", theta=0.8, e=0.01, dt=1e-4, leaf_size=16,
                       traversal="warp")
    with pg.Simulation(s, cfg) as sim:
        sim.step(2)
        want = sim.download()
    pg.lib.physim_gpu_set_wait_limit(1000)
    pg.lib.physim_gpu_test_stall_build(0)
    try:
        with pg.Simulation(s, cfg) as sim:
            sim.step(1)
            with pytest.raises(pg.PhysimError) as err:
                sim.synchronize()
            assert err.value.code == 5  # PHYSIM_ERR_TIMEOUT
            pg.lib.physim_gpu_test_stall_build(-1)
            pg.lib.physim_gpu_set_wait_limit(0)
            sim.set_profiling(True)  # (drops the graph that was captured with the hook)
            sim.set_profiling(False)
            sim.upload(s)
            sim.step(2)
            assert sim.download().tobytes() == want.tobytes()
    finally:
        pg.lib.physim_gpu_test_stall_build(-1)
        pg.lib.physim_gpu_set_wait_limit(0)
