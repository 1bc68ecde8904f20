"""The warp traversal's teams (csrc/bh.cu: traverse_warp_kernel, bh_team): one or
four warps walk for a group of 32 bodies.  With theta < 0 every cell is opened, so
the accelerations are the direct sum's, through the whole stack and queue
machinery: compared with the f64 direct sum at the sizes of a part group, a whole
one and several (theta < 0.8 and few groups: four warps).  Tolerance: the FP32 pair
law and compensated sums, 1e-5 relative per body, as for the direct sum's kernels.
With theta 0.5 the error against the f64 direct sum is the same on both sides of the
rule's line (over 8, or with the accuracy options 24, groups per SM: one warp)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vec(a):
    return np.stack([a["x"], a["y"], a["z"]], 1)


@pytest.mark.parametrize("quad", [False, True], ids=["mono", "quad"])
@pytest.mark.parametrize("leaf", [1, 16, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 1000, 5003])
def test_open_everything_is_the_direct_sum(oracle_mod, n, leaf, quad):
    import physim_gb300 as pg
    from physim_gb300 import ics
    s = ics.cube_with_stars(n, seed=n)
    cfg = pg.SimConfig(gravity="astro2", theta=-1.0, e=0.01, leaf_size=leaf, traversal="warp",
                       quadrupole=quad)
    with pg.Simulation(s, cfg) as sim:
        got = _vec(sim.accelerations())
    want = _vec(oracle_mod.simple_astro(s, 0.01, pg.accelerations(n)))
    err = np.linalg.norm(got - want, axis=1) / np.maximum(np.linalg.norm(want, axis=1), 1e-300)
    assert err.max() < 1e-5 if n > 1 else np.all(got == 0.0)


@pytest.mark.parametrize("quad,com_theta", [(False, 0.0), (True, 0.6)])
def test_one_and_four_warps_agree(quad, com_theta):
    """The same distribution below and above the rule's line: the relative error
    of a sample against f64 is a property of theta, not of the size."""
    import physim_gb300 as pg
    from physim_gb300 import ics
    lo, hi = (110000, 125000) if quad else (35000, 42000)
    cfg = pg.SimConfig(gravity="astro2", theta=0.5, e=0.01, leaf_size=16, traversal="warp",
                       quadrupole=quad, com_theta=com_theta)
    out = []
    for n in (lo, hi):
        with pg.Simulation(ics.cube_with_stars(n, seed=9), cfg) as sim:
            idx = np.arange(0, lo, 131)
            got = _vec(sim.accelerations())[idx]
            ref = _vec(sim.accelerations_f64(idx))
            out.append(np.sqrt(np.mean(np.sum((got - ref) ** 2, 1) / np.sum(ref ** 2, 1))))
    assert 0.5 < out[1] / out[0] < 2.0, out
