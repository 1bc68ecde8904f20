"""The exact traversal's teams (csrc/bh.cu: traverse_exact_kernel, exact_team): one,
four or eight warps walk each group's own reference lists.  Sizes on both sides of
each line of the rule (2.5 and 16 groups per SM on 152 SMs) and part groups,
against the reference restatement: 1e-5 relative per body, as for the reference
lists at other sizes."""
from __future__ import annotations

import numpy as np
import pytest

from test_bh_gpu import RTOL, _vec, rel_err

pytestmark = pytest.mark.gpu

LINES = (int(2.5 * 32 * 152), 16 * 32 * 152)


def _accelerations(s, name, theta):
    import physim_gb300 as pg
    with pg.Simulation(s, pg.SimConfig(gravity=name, theta=theta, e=0.01)) as sim:
        return sim.accelerations()


@pytest.mark.parametrize("theta", [0.3, 0.79, 0.8])
@pytest.mark.parametrize("name,nchild", [("astro2", 8), ("astro", 4)])
@pytest.mark.parametrize("n", [1, 31, 33, 2000, LINES[0], LINES[0] + 1])
def test_reference_lists(oracle_mod, n, name, nchild, theta):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n) if n > 1 else ics.cube_with_stars(1, seed=1)
    idx = np.unique(np.linspace(0, n - 1, min(n, 300)).astype(np.int64))
    got = _accelerations(s, name, theta)[idx]
    want = oracle_mod.barnes_hut(s, theta, 0.01, nchild=nchild, idx=idx)
    if n == 1:
        assert np.all(_vec(got) == 0.0)
    else:
        assert rel_err(got, want).max() < RTOL


@pytest.mark.parametrize("n", [LINES[1], LINES[1] + 1])
def test_the_upper_line(oracle_mod, n):
    from physim_gb300 import ics
    s = ics.cube_with_stars(n, seed=5)
    idx = np.linspace(0, n - 1, 200).astype(np.int64)
    got = _accelerations(s, "astro2", 0.5)[idx]
    want = oracle_mod.barnes_hut(s, 0.5, 0.01, nchild=8, idx=idx)
    assert rel_err(got, want).max() < RTOL
