"""The tree built in one launch (csrc/bh.cu: tree_build_kernel) against the
separate launches of the same stages: same nodes and bodies, same moments, bit
for bit (both sum the same groups in the same order).  Sizes at the edges of a
build tile (512) and of the rule, a tile for each of 152 SMs; leaves of 1 to 64
bodies; states of which two thirds are at one position."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS, TILE = 152, 512


def _state(n, kind):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n % 89) if kind == "plummer" else ics.cube_with_stars(n, seed=n % 97)
    if kind == "heap":  # most of it at one position
        for f in "xyz":
            s[f][n // 3:] = 0.1
    s["mass"] = np.random.default_rng(n).uniform(0.5, 1.5, size=n)
    return s


def _snapshot(state, cfg, single):
    import physim_gb300 as pg
    pg.lib.physim_gpu_set_sort_single_launch(single)
    try:
        with pg.Simulation(state, cfg) as sim:
            return sim.tree_snapshot()
    finally:
        pg.lib.physim_gpu_set_sort_single_launch(1)


def _check(state, gravity, **options):
    import physim_gb300 as pg
    cfg = pg.SimConfig(gravity=gravity, theta=1.0, e=0.01, **options)
    a, b = _snapshot(state, cfg, 1), _snapshot(state, cfg, 0)
    assert a.keys() == b.keys()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n", [1, 2, 3, TILE - 1, TILE, TILE + 1, 2 * TILE + 71, 31 * TILE,
                               32 * TILE, 33 * TILE + 1, 150 * TILE + 2, 151 * TILE + 1, SMS * TILE,
                               SMS * TILE + 1])
def test_sizes(n):
    _check(_state(n, "plummer"), "astro2", leaf_size=16, traversal="warp")


@pytest.mark.parametrize("kind", ["cube", "heap"])
@pytest.mark.parametrize("gravity,traversal,leaf,quad",
                         [("astro2", "exact", 1, False), ("astro2", "warp", 1, True),
                          ("astro2", "warp", 64, False), ("astro", "exact", 1, False),
                          ("astro", "warp", 7, True)])
@pytest.mark.parametrize("n", [5, 700, 20011, 70001])
def test_options(n, gravity, traversal, leaf, quad, kind):
    _check(_state(n, kind), gravity, leaf_size=leaf, traversal=traversal, quadrupole=quad)
