"""The resident sort of few bodies by ranks (csrc/bh.cu: rank_sort_kernel) against
the separate launches of the radix passes: same keys, same stable order, same
extent, bit for bit.  Sizes at the edges of a tile (256), of odd and even counts
(keys are copied in pairs) and of the rule (18,432); states where keys are equal
within and across tiles, differ in their last digits only, or are all equal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE, LARGEST = 256, 18432


def _state(n, kind):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n % 89)
    rng = np.random.default_rng(n)
    if kind == "shared":  # a few positions, each of them in every tile
        at = rng.integers(5, size=n)
        for f in "xyz":
            s[f] = rng.uniform(-1, 1, size=5)[at]
    elif kind == "near":  # within the last key bits of one another, but for one body
        for f in "xyz":
            s[f] = 0.3 + rng.uniform(size=n) * 2.0 ** -17
        s["x"][n // 2] = 1.0
    elif kind == "origin":
        for f in "xyz":
            s[f] = 0.0
    return s


def _snapshot(state, gravity, single):
    import physim_gb300 as pg
    pg.lib.physim_gpu_set_sort_single_launch(single)
    try:
        cfg = pg.SimConfig(gravity=gravity, theta=1.5, e=0.01, leaf_size=64, traversal="warp")
        with pg.Simulation(state, cfg) as sim:
            return sim.tree_snapshot()
    finally:
        pg.lib.physim_gpu_set_sort_single_launch(1)


def _check(state, gravity):
    a, b = _snapshot(state, gravity, 1), _snapshot(state, gravity, 0)
    for k in ("extent", "keys", "order", "flags"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n", [1, 2, 3, TILE - 1, TILE, TILE + 1, 2 * TILE, 2 * TILE + 1, 8195,
                               LARGEST - 1, LARGEST, LARGEST + 1])
def test_sizes(n):
    _check(_state(n, "plummer"), "astro2")


@pytest.mark.parametrize("gravity", ["astro2", "astro"])
@pytest.mark.parametrize("kind", ["shared", "near", "origin"])
@pytest.mark.parametrize("n", [200, 3 * TILE + 5, 8195])
def test_equal_and_near_keys(n, kind, gravity):
    _check(_state(n, kind), gravity)
