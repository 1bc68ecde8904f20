"""The resident tree sort (csrc/bh.cu: tree_sort_kernel) against the separate
launches (extent, keys, one launch per radix pass): same keys, same stable
order, same extent, bit for bit.  Sizes at the edges of a sort tile, of each
number of keys per thread on 152 SMs, and of what is resident at all; states
whose runs of equal top digits are short, exactly at and over the limit at
which all seven passes run, and all equal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS, THREADS, RUN = 152, 512, 64


def _uniform(n, seed):
    from physim_gb300 import ics
    return ics.cube_with_stars(n, seed=seed)


def _clumps(n, seed):
    """Groups of bodies closer than the cells of the top 36 key bits (2^-12 of
    the extent): groups of 2, RUN, RUN + 1 and 5 RUN + 3 bodies in shuffled
    order, and as many at exactly one position."""
    s = _uniform(n, seed)
    rng = np.random.default_rng(seed)
    free = rng.permutation(np.arange(1, n))
    s[0]["x"] = 0.5  # the extent
    at = 0
    for k, size in enumerate((2, RUN, RUN + 1, 5 * RUN + 3, RUN, RUN + 1)):
        idx, at = free[at:at + size], at + size
        if len(idx) < size:
            break
        base = np.array([0.5, -0.25, 0.125]) / (k + 3) + 0.3 / 4096
        for c, f in enumerate("xyz"):
            spread = 2.0 ** -14 if k < 4 else 0.0
            s[f][idx] = base[c] + spread * rng.uniform(size=size)
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
    assert a["extent"] == b["extent"]
    assert np.array_equal(a["keys"], b["keys"])
    assert np.array_equal(a["order"], b["order"])
    # a stable order of the keys
    assert np.all(a["keys"][1:] >= a["keys"][:-1])
    same = a["keys"][1:] == a["keys"][:-1]
    assert np.all(a["order"][1:][same] > a["order"][:-1][same])


@pytest.mark.parametrize("n", [1, 2, THREADS - 1, THREADS, THREADS + 1,
                               17 * THREADS,  # the first size with two count groups
                               SMS * THREADS, SMS * THREADS + 1, SMS * THREADS * 2 + 1,
                               SMS * THREADS * 4 + 1, SMS * THREADS * 8 + 1,
                               SMS * THREADS * 16, SMS * THREADS * 16 + 1])
def test_sizes(n):
    _check(_uniform(n, seed=n % 97), "astro2")


@pytest.mark.parametrize("gravity", ["astro2", "astro"])
@pytest.mark.parametrize("n", [700, 20011, 160001])
def test_runs(n, gravity):
    _check(_clumps(n, seed=5), gravity)


@pytest.mark.parametrize("n", [3, 1500])
def test_all_at_one_position(n):
    s = _uniform(n, seed=2)
    for f in "xyz":
        s[f] = 0.25
    _check(s, "astro2")
    for f in "xyz":
        s[f] = 0.0  # extent 0: every key is 0
    _check(s, "astro2")
