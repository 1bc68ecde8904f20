"""Sizes at which kernels that are chosen by size go through all their forms.

  * whole steps of a small direct sum (csrc/direct_small.cu, up to 7,400 bodies): the
    bodies held at once (4,608) and one more, which takes a second pass over them, and
    the largest state, against the separate launches, bit for bit; accelerations there
    against the oracle;
  * the resident sort by digits (csrc/bh.cu: tree_sort_kernel, from 18,433 bodies): its
    smallest state, whole count groups of 16 tiles of 512 and one tile more, equal keys,
    extent 0 and runs that every block finds too long, against the separate radix passes, bit for bit;
  * each pair once with one, two, four and eight blocks to a tile pair
    (csrc/direct_sym.cu: pair_parts), against the one-pair kernels to 2e-6, as plans of
    the direct sum agree, and repeated bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls", [[1], [5], [1, 4], [3, 2, 1]])
@pytest.mark.parametrize("n", [4607, 4608, 4609, 6001, 7399, 7400])
def test_small_steps(n, calls):
    import physim_gb300 as pg
    from test_direct_gpu import _vec
    from test_direct_small_gpu import _state
    s = _state(n, seed=n + 1)
    out = []
    for profiling in (False, True):
        with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01, dt=1e-4)) as sim:
            assert not sim.plan()["symmetric"]
            sim.set_profiling(profiling)
            for k in calls:
                sim.step(k)
            out.append((sim.download().tobytes(), _vec(sim.accelerations()).tobytes()))
    assert out[0] == out[1]


@pytest.mark.parametrize("n", [4610, 6001, 7399, 7400])
def test_small_accelerations(oracle_mod, n):
    import physim_gb300 as pg
    from test_direct_gpu import RTOL, _vec, rel_err
    from test_direct_small_gpu import _state
    s = _state(n)
    with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01)) as sim:
        got = sim.accelerations()
    want = oracle_mod.simple_astro(s, 0.01)
    bad = np.isnan(_vec(want)).any(axis=1)
    assert np.array_equal(np.isnan(_vec(got)).any(axis=1), bad)
    assert np.all(rel_err(got[~bad], want[~bad]) < RTOL)


@pytest.mark.parametrize("kind", ["uniform", "clumps", "one position", "origin", "far body"])
@pytest.mark.parametrize("n", [18433, 32 * 512, 48 * 512, 48 * 512 + 1, 160001])
def test_resident_sort(n, kind):
    from test_tree_sort_gpu import _check, _clumps, _uniform
    n = max(n, 18433)
    s = _clumps(n, seed=3) if kind == "clumps" else _uniform(n, seed=n % 97)
    if kind == "far body":  # all others within a few cells of the top digits
        s["x"][n // 3] = 1e4
    if kind in ("one position", "origin"):
        for f in "xyz":
            s[f] = 0.25 if kind == "one position" else 0.0
    _check(s, "astro2")


@pytest.mark.parametrize("n,parts", [(14900, 8), (15300, 4), (20479, 8), (24000, 1), (52700, 2),
                                     (60500, 2), (61500, 1)])
def test_blocks_to_a_tile_pair(n, parts):
    import physim_gb300 as pg
    from physim_gb300 import ics
    from test_direct_gpu import rel_err
    s = ics.plummer(n, seed=n % 89)
    s["mass"][: n // 2] *= np.random.default_rng(n).uniform(0.5, 1.5, size=n // 2)
    cfg = pg.SimConfig(gravity="simple_astro", e=0.01)
    with pg.Simulation(s, cfg) as a, pg.Simulation(s, cfg) as b:
        assert a.plan()["symmetric"]
        b.set_plan(block=128, ipt=4, splits=4)
        got, want = a.accelerations(), b.accelerations()
        assert a.accelerations().tobytes() == got.tobytes()
    assert np.all(rel_err(got, want) < 2e-6)
