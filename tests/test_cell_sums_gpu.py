"""Mass, centre of mass and second moments of every cell (csrc/bh.cu:
boundary_kernel, top_groups, cell_kernel), which are summed from groups of
consecutive sorted bodies, against f64 sums over each cell's own bodies.  Sizes
at the edges of a group (4), of a block's groups (1,024) and where the second
kernel's groups begin and end; unequal masses, one of them far heavier than the
rest, so that a body counted twice or not at all shows.

Tolerances: the kernels sum the f32 masses and positions exactly to 2^-45 and
round the quotient once to f32, so against the same f32 values in f64 a mass is
within 2^-23 and a centre within 2^-23 of itself plus 2^-40 of the extent (the
sums of both signs).  Second moments are f32 sums of non-negative diagonal terms
through at most 40 joins: 1e-5 of the trace, plus the centres' rounding, a
hundredth of 2^-22 of mass times extent times the cell's size."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, seed):
    from physim_gb300 import ics
    s = ics.cube_with_stars(n, seed=seed)
    rng = np.random.default_rng(seed)
    s["mass"] = rng.uniform(0.5, 1.5, size=n)
    s["mass"][rng.integers(n)] = 1e6
    return s


@pytest.mark.parametrize("traversal,leaf", [("exact", 1), ("warp", 16)])
@pytest.mark.parametrize("quad", [False, True], ids=["mono", "quad"])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 1024, 1025, 2047, 2048, 5 * 1024 + 7, 32 * 1024,
                               33 * 1024 + 2, 1024 * 1024 + 1030])
def test_cells_against_f64(n, quad, traversal, leaf):
    import physim_gb300 as pg
    if n > 100_000 and leaf == 1:
        pytest.skip("the large size once, with the smaller tree")
    s = _state(n, seed=n % 89)
    cfg = pg.SimConfig(gravity="astro2", theta=1.5, e=0.01, leaf_size=leaf, traversal=traversal,
                       quadrupole=quad)
    with pg.Simulation(s, cfg) as sim:
        g = sim.tree_snapshot()
    assert g["flags"] == 0
    order = g["order"]
    p = np.stack([s[f] for f in "xyz"], 1).astype(np.float32).astype(np.float64)[order]
    m = s["mass"].astype(np.float32).astype(np.float64)[order]
    b, e = g["begin"].astype(np.int64), (g["begin"] + g["count"]).astype(np.int64)
    rng = np.random.default_rng(1)
    pick = np.unique(np.concatenate([np.arange(min(len(b), 600)),
                                     rng.integers(len(b), size=1500)]))
    X = g["extent"]
    for k in pick:
        mk, pk = m[b[k]:e[k]], p[b[k]:e[k]]
        M = mk.sum()
        c = (mk[:, None] * pk).sum(0) / M
        got = g["com"][k].astype(np.float64)
        assert abs(got[3] - M) <= 2.0 ** -23 * M, k
        assert np.all(np.abs(got[:3] - c) <= 2.0 ** -23 * np.abs(c) + 2.0 ** -40 * X), k
        if quad:
            d = pk - got[:3]
            S = np.einsum("i,ij,ik->jk", mk, d, d)
            want = np.array([S[0, 0], S[1, 1], S[2, 2], np.trace(S), S[0, 1], S[0, 2], S[1, 2]])
            size = np.abs(d).max()
            tol = 1e-5 * want[3] + 2.0 ** -22 * X * size * M * 1e-2
            assert np.all(np.abs(g["quad"][k][:7] - want) <= tol), (k, g["quad"][k], want)
