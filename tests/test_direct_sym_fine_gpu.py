"""The each-pair-once plan where the one-pair kernels would serve otherwise (7,401 to
20,479 bodies, csrc/direct_sym.cu: kSymFine): its error against the direct sum in 64
bits is no larger than theirs.  Equal masses, masses that differ, and a cube whose
four stars hold two sevenths of the mass, in its own order (the stars last, where the
one-pair kernels add nothing after them) and shuffled; sizes with whole tiles of
1,024 bodies and a few more or less, and those at which each number of blocks shares
a tile pair.  The kernels' chains are shorter than the one-pair kernels' 128 terms, so
their error is smaller or, where the arithmetic of the pairs is most of it, the same:
5% are left for what three states of a kind differ by."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(kind, n, seed):
    from physim_gb300 import ics
    rng = np.random.default_rng(1000 * seed + n)
    if kind in ("plummer", "masses"):
        s = ics.plummer(n, seed=seed)
        if kind == "masses":
            s["mass"] *= rng.uniform(0.5, 1.5, size=n)
        return s
    s = ics.cube_with_stars(n - 4, seed=seed, stars=ics.STARS_4, star_mass=0.1 * n)
    s["mass"] /= n
    return s[rng.permutation(n)] if kind == "shuffled" else s


def _exact(torch, s, e):
    """The law on the f32 values that the kernels take, in f64."""
    x = torch.tensor(np.stack([s[c] for c in "xyz"], 1).astype(np.float32), device="cuda").double()
    m = torch.tensor(s["mass"].astype(np.float32), device="cuda").double()
    out = torch.empty_like(x)
    for a in range(0, len(s), 1024):
        d = x[None] - x[a:a + 1024, None]
        r2 = (d * d).sum(2)
        w = m[None] / (torch.sqrt(r2) * (r2 + e))
        w = torch.where(r2 > 0, w, torch.zeros_like(w))
        out[a:a + 1024] = (w[..., None] * d).sum(1)
    return out.cpu().numpy()


@pytest.mark.parametrize("kind", ["plummer", "masses", "stars", "shuffled"])
@pytest.mark.parametrize("n", [7401, 8192, 8195, 10007, 12600, 15300, 16387, 18001, 20479])
def test_error_against_one_pair_kernels(n, kind):
    torch = pytest.importorskip("torch")
    import physim_gb300 as pg
    square = {"plan": 0.0, "one": 0.0}
    for seed in range(3):
        s = _state(kind, n, seed)
        want = _exact(torch, s, 0.01)
        for name in square:
            with pg.Simulation(s, pg.SimConfig(gravity="simple_astro", e=0.01)) as sim:
                if name == "one":
                    sim.set_plan(block=128, ipt=4, splits=8)
                else:
                    assert sim.plan()["symmetric"]
                a = sim.accelerations()
            err = np.linalg.norm(np.stack([a[c] for c in "xyz"], 1) - want, axis=1)
            square[name] += np.mean((err / np.linalg.norm(want, axis=1)) ** 2)
    assert np.sqrt(square["plan"]) <= 1.05 * np.sqrt(square["one"])
