"""A member of an ensemble has the same bits alone and beside any others, also when
these are exchanged in mid-run.  (With so long a time step the last bits of the
accelerations reach the state.)"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _member(n):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n % 89)
    if n % 2:
        s["mass"] *= np.random.default_rng(n).uniform(0.5, 1.5, size=n)
    s["fixed"][n // 2] = 1
    return s


def _config():
    import physim_gb300 as pg
    return pg.SimConfig(gravity="simple_astro", e=0.01, dt=0.25)


def _alone(n, steps):
    import physim_gb300 as pg
    with pg.Ensemble([_member(n)], _config()) as ens:
        ens.step(steps)
        return ens.download(0).tobytes()


def _beside(sizes, others, steps):
    import physim_gb300 as pg
    with pg.Ensemble([_member(n) for n in sizes + others], _config()) as ens:
        ens.step(steps)
        return [ens.download(k).tobytes() for k in range(len(sizes))]


# 2,432 tile pairs (16 per SM) and more: one block per pair instead of a cluster
@pytest.mark.parametrize("others", [[8192], [40000], [40000] * 3, [40000] * 4])
def test_each_pair_once(others):
    sizes = [8193, 9216, 12345, 16383, 16384, 20011]
    for n, got in zip(sizes, _beside(sizes, others, 3)):
        assert got == _alone(n, 3), n


# few one-pair units, and more than four for each of the blocks that draw them
@pytest.mark.parametrize("others", [[300], [5000] * 3, [8191] * 40])
def test_one_pair_units(others):
    sizes = [1, 257, 700, 2049, 4097, 8191]
    for n, got in zip(sizes, _beside(sizes, others, 3)):
        assert got == _alone(n, 3), n


@pytest.mark.parametrize("n", [3001, 9001])
def test_exchanged_in_mid_run(n):
    import physim_gb300 as pg
    steps = 2
    ens = pg.Ensemble.slots([n, 70000], _config())
    try:
        ens.resize_member(0, n)
        ens.upload(0, _member(n))
        ens.set_member(0, 0.01, 0.25, 3 * steps)
        for other in (300, 70000, 9000):
            ens.resize_member(1, other)
            ens.upload(1, _member(other))
            ens.set_member(1, 0.01, 0.25, steps)
            ens.step(steps)
        got = ens.download(0).tobytes()
    finally:
        ens.close()
    assert got == _alone(n, 3 * steps)
