"""Downloads packed straight into the caller's host array against downloads through
a device copy (host access COPY): the same 80 bytes of every body, for simulations
and ensemble members, at the edges of a block's records (256), into arrays that are
16- and only 8-byte aligned, and above the size (32 MB) from which both copy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n):
    from physim_gb300 import ics
    s = ics.plummer(n, seed=n % 97)
    s["id"] = np.arange(n)[::-1]
    s["fixed"][n // 2] = 1
    return s


def _into(call, n, shift):
    """The bytes that call(pointer) leaves in an array `shift` bytes past a 16-byte
    boundary, and the bytes around it."""
    raw = np.full(n * 80 + 64, 0xA5, np.uint8)
    at = (-raw.ctypes.data) % 16 + shift
    call(raw.ctypes.data + at)
    return raw[at:at + n * 80].tobytes(), raw[:at].tobytes() + raw[at + n * 80:].tobytes()


@pytest.mark.parametrize("gravity", ["simple_astro", "astro2"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 5001, 419430, 419431])
def test_simulation(n, gravity):
    import physim_gb300 as pg
    cfg = pg.SimConfig(gravity=gravity, theta=1.0, e=0.01, leaf_size=16, traversal="warp")
    with pg.Simulation(_state(n), cfg) as sim:
        sim.step(1)
        got = {}
        for mode in (0, 1):
            pg.lib.physim_gpu_set_host_access(mode)
            try:
                for shift in (0, 8):
                    def call(p):
                        assert pg.lib.physim_gpu_sim_download(sim.handle, p, n) == 0
                    got[mode, shift], around = _into(call, n, shift)
                    assert set(around) == {0xA5}
            finally:
                pg.lib.physim_gpu_set_host_access(0)
    assert len(set(got.values())) == 1


def test_ensemble_members():
    import physim_gb300 as pg
    sizes = [1, 255, 256, 257, 3000]
    ens = pg.Ensemble([_state(n) for n in sizes], pg.SimConfig(e=0.01))
    ens.step(2)
    for k, n in enumerate(sizes):
        got = {}
        for mode in (0, 1):
            pg.lib.physim_gpu_set_host_access(mode)
            try:
                for shift in (0, 8):
                    def call(p):
                        assert pg.lib.physim_gpu_ensemble_download(ens.handle, k, p, n) == 0
                    got[mode, shift], around = _into(call, n, shift)
                    assert set(around) == {0xA5}
            finally:
                pg.lib.physim_gpu_set_host_access(0)
        assert len(set(got.values())) == 1
    ens.close()
