"""A run of steps whose wait for its CTAs gives up, which the library brings about after a few polls
(nfx_run_timeout_check): the status says so, further runs return at once instead of waiting their time
out each, and setting the mesh or loading a checkpoint makes the handle good again."""

import time

import numpy as np
import pytest

from nofluidx3d_gb300 import _lib
from nofluidx3d_gb300.core import CellSim
from nofluidx3d_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


def state(s):
    return [s.points(), s.velocities(), s.plastic_tensor_soa(), s.curve()]


@pytest.mark.parametrize("radius", [5.0, 16.0])  # four and six tiles to an SM
@pytest.mark.parametrize("again", ["set_mesh", "checkpoint"])
def test_wait_that_runs_out(radius, again):
    w = Workload("timeout", radius=radius, material="mr_vp", indenter="sphere", sphere_radius=4.0, speed=2e-3,
                 record_every=20)
    mesh = w.mesh()
    sound, s = CellSim(0), CellSim(0)
    for t in (sound, s):
        w.configure(t, mesh, max_rows=100)
        t.step(50)
    saved = s.checkpoint()
    _lib.check(s._L.nfx_run_timeout_check(s._h, 100))
    assert s.status() & _lib.STATUS_TIMEOUT
    assert s.time == 54
    begin = time.perf_counter()
    s.step(66)  # three stretches of 17 or 18 plain steps
    assert s.status() & _lib.STATUS_TIMEOUT
    assert time.perf_counter() - begin < 0.5
    if again == "checkpoint":
        s.restore(saved)
    else:
        with pytest.raises(_lib.NfxError, match="NFX_ERR_STATE"):  # the viscoplastic state went with the mesh
            s.set_mesh(mesh.points, mesh.tets)
        s.set_viscoplastic(w.vp_params())
        s.set_record(1, 20, 100)
        s.step(50)
    assert s.status() == 0
    for t in (sound, s):
        t.step(70)
    assert s.status() == 0
    for a, b in zip(state(sound), state(s)):
        assert np.array_equal(a, b)
    for t in (sound, s):
        t.close()


def test_refused():
    w = Workload("timeout", radius=5.0, material="nh")
    s = CellSim(0)
    with pytest.raises(_lib.NfxError, match="NFX_ERR_STATE"):
        _lib.check(s._L.nfx_run_timeout_check(s._h, 100))
    w.configure(s, max_rows=10)
    for polls in (0, 65537):
        with pytest.raises(_lib.NfxError, match="out of range"):
            _lib.check(s._L.nfx_run_timeout_check(s._h, polls))
    s.set_record(1, 2, 10)  # two passes only
    with pytest.raises(_lib.NfxError, match="NFX_ERR_STATE"):
        _lib.check(s._L.nfx_run_timeout_check(s._h, 100))
    s.step(10)
    assert s.status() == 0
    s.close()
