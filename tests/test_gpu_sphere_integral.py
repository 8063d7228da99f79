"""The integrated sphere contact leaves out tiles whose forces could only round to zero. With the
force recorded every step no tile is left out, so both runs must agree bit for bit — for a density
that decays within a tile, one that reaches the whole cell, and one in between."""

import numpy as np
import pytest

from nofluidx3d_gb300.core import CellSim
from nofluidx3d_gb300.workloads import Workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [64, 128, 512])
@pytest.mark.parametrize("decay", [0.3, 4.0, 12.0, 300.0])
def test_far_tiles_change_nothing(monkeypatch, tile, decay):
    monkeypatch.setenv("NFX_TILE_TETS", str(tile))
    w = Workload("si", radius=9.3, material="mr", indenter="sphere_integral", sphere_radius=2.5, d0=0.4 if decay > 1 else 60.0,
                 speed=2e-3, si_k=decay)
    mesh = w.mesh()
    out = []
    for every, rows in ((1, 200), (100000, 1)):
        s = CellSim(0)
        w.configure(s, mesh, max_rows=rows)
        s.set_record(1, every, rows)
        s.step(150)
        assert s.status() == 0
        # at 300 the density is e^-120 at the gap of 0.4, which is zero in single precision
        assert (s.indenter_force(1) != 0.0) == (decay < 300.0)
        out.append((s.points(), s.velocities()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
