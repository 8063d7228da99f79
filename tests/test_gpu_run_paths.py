"""Which way a cell's steps go: in runs of one launch, in either form, where the cell and the call allow
it, and by the two passes elsewhere — so that a comparison of the two is one."""

import numpy as np
import pytest

from nofluidx3d_gb300.core import Batch, CellSim
from nofluidx3d_gb300.workloads import Workload

pytestmark = pytest.mark.gpu

# radius, material, indenter, record_every, tile size, a loose node, and where 120 steps go
CASES = [(1.2, "mr", "plane", 50, 128, False, "run4"), (8.0, "mr", "plane", 50, 128, False, "run4"),
         (14.0, "mr_vp", "plane", 50, 128, False, "run4"), (14.9, "mr", "sphere", 50, 128, False, "run6"),
         (16.4, "mr_vp", "sphere", 30, 128, False, "run6"), (8.0, "mr", "plane", 7, 128, False, "passes"),
         (20.0, "mr", "sphere", 50, 128, False, "passes"), (8.0, "mr", "sphere_integral", 50, 128, False, "passes"),
         (8.0, "mr", "plane", 50, 256, False, "passes"), (8.0, "mr", "plane", 50, 128, True, "passes")]


@pytest.mark.parametrize("radius,material,indenter,every,tile,loose,way", CASES)
def test_way_of_the_steps(monkeypatch, radius, material, indenter, every, tile, loose, way):
    monkeypatch.setenv("NFX_TILE_TETS", str(tile))
    w = Workload("ways", radius=radius, material=material, indenter=indenter, speed=2e-3, sphere_radius=2.0,
                 record_every=every)
    mesh = w.mesh()
    if loose:
        mesh.points = np.concatenate([mesh.points, [[0.0, mesh.radius - 0.3, 0.0]]])
    s = CellSim(0)
    w.configure(s, mesh, max_rows=50)
    s.step(3)
    got = s.step_counts()
    assert got["passes"] == 3 and got["launches"] == (10 if indenter == "sphere_integral" else 7)
    s.step(117)
    got = s.step_counts()
    s.close()
    assert got["run4"] + got["run6"] + got["passes"] == 120
    if way == "passes":
        assert got["passes"] == 120
    else:  # the few steps that record or write fields, and the three above, go by the two passes
        assert got[way] >= 100 and got["passes"] == 120 - got[way]


def test_loaded_device_changes_the_way_of_larger_cells_only():
    """A cell of which fewer than four fit the GPU side by side leaves runs to a handle that is at work."""
    w = Workload("ways", radius=13.0, material="nh", indenter="sphere", sphere_radius=4.0, speed=2e-3)
    busy, s, small = CellSim(0), CellSim(0), CellSim(0)
    for t in (busy, s):
        w.configure(t, max_rows=500)
    w.with_(radius=6.0).configure(small, max_rows=500)
    s.sync()
    small.sync()
    busy.step(20000)  # some 0.1 s of work
    s.step(50)
    small.step(50)
    assert s.step_counts()["passes"] == 50
    assert small.step_counts()["run4"] >= 40
    busy.sync()
    s.step(50)
    assert s.step_counts()["run4"] >= 40
    for t in (busy, s, small):
        t.close()


def test_larger_cells_give_way_to_a_batch():
    w = Workload("ways", radius=13.0, material="nh", indenter="sphere", sphere_radius=4.0, speed=2e-3)
    batch, s = Batch(0, 128), CellSim(0)
    for r in (4.0, 5.0, 6.0):
        w.with_(radius=r).add_to_batch(batch)
    batch.set_record(1, 50, 1000)
    batch.finalize()
    w.configure(s, max_rows=500)
    s.sync()
    batch.step(20000)  # some 0.1 s of work
    s.step(50)
    assert s.step_counts()["passes"] == 50
    batch.status()  # waits for the batch
    s.step(50)
    assert s.step_counts()["run4"] >= 40
    batch.close()
    s.close()
