"""Runs of steps in one cooperative launch (small cells) against the two passes: a call for fewer than
four steps always takes the two passes, so stepping in threes and in one call must agree bit for bit —
for both forms of the launch, one tile, every material, integrator and contact, pinned nodes, a host
position table, rows recorded inside the run, and a node in no tetra (which keeps the two passes)."""

import numpy as np
import pytest

from nofluidx3d_gb300.core import CellSim
from nofluidx3d_gb300.workloads import Workload

pytestmark = pytest.mark.gpu

CASES = [dict(radius=1.2, material="mr", indenter="plane"),
         dict(radius=2.0, material="nh", indenter="sphere", integrator="vv2", xi=0.05),
         dict(radius=5.3, material="mr_vp", indenter="sphere"),
         dict(radius=8.0, material="mr", indenter="plane", record_every=7),
         dict(radius=14.0, material="mr_vp", indenter="plane"),
         dict(radius=14.9, material="mr", indenter="sphere"),
         dict(radius=16.4, material="mr_vp", indenter="sphere", record_every=30)]
PRESSED = [dict(radius=6.0, material="mr", indenter="plane", speed=2e-2),  # 2 of 6 by the last row
           dict(radius=9.0, material="mr_vp", indenter="sphere", speed=2e-2),
           dict(radius=15.0, material="mr", indenter="sphere", speed=2e-2, integrator="vv2")]


def state(s):
    return [s.points(), s.velocities(), s.force_old(), s.plastic_tensor_soa(), s.tet_field(0), s.tet_field(2), s.curve()]


@pytest.mark.parametrize("options", CASES + PRESSED, ids=lambda c: "-".join(str(v) for v in c.values()))
@pytest.mark.parametrize("extra", ["", "svk", "svkk", "pinned", "table", "loose"])
def test_run_equals_two_passes(options, extra):
    w = Workload("run", **{"speed": 2e-3, "sphere_radius": 2.0, "record_every": 50, **options})
    mesh = w.mesh()
    if extra == "loose":  # a node above the cell that no tetra uses, under the indenter's way
        mesh.points = np.concatenate([mesh.points, [[0.0, mesh.radius - 0.3, 0.0]]])
    n = 120
    rng = np.random.default_rng(3)
    v = 1e-3 * rng.standard_normal(mesh.points.shape)
    out = []
    for chunk in (3, n):
        s = CellSim(0)
        w.configure(s, mesh, max_rows=50)
        if extra in ("svk", "svkk"):
            s.set_tetra({"svk": 1, "svkk": 2}[extra], *w.tetra_params()[1:])
        if extra == "pinned" and w.integrator == "vv":
            s.set_integrator(w.xi, True)
        if extra == "table":
            s.set_contact_table(1, 0, w.contacts(mesh)[1]["p0"] - 1e-3 * np.arange(n) ** 1.1)
        s.set_velocities(v)
        for _ in range(n // chunk):
            s.step(chunk)
        out.append([np.array(s.status())] + state(s))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
    if options not in PRESSED:  # some of those invert elements, in both alike
        assert out[0][0] == 0 and np.isfinite(out[0][1]).all()
    elif extra != "table":
        assert np.abs(out[0][7]).max() > 0 and len(out[0][7]) == 3


@pytest.mark.parametrize("radius", [5.0, 13.0])
def test_handles_side_by_side(radius):
    """Cells stepped by several threads at once, where some calls meet other handles at work and take the
    two passes, against the same cell stepped alone."""
    import threading
    w = Workload("run", radius=radius, material="mr_vp", indenter="sphere", sphere_radius=4.0, speed=2e-3)
    mesh = w.mesh()
    sims = [CellSim(0) for _ in range(4)]
    for s in sims:
        w.configure(s, mesh, max_rows=50)

    def steps(s):
        for n in (50, 4, 1, 145):
            s.step(n)

    steps(sims[0])
    want = state(sims[0])
    threads = [threading.Thread(target=steps, args=(s,)) for s in sims[1:]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in sims[1:]:
        for a, b in zip(state(s), want):
            assert np.array_equal(a, b)
    for s in sims:
        s.close()
