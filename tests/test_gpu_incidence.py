"""The element pass's incidence lists at their longest: meshes in which one node belongs to every
tetra of its tiles (a triangulated sphere joined to its centre), so a list has more words than the
CTA has threads, for every tile size; and a single tetra."""

import numpy as np
import pytest

import oracle as O
from nofluidx3d_gb300.core import CellSim
from nofluidx3d_gb300.mesh import CellMesh, signed_volumes
from nofluidx3d_gb300.workloads import Workload
from tests.helpers import oracle_problem, rel_disp, rel_traj

pytestmark = pytest.mark.gpu


def fan(n: int) -> CellMesh:
    """About n tetrahedra that share their centre node (node 0)."""
    from scipy.spatial import ConvexHull

    m = n // 2 + 2
    k = np.arange(m) + 0.5
    phi, z = np.pi * (1 + 5 ** 0.5) * k, 1 - 2 * k / m
    r = np.sqrt(1 - z * z)
    p = 6.0 * np.stack([r * np.cos(phi), z, r * np.sin(phi)], 1)
    tri = ConvexHull(p).simplices.astype(np.int64) + 1
    pts = np.concatenate([np.zeros((1, 3)), p])
    tets = np.concatenate([np.zeros((tri.shape[0], 1), np.int64), tri], 1)
    bad = signed_volumes(pts, tets) < 0
    tets[bad, 2], tets[bad, 3] = tets[bad, 3].copy(), tets[bad, 2].copy()
    return CellMesh(points=pts, tets=tets, radius=6.0)


@pytest.mark.parametrize("tile", [64, 128, 256, 512])
@pytest.mark.parametrize("tets,material", [(1, "mr"), (129, "mr"), (1100, "mr_vp")])
def test_shared_node_matches_oracle(monkeypatch, tile, tets, material):
    """200 steps from a deformed start against the FP64 oracle, at the bars of the parity suite: 1e-5 of
    the positions, 1e-3 of the displacements."""
    monkeypatch.setenv("NFX_TILE_TETS", str(tile))
    if tets == 1:
        mesh = CellMesh(points=np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]),
                        tets=np.array([[0, 1, 2, 3]], np.int64), radius=1.0)
    else:
        mesh = fan(tets)
    w = Workload("fan", radius=mesh.radius, material=material, speed=0.0, sphere_radius=2.0, indenter="sphere", d0=5.0)
    x0 = mesh.points * np.array([1.02, 0.99, 1.0])
    st = O.State(oracle_problem(w, mesh), "f64")
    st.points[:] = x0.T.reshape(-1)
    st.run(200, 100)
    s = CellSim(0)
    w.configure(s, mesh, max_rows=10)
    s.set_points(x0)
    s.step(200)
    assert s.status() == 0
    assert rel_traj(st.positions(), s.points()) < 1e-5
    assert rel_disp(st.positions(), s.points(), mesh.points) < 1e-3
    s.close()
