"""Handles of different sizes at work in several threads. The limit on a kernel's dynamic shared memory
is one for the process: were it set to each handle's own need, one thread's launch would fail when
another had lowered it in between. Networks of 16 and 1024 wide, and two meshes in 512-tetra tiles
whose incidence lists differ in length, each against the same work done alone."""

import threading

import numpy as np
import pytest

from nofluidx3d_gb300.core import CellSim
from nofluidx3d_gb300.mlp import MLP
from nofluidx3d_gb300.workloads import Workload
from tests.test_gpu_incidence import fan

pytestmark = pytest.mark.gpu


def side_by_side(jobs):
    """Results of the jobs, each in a thread of its own; the first exception of any is raised."""
    out, errors = [None] * len(jobs), []

    def run(k):
        try:
            out[k] = jobs[k]()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return out


def training(width, n_out, calls):
    rng = np.random.default_rng(width)
    with MLP(6, width, 2, n_out, 8) as m:
        p = rng.normal(0, 0.05, m.num_params).astype(np.float32)
        m.set_params(p)
        x = rng.uniform(-1, 1, (8, 6)).astype(np.float32)
        t = rng.normal(0, 1, (8, n_out)).astype(np.float32)
        for _ in range(calls):
            m.train(x, t, steps=100, batch=8, lr=1e-4)
        return m.params()


def test_networks_of_different_widths():
    jobs = [lambda: training(16, 8, 30), lambda: training(1024, 1024, 30)]
    alone = [job() for job in jobs]
    for a, b in zip(alone, side_by_side(jobs)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("indenter", ["sphere", "sphere_integral"])
def test_meshes_of_different_lists_in_wide_tiles(monkeypatch, indenter):
    monkeypatch.setenv("NFX_TILE_TETS", "512")

    def steps(mesh):
        w = Workload("t", radius=mesh.radius, material="mr", speed=0.0, sphere_radius=2.0, indenter=indenter, d0=5.0)
        s = CellSim(0)
        w.configure(s, mesh, max_rows=1000)
        for _ in range(200):
            s.step(40)
        out = s.points()
        s.close()
        return out

    jobs = [lambda: steps(fan(1100)), lambda: steps(Workload("c", radius=5.0).mesh())]
    alone = [job() for job in jobs]
    for a, b in zip(alone, side_by_side(jobs)):
        assert np.array_equal(a, b)
