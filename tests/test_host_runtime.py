"""The host runtime of a simulation (nfx_api.cpp) against a fake CUDA runtime, without a GPU: what a
call allocates and launches, and what it does when an allocation fails."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from nofluidx3d_gb300 import build as nbuild
from nofluidx3d_gb300 import core
from nofluidx3d_gb300._lib import _SIGS, NfxError
from nofluidx3d_gb300.workloads import Workload

HERE = Path(__file__).resolve().parent
MALLOCS, QUERIES, TETS, NODES, SIS, RUNS, ADVANCES, GRAPHS, CAPTURES, RUN_STEPS = range(10)
VP = (1e-3, 0.0, 1e-2, 1.0, 2e-4, 4e-3, 1.0, 0.0)


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake") / "libnfx_fake.so"
    cuda = Path(nbuild.nvcc_path()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-pthread", f"-I{cuda}",
                    f"-I{nbuild.INCLUDE}", f"-I{nbuild.CSRC}", str(HERE / "emulation" / "fake_cuda.cpp"),
                    str(nbuild.CSRC / "nfx_api.cpp"), str(nbuild.CSRC / "nfx_mesh.cpp"), "-ldl", "-o", str(out)],
                   check=True)
    lib = C.CDLL(str(out))
    for name, (args, res) in _SIGS.items():
        if not name.startswith(("nfx_batch", "nfx_mlp", "nfx_indenter_force_noalloc")):
            f = getattr(lib, name)
            f.argtypes, f.restype = args, res
    lib.fake_count.restype = C.c_long
    lib.fake_fail_malloc.argtypes = [C.c_long]
    return lib


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """The fake library in place of the real one for the handles of core; no allocation fails, runs
    are not possible, no stream is busy."""
    monkeypatch.setattr("nofluidx3d_gb300._lib._lib", fake_lib)
    fake_lib.fake_fail_malloc(-1)
    fake_lib.fake_run_tiles(0, 0)
    fake_lib.fake_busy(0)
    fake_lib.fake_reset()
    return fake_lib


def cell(radius=3.0, material="nh", **kw):
    w = Workload("host", radius=radius, material=material, **{"speed": 1e-3, "record_every": 10 ** 6, **kw})
    s = core.CellSim(0)
    s.mesh_of = w.configure(s, max_rows=10)
    return s


@pytest.mark.parametrize("nth", range(5))
def test_failed_allocation_of_the_viscoplastic_state(fake, nth):
    """Whichever of the state's arrays cannot be had, the call fails, and a later one that succeeds leaves
    every array in place."""
    s = cell()
    fake.fake_fail_malloc(nth)
    with pytest.raises(NfxError, match="NFX_ERR_NOMEM"):
        s.set_viscoplastic(VP)
    s.step(1)  # the elastic material is still there
    s.set_viscoplastic(VP)
    s.step(1)
    for k in range(3):
        s.tet_field(k)
    s.set_plastic_tensor_soa(s.plastic_tensor_soa())
    s.close()


def test_steps_allocate_nothing(fake):
    """Every array of the steps is there once the cell is set up, whichever way its steps go; a call for
    fewer steps than a run takes asks no other handle's stream."""
    fake.fake_run_tiles(4, 912)
    others = [cell() for _ in range(3)]
    s = cell()
    fake.fake_reset()
    s.step(1)
    for o in others:
        o.step(3)
    assert fake.fake_count(QUERIES) == 0 and fake.fake_count(TETS) == 10
    for n in (10, 500):
        s.step(n)
    assert fake.fake_count(RUNS) > 0 and fake.fake_count(MALLOCS) == 0
    for o in others + [s]:
        o.close()


def test_no_room_for_the_accumulators_of_runs(fake):
    """The mesh is set and the two passes serve."""
    fake.fake_run_tiles(608, 912)
    s = core.CellSim(0)
    w = Workload("host", radius=3.0, material="nh")
    m = w.mesh()
    s.set_mesh(m.points, m.tets)
    n = fake.fake_count(MALLOCS)
    fake.fake_reset()
    s.set_mesh(m.points, m.tets)
    arrays = fake.fake_count(MALLOCS)
    assert n > arrays
    fake.fake_fail_malloc(arrays - 1)  # the last one
    w.configure(s, m, max_rows=10)
    fake.fake_reset()
    s.step(20)
    assert fake.fake_count(RUNS) == 0 and fake.fake_count(TETS) == 20
    s.close()


def test_idle_handles_are_asked_once(fake):
    """A cell of which fewer than four fit the GPU side by side asks whether others are at work: a handle
    found idle is asked again only when it has stepped since."""
    fake.fake_run_tiles(4, 912)
    others = [cell() for _ in range(5)]
    s = cell()
    for o in others:
        o.step(2)
    fake.fake_reset()
    for _ in range(20):
        s.step(10)
    assert fake.fake_count(QUERIES) == 5 and fake.fake_count(RUNS) == 20
    others[2].step(2)
    fake.fake_busy(1)
    fake.fake_reset()
    s.step(10)
    assert fake.fake_count(QUERIES) == 1 and fake.fake_count(RUNS) == 0
    s.step(10)
    assert fake.fake_count(QUERIES) == 2  # still at work, so asked again
    fake.fake_busy(0)
    s.step(10)
    s.step(10)
    assert fake.fake_count(QUERIES) == 3 and fake.fake_count(RUNS) == 2
    for o in others + [s]:
        o.close()


@pytest.mark.parametrize("material,tiles,every,runs", [
    ("nh", 608, 1, False), ("nh", 608, 5, False), ("nh", 608, 9, False), ("nh", 608, 10, True), ("mr_vp", 608, 10, False),
    ("mr_vp", 608, 11, True), ("nh", 4, 6, False), ("nh", 4, 7, True), ("mr_vp", 4, 7, False), ("mr_vp", 4, 8, True)])
def test_short_record_intervals_keep_the_graph(fake, material, tiles, every, runs):
    """Where the steps between two that record are too few for a run to pay, a call replays the graph of
    the two passes, whose remainder is launched step by step."""
    fake.fake_run_tiles(tiles, 912)
    s = cell(material=material, record_every=every)
    fake.fake_reset()
    s.step(430)
    steps = fake.fake_count(TETS) + 100 * fake.fake_count(GRAPHS) + fake.fake_count(RUN_STEPS)
    assert steps == 430 and fake.fake_count(TETS) == fake.fake_count(NODES)
    if runs:
        assert fake.fake_count(GRAPHS) == 0 and fake.fake_count(RUNS) == len(range(0, 430 - 4, every))
    else:
        assert fake.fake_count(RUNS) == 0 and fake.fake_count(GRAPHS) == 4 and fake.fake_count(TETS) == 30
        assert fake.fake_count(ADVANCES) == 1
    s.close()


@pytest.mark.parametrize("run_tiles,indenter,every", [((608, 912), "plane", 50), ((4, 912), "plane", 7), ((0, 0), "plane", 50),
                                                      ((608, 912), "sphere_integral", 50), ((608, 912), "plane", 3)])
def test_step_counts_are_what_was_launched(fake, run_tiles, indenter, every):
    fake.fake_run_tiles(*run_tiles)
    s = cell(indenter=indenter, record_every=every)
    fake.fake_reset()
    before = s.step_counts()
    for n in (1, 3, 57, 430, 0, 12):
        s.step(n)
    got = {k: v - before[k] for k, v in s.step_counts().items()}
    graphs = fake.fake_count(GRAPHS)
    each = 3 if indenter == "sphere_integral" else 2
    assert got["passes"] == fake.fake_count(TETS) + 100 * graphs
    assert got["run4"] + got["run6"] == fake.fake_count(RUN_STEPS) == 503 - got["passes"]
    assert (got["run4"] > 0) == (run_tiles[0] > 4 and indenter == "plane" and every == 50)
    assert (got["run6"] > 0) == (run_tiles[0] == 4)
    assert got["launches"] == sum(fake.fake_count(k) for k in (TETS, NODES, SIS, RUNS, ADVANCES)) + graphs * (100 * each + 1)
    s.close()


@pytest.mark.parametrize("material", ["nh", "mr_vp"])
@pytest.mark.parametrize("every", [2 ** 63 - 1, 2 ** 63 - 2, 2 ** 62])
def test_record_interval_at_the_end_of_its_range(fake, material, every):
    """An interval that never comes, up to the largest: each step is enqueued once, the due ones by the passes."""
    fake.fake_run_tiles(608, 912)
    s = cell(material=material)
    s.set_record(1, every, 10)
    fake.fake_reset()
    for n in (10, 100, 7):  # step 0 records a row
        s.step(n)
        assert fake.fake_count(ADVANCES) < 20
    assert s.time == 117
    assert fake.fake_count(RUN_STEPS) == 116 and fake.fake_count(TETS) == 1
    s.close()
