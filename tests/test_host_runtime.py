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
