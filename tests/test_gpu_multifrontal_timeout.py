"""The multifrontal factorization's waits between its blocks running out: the library built with their limit at 0
(BL_MF_WAIT_NS), loaded by a process of its own. The launch ends by itself: BL_GPU_DEVERR_TIMEOUT is raised, every component
counts a failed factorization each substep and takes the elements' forces, the nodes stay finite; and a world of the library as
it is steps afterwards on the same device as it did before."""
import subprocess
import sys

import numpy as np
import pytest

from beamlab_b200 import build, rigs, world_from_rig
from conftest import ROOT

pytestmark = pytest.mark.gpu

DEVERR_TIMEOUT = 1 << 6

CHILD = """
import sys
sys.path.insert(0, {root!r})
from beamlab_b200 import _lib
_lib.LIB_PATH = {lib!r}
import numpy as np
from beamlab_b200 import rigs, world_from_rig
for make in (lambda: rigs.shell_plate(63), lambda: rigs.shell_body(10000)):
    w = world_from_rig(make())
    w.step_substeps(2)
    w.synchronize()
    st, body = w.stats(), w.bodies()[0]
    print(st["device_errors"], body.state()["fem_failures"], int(np.isfinite(body.nodes()["p"]).all()))
    w.close()
"""


def step():
    w = world_from_rig(rigs.shell_plate(63))
    w.step_substeps(10)
    p = np.ascontiguousarray(w.bodies()[0].nodes()["p"]).view(np.uint32).copy()
    assert w.stats()["device_errors"] == 0 and w.bodies()[0].state()["fem_failures"] == 0
    w.close()
    return p


def test_waits_that_run_out_end_the_launch(tmp_path):
    before = step()
    lib = str(tmp_path / "libbeamlab_timeout.so")
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-DBL_MF_WAIT_NS=0ull", "-o", lib, *build.SOURCES], check=True)
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, lib=lib)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr[-2000:]
    rows = [[int(x) for x in line.split()] for line in out.stdout.splitlines()]
    assert len(rows) == 2
    for errors, failures, finite in rows:
        assert errors & DEVERR_TIMEOUT and failures == 2 and finite == 1, rows
    assert np.array_equal(before, step())
