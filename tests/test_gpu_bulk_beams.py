"""The bulk-copy beams' kernel (beam_kernel 2: at any size) against the CPU restatement and against plain loads, bit for bit:
beams that yield and break, in builder order and shuffled; fewer tiles of 512 beams than a block keeps in flight and a last
tile in part; wheels and shocks after a block's tiles; and beams whose tiles span more nodes than 16-bit ends hold."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig
from gpu_adapter import GpuWorld
from oracle.oracle import PortWorld, build_world
from test_gpu_parity import _wall_crash, assert_same

pytestmark = pytest.mark.gpu


def equal_port(rig, frames, n, bodies=1):
    gw, ow = GpuWorld(rig, beam_kernel=2), build_world(PortWorld, rig)
    for f in range(frames):
        gw.step_substeps(n)
        ow.step_substeps(n)
    assert_same(gw, ow, bodies)
    assert gw.w.stats()["device_errors"] == 0
    return gw


@pytest.mark.parametrize("shuffle", [False, True])
def test_yield_and_break_equal_port(port_lib, shuffle):
    gw = equal_port(_wall_crash(5, shuffle), 12, 25)
    assert gw.body(0)["broken_beams"] > 100


@pytest.mark.parametrize("dims", [(2, 2, 2), (11, 3, 1), (20, 4, 5), (25, 16, 16)])
def test_sizes_equal_port(port_lib, dims):
    equal_port(rigs.truss_car(3, speed=15.0, dims=dims), 2, 20)


def test_ends_past_16_bits_equal_port(port_lib):
    """The crash's nodes at both ends of 70,000 others: every tile's ends 69,000 nodes apart and more."""
    rig = _wall_crash(5, shuffle=True)
    b = dict(rig["bodies"][0])
    n, lone = len(b["mass"]), 70000
    place = np.where(np.arange(n) % 2 == 0, np.arange(n), np.arange(n) + lone)
    rest = np.setdiff1d(np.arange(n + lone), place)
    for k in ("pos", "vel", "mass", "node_flags", "friction", "radius"):
        a = np.zeros((n + lone,) + b[k].shape[1:], b[k].dtype)
        a[place] = b[k]
        a[rest] = b[k][0]
        b[k] = a
    b["pos"][rest] = (0.0, 50.0, 5.0)
    b["ab"] = place[b["ab"].astype(np.int64)].astype(np.uint32)
    span = [np.ptp(b["ab"][t:t + 512].astype(np.int64)) for t in range(0, len(b["ab"]), 512)]
    assert max(span) >= 65536
    equal_port(dict(rig, bodies=[b]), 6, 25)


def test_wheels_and_shocks_equal_plain_loads():
    rig = rigs.wheeled_car(shocks=rigs.SHOCK_TYPES[2])
    worlds = [world_from_rig(rig, beam_kernel=k) for k in (2, 1)]
    for w in worlds:
        w.bodies()[0].set_wheel_drive(0, 300.0)
        for _ in range(6):
            w.step_substeps(33)
    a, b = (w.bodies()[0].nodes() for w in worlds)
    assert np.array_equal(a["p"].view(np.uint32), b["p"].view(np.uint32)) and np.array_equal(a["v"].view(np.uint32), b["v"].view(np.uint32))
    a, b = (w.bodies()[0].beams() for w in worlds)
    assert np.array_equal(a["stress"].view(np.uint32), b["stress"].view(np.uint32))
    assert worlds[0].stats()["device_errors"] == 0
    for w in worlds:
        w.close()
