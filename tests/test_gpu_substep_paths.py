"""The explicit substep's ways over world sizes, against the CPU restatement bit for bit: nodes of up to 6,000 a warp each and
above that a thread each (sizes on both sides of a warp's width and of the line between them), and hubs of more beams than a
warp's lanes; and the bulk-copy launch of the largest worlds against the plain one, wheels and shocks included."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig
from oracle.oracle import PortWorld, build_world

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def equal_port(rig):
    w, p = world_from_rig(rig), build_world(PortWorld, rig)
    for f in range(2):
        w.step_substeps(20)
        p.step_substeps(20)
        g, r = w.bodies()[0].nodes(), p.nodes(0)
        assert np.array_equal(bits(g["p"]), bits(r["pos"])) and np.array_equal(bits(g["v"]), bits(r["vel"])), f
    w.close()


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 4, 2), (11, 3, 1), (20, 4, 5), (25, 15, 16), (25, 16, 16)])
def test_sizes_equal_port(dims):
    equal_port(rigs.truss_car(3, speed=15.0, dims=dims))


@pytest.mark.parametrize("dims,beams", [((4, 4, 2), 31), ((6, 4, 4), 70), ((25, 16, 16), 300)])
def test_hub_equals_port(dims, beams):
    """The first node tied to `beams` others besides its neighbours: more than a warp's lanes, several times over."""
    rig = rigs.truss_car(3, speed=15.0, dims=dims)
    b = dict(rig["bodies"][0])
    n = beams if beams < len(b["mass"]) else len(b["mass"]) - 1
    b["ab"] = np.concatenate([b["ab"], np.stack([np.zeros(n, np.uint32), np.arange(1, n + 1, dtype=np.uint32)], 1)])
    for k in ("k", "d", "strength", "deform", "beam_type", "beam_flags"):
        b[k] = np.concatenate([b[k], np.resize(b[k], n)])
    b["k"][-n:] = 2e4
    equal_port(dict(rig, bodies=[b]))


def test_bulk_copies_equal_plain_loads():
    """One car on wheels and shocks (plain loads) and 2,100 of the same in one world (4.07 M beams: bulk copies, the shocks
    and wheels after a block's tiles): each the same bits after two frames."""
    rig = rigs.wheeled_car(shocks=rigs.SHOCK_TYPES[2])
    one = world_from_rig(rig)
    many = world_from_rig(dict(rig, bodies=rig["bodies"] * 2100))
    for _ in range(2):
        one.step_substeps(33)
        many.step_substeps(33)
    want = one.bodies()[0].nodes()
    hs = many.bodies()
    for k in (0, 1, 700, 1399, 2098, 2099):
        got = hs[k].nodes()
        assert np.array_equal(bits(got["p"]), bits(want["p"])) and np.array_equal(bits(got["v"]), bits(want["v"])), k
    assert many.stats()["device_errors"] == 0
    one.close()
    many.close()
