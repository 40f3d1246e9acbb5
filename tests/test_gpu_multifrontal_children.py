"""Fronts of many children (fem_dense_front 2): a star of members, its hub carried by `arms` arms of six whose outer ends are
anchored - every arm a subtree of its own, so the hub's front gathers nearly as many children, 16 at a time - against
block column by block column in the reference's order (fem_dense_front 0): after 40 substeps the nodes agree to 1e-9 m and
every solution's residual is at rounding level."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig

pytestmark = pytest.mark.gpu


def star(arms, length=6, seed=1):
    rig = rigs.frame_ladder(2)
    b = dict(rig["bodies"][0])
    gen = np.random.default_rng(seed)
    pos, members = [(0.0, 1.0, 0.0)], []
    for _ in range(arms):
        d = gen.normal(size=3)
        d /= np.linalg.norm(d)
        for k in range(length):
            members.append((0 if k == 0 else len(pos) - 1, len(pos)))
            pos.append(tuple(np.array((0.0, 1.0, 0.0)) + 0.25 * (k + 1) * d))
    n, m = len(pos), len(members)
    flags = np.zeros(n, np.uint16)
    flags[length::length] = rigs.NF_FIXED
    b.update({"pos": np.asarray(pos, np.float32), "vel": np.zeros((n, 3), np.float32), "mass": np.full(n, 0.6, np.float32), "node_flags": flags,
              "friction": np.ones(n, np.float32), "radius": np.zeros(n, np.float32), "fem_members": np.asarray(members, np.uint32),
              "member_section": np.zeros(m, np.uint16), "member_ends": np.zeros((m, 2), np.uint8), "member_mass": np.zeros(m, np.float32),
              "loads": [(0, (100.0, -500.0, 50.0))]})
    return dict(rig, bodies=[b], name=f"star(arms={arms})")


@pytest.mark.parametrize("arms", (15, 16, 17, 40))
def test_many_children_agree_with_block_columns(arms):
    pos = []
    for dense in (0, 2):
        w = world_from_rig(star(arms), fem_dense_front=dense, fem_check_residual=True)
        for _ in range(2):
            w.step_substeps(20)
        st = w.fem_stats()
        assert st["max_residual"] < 1e-11 and (st["fronts"] > 0) == (dense == 2)
        assert w.bodies()[0].state()["fem_failures"] == 0 and w.stats()["device_errors"] == 0
        pos.append(np.ascontiguousarray(w.bodies()[0].nodes()["p"]).astype(np.float64))
        w.close()
    assert np.abs(pos[0] - pos[1]).max() < 1e-9 and np.abs(pos[0][0] - (0.0, 1.0, 0.0)).max() > 1e-7  # (the hub moves)
