"""The multifrontal factorization in one launch (fem_dense_front 2) at the sizes where its tiles can go wrong - fronts of
fewer, exactly and one more than the 8 nodes of a tile, right sides alone in a row tile, one front, several trees in one
context - against block column by block column in the reference's order (fem_dense_front 0): the same system solved in
another order of sums, so after 40 substeps the nodes agree to 1e-9 m (the bound the two other orders are held to), and
every solution's residual is at rounding level."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig

pytestmark = pytest.mark.gpu


def ladders(*rails):
    """Ladders of `rails` rungs side by side in one context (a tree of fronts each)."""
    parts = [rigs.frame_ladder(r, origin=(0.0, 1.0, 3.0 * k)) for k, r in enumerate(rails)]
    return dict(parts[0], bodies=[p["bodies"][0] for p in parts])


RIGS = {
    "ladder2": lambda: ladders(2), "ladder4": lambda: ladders(4), "ladder5": lambda: ladders(5),
    "ladders": lambda: ladders(3, 8, 9, 16, 17, 33), "plate1": lambda: rigs.shell_plate(1), "plate2": lambda: rigs.shell_plate(2),
    "plate7": lambda: rigs.shell_plate(7), "plate13": lambda: rigs.shell_plate(13), "plate31": lambda: rigs.shell_plate(31),
    "rails": lambda: rigs.plate_with_rails(15), "shell": lambda: rigs.shell_body(2500)}


@pytest.mark.parametrize("name", list(RIGS))
def test_one_launch_agrees_with_block_columns(name):
    pos = []
    for dense in (0, 2):
        w = world_from_rig(RIGS[name](), fem_dense_front=dense, fem_check_residual=True)
        for _ in range(2):
            w.step_substeps(20)
        st = w.fem_stats()
        assert st["max_residual"] < 1e-11 and (st["fronts"] > 0) == (dense == 2)
        assert all(h.state()["fem_failures"] == 0 for h in w.bodies())
        assert w.stats()["device_errors"] == 0
        pos.append(np.concatenate([np.ascontiguousarray(h.nodes()["p"]) for h in w.bodies()]).astype(np.float64))
        w.close()
    assert np.abs(pos[0] - pos[1]).max() < 1e-9


def test_wide_level_and_many_children():
    """A shell body of 10,000 nodes: its lowest level's fronts go a block each (more than 3,000 tiles' tasks otherwise), and the
    separators above gather many children: every solution's residual is at rounding level."""
    w = world_from_rig(rigs.shell_body(10000), fem_dense_front=2, fem_check_residual=True)
    w.step_substeps(6)
    st = w.fem_stats()
    assert st["max_residual"] < 1e-11 and st["fronts"] > 0 and w.stats()["device_errors"] == 0
    assert all(h.state()["fem_failures"] == 0 for h in w.bodies())
    w.close()
