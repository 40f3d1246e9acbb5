"""A plate rolled up in eight turns, whose factorization takes the minimum-degree order because planes cut it badly
(tests/test_fem_order.py): multifrontal against block column by block column in the reference's order. The solutions differ in
the order of the sums alone, so a node's position in float32 differs by its last place at most."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig

pytestmark = pytest.mark.gpu


def rolled_plate(n, turns):
    rig = rigs.shell_plate(n)
    b = dict(rig["bodies"][0])
    x = b["pos"].astype(np.float64)
    a = 2 * np.pi * turns * (x[:, 0] - x[:, 0].min()) / np.ptp(x[:, 0])
    r = 0.5 / (np.pi * turns) * (1.0 + a / (2 * np.pi * turns))
    b["pos"] = np.stack([r * np.cos(a), 1.0 + r * np.sin(a), x[:, 2]], 1).astype(np.float32)
    return dict(rig, bodies=[b])


def test_rolled_plate_agrees_with_block_columns():
    pos = []
    for dense in (0, 2):
        w = world_from_rig(rolled_plate(63, 8), fem_dense_front=dense, fem_check_residual=True)
        for _ in range(2):
            w.step_substeps(10)
        assert w.fem_stats()["max_residual"] < 1e-11 and w.bodies()[0].state()["fem_failures"] == 0
        pos.append(np.ascontiguousarray(w.bodies()[0].nodes()["p"]).astype(np.float64))
        w.close()
    assert np.isfinite(pos[0]).all() and np.abs(pos[0] - pos[1]).max() <= float(np.spacing(np.float32(np.abs(pos[0]).max()))) + 1e-9
