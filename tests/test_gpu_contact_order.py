"""How an island's contacts are ordered - each contact's record made by its own thread and the levels found from lists
by one warp (up to 448), records half a buffer at a time beside the levels' chain (up to 2,048 with the levels from lists,
above in pair order) - against the way of the largest islands, a chunk at a time: the same node states bit for bit in
every substep. Two lattices of one layer pressed face to face, their faces sized for each way."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,hull,low,high", [(4, False, 1, 448), (4, True, 1, 448), (10, False, 449, 2048), (20, False, 2049, 6144)])
def test_contact_order_whole_equals_chunks(side, hull, low, high):
    rig = rigs.crash_pair(3, speed_a=15.0, speed_b=15.0, gap=0.02, hull=hull, dims=(3, side, side))
    a, b = world_from_rig(rig), world_from_rig(rig, contact_whole_max=0)
    peak = before = 0
    for k in range(24):
        a.step_substeps(1)
        b.step_substeps(1)
        now = a.stats()["contacts"]
        peak, before = max(peak, now - before), now
        for i in range(len(rig["bodies"])):
            x, y = a.bodies()[i].nodes(), b.bodies()[i].nodes()
            assert np.array_equal(x["p"].view(np.uint32), y["p"].view(np.uint32)) and np.array_equal(x["v"].view(np.uint32), y["v"].view(np.uint32)), k
    print("peak", peak)
    assert low <= peak <= high  # (the way meant)
    assert a.stats()["device_errors"] == b.stats()["device_errors"] == 0
    a.close()
    b.close()
