"""Bodies without nodes (bl_gpu_add_body takes them): a world of them alone steps, as a graph and launch by launch, and beside
a truss they change nothing of it."""
import numpy as np
import pytest

from beamlab_b200 import SoftBody, rigs, world_from_rig

pytestmark = pytest.mark.gpu


def empty():
    body = SoftBody("empty")
    body.finalize()
    return body


@pytest.mark.parametrize("graphs", [True, False])
def test_bodies_without_nodes_step(graphs):
    w = world_from_rig({"settings": {}, "statics": {}, "bodies": []}, graphs=graphs)
    w.add_body(empty())
    for _ in range(2):
        w.step_substeps(3)
    w.synchronize()
    assert w.stats()["device_errors"] == 0 and w.stats()["total_substeps"] == 6
    w.close()


def test_an_empty_body_beside_a_truss():
    rig = rigs.truss_car(3, dims=(4, 4, 2))
    a, b = world_from_rig(rig), world_from_rig(rig)
    b.add_body(empty())
    for w in (a, b):
        w.step_substeps(20)
    x, y = a.bodies()[0].nodes(), b.bodies()[0].nodes()
    assert np.array_equal(x["p"].view(np.uint32), y["p"].view(np.uint32))
    a.close()
    b.close()
