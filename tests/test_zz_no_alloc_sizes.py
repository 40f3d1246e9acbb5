"""bl_gpu_substep_noalloc on bodies of a few to some thousand nodes - parts of its blocks, nodes of more beams than it loads at
a time (8) and none - twice in a row on the caller's buffers: bitwise the context API's substeps."""
import ctypes as C

import numpy as np
import pytest

from beamlab_b200 import NODE_DTYPE, SoftBody, World, WorldSettings, _lib, rigs
from test_zz_no_alloc import bits, incidence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,lone", [((2, 2, 2), 0), ((4, 4, 4), 1), ((5, 4, 3), 4), ((20, 4, 5), 0), ((40, 7, 9), 3)])
def test_noalloc_sizes_match_the_context_api(dims, lone):
    import torch
    rig = rigs.truss_car(2, speed=20.0, dims=dims)
    body = SoftBody.from_arrays(rig["bodies"][0])
    if lone:  # (the last nodes lose their beams)
        keep = (body.beams["a"] < len(body.nodes) - lone) & (body.beams["b"] < len(body.nodes) - lone)
        body.beams = body.beams[keep].copy()
    body.nodes["v"] += np.random.default_rng(4).uniform(-3.0, 3.0, body.nodes["v"].shape).astype(np.float32)
    body.beams["strength"][::7] = 1e3
    g, dt = (0.0, -9.81, 0.0), 0.0005
    w = World(WorldSettings(gravity=g, dt=dt))
    h = w.add_body(body)
    ptr, inc = incidence(body.beams, len(body.nodes))
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a).copy().view(np.uint8)).cuda()
    dn, db, dp, di = to(body.nodes), to(body.beams), to(ptr), to(inc)
    lib, grav = _lib.lib(), (C.c_float * 3)(*g)
    for step in range(2):
        w.step_substeps(1)
        rc = lib.bl_gpu_substep_noalloc(dn.data_ptr(), len(body.nodes), db.data_ptr(), len(body.beams), dp.data_ptr(), di.data_ptr(), grav, dt, 1, 1, 0,
                                        None)
        torch.cuda.synchronize()
        assert rc == 0
        got = dn.cpu().numpy().view(NODE_DTYPE)
        want = h.nodes()
        assert np.array_equal(bits(got["p"]), bits(want["p"])) and np.array_equal(bits(got["v"]), bits(want["v"])), step
    w.close()
