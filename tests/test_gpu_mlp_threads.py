"""The network's calls from several host threads on one context: training beside gradients and forwards of other batches, which
share the context's device buffers. Training's weights are what it leaves alone; the others' results are those of one thread."""
import threading

import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def recorded():
    w = world_from_rig(rigs.shell_plate(6))
    w.mlp_init(3)
    w.mlp_record(4096)
    w.step_substeps(20)
    w.synchronize()
    return w


def run_all(calls):
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:  # (a thread's assertion reaches the test)
            errors.append(e)
    ts = [threading.Thread(target=guarded, args=(f,)) for f in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_training_beside_gradients_leaves_the_same_weights():
    rng = np.random.default_rng(2)
    x, t, wt = rng.normal(size=(20000, 36)).astype(np.float32), rng.normal(size=(20000, 12)).astype(np.float32), rng.uniform(size=(20000, 12)).astype(np.float32)
    a, b = recorded(), recorded()
    assert a.mlp_samples() == b.mlp_samples() > 0
    la = a.mlp_train(20, batch=64, lr=1e-3, seed=5)
    lb = []
    run_all([lambda: lb.append(b.mlp_train(20, batch=64, lr=1e-3, seed=5)), lambda: [b.mlp_gradient(x, t, wt) for _ in range(20)]])
    assert lb == [la] and np.array_equal(a.mlp_weights().view(np.uint32), b.mlp_weights().view(np.uint32))
    a.close()
    b.close()


def test_gradients_and_forwards_of_several_threads():
    rng = np.random.default_rng(3)
    w = world_from_rig(rigs.shell_plate(3))
    w.set_mlp_weights(rng.normal(0, 0.2, mo.N_PARAMS).astype(np.float32))
    data = [tuple(rng.normal(size=(n, k)).astype(np.float32) for k in (36, 12, 12)) for n in (33, 5000, 12000)]
    want = [(w.mlp_forward(x), *w.mlp_gradient(x, t, wt)) for x, t, wt in data]

    def check(k):
        x, t, wt = data[k]
        for _ in range(10):
            y, (g, loss) = w.mlp_forward(x), w.mlp_gradient(x, t, wt)
            assert np.array_equal(y, want[k][0]) and np.array_equal(g, want[k][1]) and loss == want[k][2]
    run_all([lambda k=k: check(k) for k in range(3)])
    w.close()
