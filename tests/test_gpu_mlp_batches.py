"""The network's kernels over batch sizes: part of a tile of 32 samples, whole tiles, and more tiles than blocks (296
for the gradient, 592 for the forward: a block's sums then run over several tiles), against the CPU restatement. The
bounds are those of the smaller batches: FP32 sums, and now and then an activation on the other side of a BF16 rounding
boundary."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1, 31, 32, 33, 296 * 32, 296 * 32 + 1, 592 * 32 + 17))
def test_mlp_batch_sizes(n):
    w = world_from_rig(rigs.shell_plate(3))
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.2, mo.N_PARAMS).astype(np.float32)
    w.set_mlp_weights(p)
    x = rng.normal(0, 1, (n, 36)).astype(np.float32)
    t = rng.normal(0, 1, (n, 12)).astype(np.float32)
    wt = rng.uniform(0, 1, (n, 12)).astype(np.float32)
    y, (yo, _) = w.mlp_forward(x), mo.forward(p, x)
    err, scale = np.abs(y - yo), np.max(np.abs(yo))
    assert np.max(err) <= 1e-5 + 3e-3 * scale
    assert np.quantile(err, 0.99) <= 1e-5 + 1e-4 * scale
    g, loss = w.mlp_gradient(x, t, wt)
    lo, go = mo.loss_and_grad(p, x, t, wt)
    err, scale = np.abs(g - go), np.max(np.abs(go))
    assert np.max(err) <= 3e-3 * scale
    assert abs(loss - lo) <= 1e-3 * lo
    w.close()
