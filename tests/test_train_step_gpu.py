"""The training step's kernels where their split can go wrong: minibatches of one to several parts of the
weight gradient, of more tiles than the blocks take at once, and of more samples than there are parts (two
rounds a part), against the NumPy backward pass of the same bf16 network with the bounds of the one-size
test; and the same step twice giving the same gradient and weights (its sums do not depend on the order
of the blocks)."""
import numpy as np
import pytest

import nsdf_ref as R

pytestmark = pytest.mark.gpu
BLOCKS = {"W1": (R.P_W1, R.P_B1), "b1": (R.P_B1, R.P_W2), "W2": (R.P_W2, R.P_B2), "b2": (R.P_B2, R.P_W3),
          "W3": (R.P_W3, R.P_B3), "b3": (R.P_B3, R.P_W4), "W4": (R.P_W4, R.P_B4), "b4": (R.P_B4, R.P_W5),
          "W5": (R.P_W5, R.P_B5), "b5": (R.P_B5, R.NPARAM)}


@pytest.mark.parametrize("batch", [512, 1536, 10240, 33280])
def test_gradient_of_one_step(ctx, batch):
    from tressfx_gb300.api import NeuralSDF
    lo, hi = np.array([-0.2, 1.3, -0.25]), np.array([0.25, 1.8, 0.2])
    seed, pool = 23, 3001
    rng = np.random.default_rng(batch)
    samples = np.zeros((pool, 8), np.float32)
    samples[:, :3] = rng.uniform(lo, hi, (pool, 3))
    samples[:, 3] = rng.uniform(-3.0, 3.0, pool)
    samples[:, 4:7] = rng.uniform(-0.6, 0.6, (pool, 3))
    samples[:, 7] = rng.uniform(0.5, 1.5, pool)
    runs = []
    for _ in range(2):
        nsdf = NeuralSDF(ctx, lo, hi, cell_size=0.004, pose_scale=1.0 / 0.7, seed=seed, max_samples=4096, max_eval_samples=0)
        p = nsdf.params()
        nsdf.set_samples(0, samples)
        loss = nsdf.train(1, batch=batch, lr=1e-3)
        runs.append((p, loss, nsdf.gradients(), nsdf.params()))
        nsdf.close()
    p, loss, g, after = runs[0]
    want, loss_np = R.train_gradients(p, samples[R.drawn_samples(seed, 1, batch, pool)], R.frame(lo, hi, 1.0 / 0.7))
    assert abs(loss - loss_np / batch) < 0.02 * loss_np / batch
    for name, (a, b) in BLOCKS.items():
        x, y = g[a:b].astype(np.float64), want[a:b].astype(np.float64)
        ny = np.linalg.norm(y)
        rel, cos = np.linalg.norm(x - y) / ny, float(x @ y / (np.linalg.norm(x) * ny))
        assert rel < 0.05 and cos > 0.998, (name, rel, cos)
    assert np.array_equal(g.view(np.uint32), runs[1][2].view(np.uint32))
    assert np.array_equal(after.view(np.uint32), runs[1][3].view(np.uint32))
