"""The network's fused training kernels at the edges of their tiles (GPU): the
output layer with the loss in its epilogue, the weight gradients with Adam in
theirs (both BF16 layouts of the new weights), the bias updates, and both tile
widths of the forward and backward GEMMs.

One Adam step from zero moments moves a weight by lr*g/(|g| + eps'), computed
here in float64 from the library's own gradient; FP32 rounding of the moments,
the root and the quotient stays below 1e-6 of the step, of the weight below
2^-24 of it.  Networks are compared with the CPU reference at the bars of
test_gpu_mlp.py (forward 5e-3, gradient 2e-2)."""
import numpy as np
import pytest

import mlp_ref
from dgbgk.warmstart import MLP

pytestmark = pytest.mark.gpu


def net_and_data(n_in, width, depth, n_out, batch, seed=5):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (batch, n_in)).astype(np.float32)
    t = rng.normal(0, 1, (batch, n_out)).astype(np.float32)
    return MLP(n_in, width, depth, n_out, batch, seed=seed), x, t


@pytest.mark.parametrize("n_in,width,depth,n_out,batch", [
    (1, 128, 1, 128, 128), (3, 128, 2, 640, 256), (64, 256, 2, 4096, 128), (5, 512, 3, 9472, 128),
    (3, 256, 9, 256, 128), (3, 384, 2, 18944, 256)])
def test_adam_step(n_in, width, depth, n_out, batch):
    m, x, t = net_and_data(n_in, width, depth, n_out, batch)
    p0 = m.get_params()
    loss, g = m.gradient(x, t)
    m.set_data(x, t)
    lr = 1e-3
    hist = m.train(1, lr=lr, seed=1)
    assert abs(hist[0] - loss) <= 1e-6 * loss
    p1 = m.get_params()
    g64 = g.astype(np.float64)
    want = p0.astype(np.float64) - lr * g64 / (np.abs(g64) + 1e-8)
    # the columns past n_in of the input layer and their moments stay as they are
    w0 = np.zeros(p0.size, dtype=bool)
    w0[:64 * width].reshape(width, 64)[:, n_in:] = True
    want[w0] = p0[w0]
    # the two gradients differ by the order of the rows of the batch only where FP32 sums do
    err = np.abs(p1 - want)
    close = np.abs(g64) > 1e-4 * np.abs(g64).max()
    assert np.all(err[close | w0] <= 1e-2 * lr)
    assert np.median(err) <= 1e-5 * lr + 2.0 ** -24 * np.abs(p0).max()
    # the new weights in both layouts: forward, and the gradient through W^T
    y = m.forward(x)
    ref, _ = mlp_ref.forward(p1, x, n_in, width, depth, n_out, bf16_points=True)
    assert np.linalg.norm(y - ref) <= 5e-3 * np.linalg.norm(ref)
    if n_out <= 4096:
        l1, g1 = m.gradient(x, t)
        rl, rg = mlp_ref.loss_and_grad(p1, x, t, n_in, width, depth, n_out)
        assert abs(l1 - rl) <= 1e-3 * rl
        assert np.linalg.norm(g1 - rg) <= 2e-2 * np.linalg.norm(rg)
    m.close()
