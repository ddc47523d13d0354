"""The surrogate's kernels at the edges of their tiles, chunks and layer widths.

Gradients of batches around the 8 samples a CTA of the training cluster takes at a time and
the 64 of one tile, at the narrowest and widest inputs and outputs, against the float64 CPU
restatement with the bound of test_gpu_mlp.py.  Predictions from and to physical units must
equal the standardised call with numpy's scaling around it bit for bit, at sizes around an
inference tile and a chunk of the pipelined path.
"""
import numpy as np
import pytest

from tensum_b200 import mlp

import mlp_oracle as M  # noqa: E402

pytestmark = pytest.mark.gpu


def _net(din, dout, seed):
    net = mlp.MLP(din, dout, seed=seed)
    rng = np.random.default_rng(seed)
    theta = rng.normal(0.0, 0.25, net.np).astype(np.float32)
    net.params = theta
    return net, theta.astype(np.float64), rng


@pytest.mark.parametrize("din,dout", [(1, 1), (3, 3), (32, 8)])
@pytest.mark.parametrize("n", [1, 7, 9, 63, 65, 129, 520])
def test_gradient_of_ragged_batches(din, dout, n):
    net, theta, rng = _net(din, dout, n)
    X = rng.normal(size=(n, din)).astype(np.float32)
    T = rng.normal(size=(n, dout)).astype(np.float32)
    loss, g = net.loss_grad(X, T)
    rl, rg = M.loss_grad(theta, X.astype(np.float64), T.astype(np.float64), din, dout)
    assert abs(loss - rl) <= 1e-5 * abs(rl)
    assert np.max(np.abs(g - rg)) <= 2e-5 * np.max(np.abs(rg))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("din,dout,n", [(3, 3, 1), (3, 3, 17), (20, 3, 33), (1, 8, 32768), (3, 3, 32769), (32, 1, 100001)])
def test_scaled_prediction_is_the_scaled_call(din, dout, n, precision):
    net, _, rng = _net(din, dout, 5)
    net.xm, net.xs = rng.normal(size=din), rng.uniform(0.5, 2.0, din)
    net.ym, net.ys = rng.normal(size=dout), rng.uniform(0.5, 2.0, dout)
    X = rng.normal(size=(n, din))
    want = net.raw_predict((X - net.xm) / net.xs, precision).astype(np.float64) * net.ys + net.ym
    assert np.array_equal(net.predict(X, precision), want)


def test_scaled_predictions_of_growing_and_shrinking_calls():
    """One net's calls share a workspace that grows; up to 2048 doubles the scaling and the
    rows travel in one copy (678 rows of three inputs and outputs)."""
    net, _, rng = _net(3, 3, 7)
    X = rng.normal(size=(33000, 3))
    net.ym, net.ys = rng.normal(size=3), rng.uniform(0.5, 2.0, 3)
    for n in (1, 256, 257, 678, 679, 5000, 2, 33000, 300):
        net.xm, net.xs = rng.normal(size=3), rng.uniform(0.5, 2.0, 3)
        want = net.raw_predict((X[:n] - net.xm) / net.xs, 1).astype(np.float64) * net.ys + net.ym
        assert np.array_equal(net.predict(X[:n], 1), want), n
