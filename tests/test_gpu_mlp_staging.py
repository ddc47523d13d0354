"""When a network's predictions are staged through pinned memory, and that it changes nothing.

A network's first call of 100 000 rows must cost no more than one and a half times the same
evaluation with the scaling in numpy around `raw_predict`, which stages nothing: page-locked
memory alone took three times that long.  The least of several new networks stands for each.
Once calls have moved enough, they are staged in chunks; predictions must equal the standardised
call bit for bit at sizes around one, two and all four lanes' chunks (21845 rows of three inputs
and outputs in 1 MiB) and after a call that makes the lanes larger.
"""
import time

import numpy as np
import pytest

from tensum_b200 import mlp

pytestmark = pytest.mark.gpu


def _net(din, dout, seed=3):
    net = mlp.MLP(din, dout, seed=seed)
    rng = np.random.default_rng(seed)
    net.params = rng.normal(0.0, 0.25, net.np).astype(np.float32)
    net.xm, net.xs = rng.normal(size=din), rng.uniform(0.5, 2.0, din)
    net.ym, net.ys = rng.normal(size=dout), rng.uniform(0.5, 2.0, dout)
    return net, rng


def _plain(net, X, precision):
    return net.raw_predict((X - net.xm) / net.xs, precision).astype(np.float64) * net.ys + net.ym


def _ms(f):
    t = time.perf_counter()
    f()
    return (time.perf_counter() - t) * 1e3


@pytest.mark.parametrize("din,rows", [(3, 100000), (32, 40000)])
def test_a_first_large_prediction_pays_for_no_later_one(din, rows):
    first, plain = [], []
    X = np.random.default_rng(1).normal(size=(rows, din))
    for i in range(8):
        a, _ = _net(din, 3, i)
        b, _ = _net(din, 3, i)
        first.append(_ms(lambda: a.predict(X)))
        plain.append(_ms(lambda: _plain(b, X, 1)))
    assert min(first) < 1.5 * min(plain), (first, plain)


@pytest.mark.parametrize("precision", [0, 1])
def test_staged_predictions_are_the_plain_ones(precision):
    net, rng = _net(3, 3)
    X = rng.normal(size=(2100000, 3))
    assert np.array_equal(net.predict(X[:400000], precision), _plain(net, X[:400000], precision))
    for n in (32769, 43690, 43691, 87379, 87380, 87381, 2100000, 32769, 131071, 200000):
        assert np.array_equal(net.predict(X[-n:], precision), _plain(net, X[-n:], precision)), n
