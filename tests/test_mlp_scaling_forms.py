"""Every form of input and output scaling that numpy broadcasts is accepted by MLP.predict.

The library is replaced by one that evaluates y = x_0 + x_1 + ... for each output, so the
expected value is numpy's own expression around it, bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

from tensum_b200 import mlp

DIN, DOUT = 3, 2


def _at(ptr, shape, ct):
    return np.ctypeslib.as_array((ct * int(np.prod(shape))).from_address(ptr)).reshape(shape)


class _Sums:
    def tg_mlp_predict(self, h, X, n, Y, precision, on_device):
        _at(Y, (n, DOUT), C.c_float)[:] = _at(X, (n, DIN), C.c_float).sum(axis=1, keepdims=True)
        return 0

    def tg_mlp_predict_scaled(self, h, X, n, xm, xs, ym, ys, Y, precision):
        v = [_at(p, (k,), C.c_double) for p, k in ((xm, DIN), (xs, DIN), (ym, DOUT), (ys, DOUT))]
        x = ((_at(X, (n, DIN), C.c_double) - v[0]) / v[1]).astype(np.float32)
        _at(Y, (n, DOUT), C.c_double)[:] = x.sum(axis=1, keepdims=True).astype(np.float64) * v[3] + v[2]
        return 0


FORMS = {
    "vectors": lambda r, n, k: r.uniform(0.5, 2.0, k),
    "scalar": lambda r, n, k: 1.5,
    "one": lambda r, n, k: r.uniform(0.5, 2.0, 1),
    "row": lambda r, n, k: r.uniform(0.5, 2.0, (1, k)),
    "per_sample": lambda r, n, k: r.uniform(0.5, 2.0, (n, k)),
    "column": lambda r, n, k: r.uniform(0.5, 2.0, (n, 1)),
    "strided": lambda r, n, k: r.uniform(0.5, 2.0, 2 * k)[::2],
    "list": lambda r, n, k: list(r.uniform(0.5, 2.0, k)),
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n", [1, 5])
def test_forms(form, n):
    r = np.random.default_rng(4)
    net = object.__new__(mlp.MLP)
    net.L, net.h, net.din, net.dout = _Sums(), None, DIN, DOUT
    f = FORMS[form]
    net.xm, net.xs, net.ym, net.ys = f(r, n, DIN), f(r, n, DIN), f(r, n, DOUT), f(r, n, DOUT)
    X = r.normal(size=(n, DIN))
    x = ((X - net.xm) / net.xs).astype(np.float32)
    y = np.repeat(x.sum(axis=1, keepdims=True), DOUT, axis=1)
    assert np.array_equal(net.predict(X), y.astype(np.float64) * net.ys + net.ym)
