"""The first steps of a new handle hide the capture of the eight-step run.

A first call of 32 steps makes that run, one of 24 steps does not.  Made ahead of the steps, its
capture costs the first call 0.14 ms on the 65 x 65 mesh; made behind single steps that are
still running, 0.02.  The bound on what the first call of 32 steps costs over a later one, more
than that of 24 steps does, lies between; the least of several new handles stands for each.
"""
import time

import numpy as np
import pytest

from tensum_b200 import abi, cases, gpu, preproc

pytestmark = pytest.mark.gpu


def test_the_capture_is_hidden():
    m = cases.kh_mesh(65, 0)
    P = abi.Problem(preproc.preprocess(m), dict(flux="kepes_tecno_roe", reconstruct="minmod", final_time=1e9,
                                                time_stamps=1, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)}))
    prim = cases.kh_ic(m.coords, *cases.kh_coefficients(3))

    def ms(s, n):
        t = time.perf_counter()
        s.step(n)
        return (time.perf_counter() - t) * 1e3

    def extra(n):
        first, later = [], []
        for _ in range(12):
            s = gpu.Solver(P)
            s.set_state(prim)
            first.append(ms(s, n))
            later += [ms(s, n) for _ in range(3)]
            s.close()
        return min(first) - min(later)
    extra(32)
    assert extra(32) - extra(24) < 0.08, (extra(32), extra(24))


def test_the_capture_is_hidden_in_a_later_call():
    """A handle's second sample makes the run, which a first one of 24 steps did not: behind eight
    steps of 32 us it costs nothing, ahead of them the 0.14 ms.  The same bound."""
    m = cases.kh_mesh(65, 0)
    P = abi.Problem(preproc.preprocess(m), dict(flux="kepes_tecno_roe", reconstruct="minmod", final_time=1e9,
                                                time_stamps=1, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)}))
    prim = cases.kh_ic(m.coords, *cases.kh_coefficients(3))

    def sample(s, n):
        s.set_state(prim)
        t = time.perf_counter()
        s.step(n)
        return (time.perf_counter() - t) * 1e3

    second, later = [], []
    for k in range(13):
        s = gpu.Solver(P)
        sample(s, 24)
        t = [sample(s, 16) for _ in range(4)]
        if k > 0:                                    # the first one of a process takes 4 ms
            second.append(t[0])
            later += t[1:]
        s.close()
    assert min(second) - min(later) < 0.08, (min(second), min(later))
