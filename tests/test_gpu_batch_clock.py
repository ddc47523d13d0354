"""The clocks of a batch: their values, and that reading them costs one copy.

Two levels of 32 and 96 members advance to an output time that takes several steps, one
member of the second made bad by a velocity field that no CFL step tolerates: elapsed
times, output counters and flags must be what each level alone has.  Reading a level's clocks
is a copy and a wait and must cost no more than 1.3 times a small member's state, a kernel, a
copy and a wait; a copy per array made it 2.0 times that.
"""
import time

import numpy as np
import pytest

from tensum_b200 import abi, batch, cases, gpu, preproc

pytestmark = pytest.mark.gpu


def _problem(n, final_time):
    m = cases.kh_mesh(n, 0)
    cfg = dict(flux="kepes_tecno_rusanov", reconstruct="minmod", final_time=final_time, time_stamps=2,
               boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)})
    return abi.Problem(preproc.preprocess(m), cfg), m


def _rows(n, first=0):
    return np.stack([cases.kh_rnd_row(first + s) for s in range(n)])


def _fill(b, level, n, first, m, wild):
    b.set_kh(level, _rows(n, first))
    if wild is not None:
        q = cases.kh_ic_rnd(m.coords, cases.kh_rnd_row(first + wild))
        q[:, 3] *= 1.0e4
        q[:, 2] += 300.0
        b.set_state(level, wild, q)


def _advance(b, instance):
    try:
        b.advance(instance)
    except gpu.TensumError:
        pass


def test_clocks_of_two_levels():
    (A, ma), (B, mb) = _problem(17, 0.02), _problem(33, 0.02)
    both, a, b = batch.Batch([(A, 32), (B, 96)]), batch.Batch([(A, 32)]), batch.Batch([(B, 96)])
    _fill(both, 0, 32, 0, ma, None)
    _fill(both, 1, 96, 40, mb, 41)
    _fill(a, 0, 32, 0, ma, None)
    _fill(b, 0, 96, 40, mb, 41)
    for instance in (1, 2):
        for x in (both, a, b):
            _advance(x, instance)
        for x, y in ((both.clock(0), a.clock(0)), (both.clock(1), b.clock(0))):
            assert all(np.array_equal(p, q) for p, q in zip(x, y))
        elapsed, counter, bad = both.clock(1)
        good = np.arange(96) != 41
        assert bad[41] and not bad[good].any() and not both.clock(0)[2].any()
        assert np.all(counter[good] == instance + 1) and np.all(np.abs(elapsed[good] - 0.01 * instance) < 1e-15)


def test_cost_of_reading_them():
    P, _ = _problem(17, 1e9)
    b = batch.Batch([(P, 32)])
    b.set_kh(0, _rows(32))
    b.advance(1, 1)

    def least(f):
        t = []
        for _ in range(300):
            a = time.perf_counter()
            f()
            t.append(time.perf_counter() - a)
        return min(t)
    clock, state = least(lambda: b.clock(0)), least(lambda: b.get_state(0, 1))
    assert clock < 1.3 * state, (clock, state)
