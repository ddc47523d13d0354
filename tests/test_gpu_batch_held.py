"""A level whose samples are all held beside one that still advances.

In a multilevel batch the coarse level reaches the output time first.  From then on its
members keep their state (src/fv.cc:2273-2275): the finer level's result must be that of
the same level alone, bit for bit, and the held one's must not move.  Nor may the held level
cost what an advancing one does.  Per vertex, sample and stage an advancing level moves
about 47 words between the passes (13 of state and gradients in the edge pass, 12 of fluxes
written and read, the rest in the gradient, update and time-step passes); a held one only
the 10 words of its state that the update carries over, 0.21 of that.  With the edge pass's
rows read all the same it would be 23 words, 0.49; the bound is the middle.
"""
import numpy as np
import pytest

from tensum_b200 import abi, batch, cases, preproc

pytestmark = pytest.mark.gpu


def _problem(n, final_time, flux="kepes_tecno_rusanov", recon="minmod"):
    m = cases.kh_mesh(n, 0)
    cfg = dict(flux=flux, reconstruct=recon, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)},
               final_time=final_time, time_stamps=1)
    return abi.Problem(preproc.preprocess(m), cfg)


def _rows(n, first=0):
    return np.stack([cases.kh_rnd_row(first + s) for s in range(n)])


def _dt(P):
    b = batch.Batch([(P, 32)])
    b.set_kh(0, _rows(32))
    b.advance(1, 1)
    return float(b.clock(0)[0].max())


@pytest.mark.parametrize("flux,recon", [("kepes_tecno_rusanov", "minmod"), ("kepes_tecno_roe", "first"), ("kepec", "first")])
@pytest.mark.parametrize("coarse,fine", [(64, 32), (96, 32), (32, 160)])
def test_held_level_beside_an_advancing_one(flux, recon, coarse, fine):
    T = 3.5 * _dt(_problem(17, 1e9, flux, recon))
    P, F = _problem(17, T, flux, recon), _problem(65, T, flux, recon)
    both, alone, low = batch.Batch([(P, coarse), (F, fine)]), batch.Batch([(F, fine)]), batch.Batch([(P, coarse)])
    both.set_kh(0, _rows(coarse))
    low.set_kh(0, _rows(coarse))
    both.set_kh(1, _rows(fine, 50))
    alone.set_kh(0, _rows(fine, 50))
    low.advance(1)
    n = 0
    while (both.clock(1)[0] < T).any():
        both.advance(1, 3)
        n += 3
    assert n >= 9                                  # the coarse level was held for most of them
    alone.advance(1)
    for s in (0, fine // 2, fine - 1):
        assert np.array_equal(both.get_state(1, s), alone.get_state(0, s))
    for s in (0, coarse // 2, coarse - 1):
        assert np.array_equal(both.get_state(0, s), low.get_state(0, s))


def test_a_held_level_costs_little():
    S, s = 768, 32
    T = 12.0 * _dt(_problem(129, 1e9))
    P, F = _problem(129, T), _problem(257, T)
    both, alone = batch.Batch([(P, S), (F, s)]), batch.Batch([(F, s)])
    both.set_kh(0, _rows(S))
    both.set_kh(1, _rows(s, 50))
    alone.set_kh(0, _rows(s, 50))
    for b in (both, alone):
        b.time_steps(1)
    active = min(both.time_steps(1) for _ in range(4))
    small = min(alone.time_steps(1) for _ in range(4))
    while (both.clock(0)[0] < T).any():
        both.advance(1, 1)
    assert not (both.clock(1)[0] >= T).any()
    held = min(both.time_steps(1) for _ in range(4))
    assert held - small < 0.35 * (active - small), (held, small, active)
