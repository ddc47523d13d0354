"""Ensemble passes at the edges of their work split.

A warp of the edge pass walks several edges where a batch has more than the grid holds at
once, reading the next one ahead; the smallest mesh leaves most of the first round empty
and an odd multiple of 32 samples half a sample group.  Samples at both ends of a batch
against the FP64 solver with the bound of test_gpu_batch.py, and samples that reach their
output time early keep their state while others step on.
"""
import numpy as np
import pytest

from tests.helpers import rel_l2
from tensum_b200 import abi, batch, cases, gpu, preproc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(5, 32), (65, 32), (65, 96)])
@pytest.mark.parametrize("flux,recon", [("kepes_tecno_rusanov", "minmod"), ("kepec", "first")])
def test_members_at_both_ends_follow_fp64(n, S, flux, recon):
    m = cases.kh_mesh(n, 2)
    cfg = dict(flux=flux, reconstruct=recon, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)},
               final_time=0.01, time_stamps=1, cfl=0.8)
    P = abi.Problem(preproc.preprocess(m), cfg)
    rows = np.stack([cases.kh_rnd_row(s) for s in range(S)])
    b = batch.Batch([(P, S)])
    b.set_kh(0, rows)
    b.advance(1)
    el, _, bad = b.clock(0)
    assert not bad.any() and np.allclose(el, 0.01, rtol=0, atol=1e-15)
    s64 = gpu.Solver(P)
    before = [b.get_state(0, s) for s in (0, S - 1)]
    for s, got in zip((0, S - 1), before):
        s64.set_state(cases.kh_ic_rnd(m.coords, rows[s]))
        s64.advance(1)
        assert rel_l2(got[:, :4], s64.get_state()[:, :4]) <= 2e-6, s
    b.time_steps(3)                      # every sample is past the end: nothing moves
    for s, got in zip((0, S - 1), before):
        assert np.array_equal(b.get_state(0, s), got)


@pytest.mark.parametrize("n,S", [(5, 32), (17, 96), (65, 160)])
@pytest.mark.parametrize("extras", [0, 2, 5, 7])
def test_moments_and_integrals_of_the_states(n, S, extras):
    """One warp per vertex walks the samples: the same sums over get_state's exact copies of the
    FP32 states, to FP64 rounding over S terms; integrals by chunks of the vertices."""
    m = cases.kh_mesh(n, 1)
    cfg = dict(flux="kepec", reconstruct="first", boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)},
               final_time=1.0, time_stamps=1, cfl=0.8)
    P = abi.Problem(preproc.preprocess(m), cfg)
    b = batch.Batch([(P, S)])
    b.set_kh(0, np.stack([cases.kh_rnd_row(s) for s in range(S)]))
    x = np.stack([b.get_state(0, s) for s in range(S)])
    T, p, u, v = (x[:, :, i] for i in range(4))
    gamma, R = float(np.float32(1.4)), 1.0       # the ensemble holds its gas in FP32
    aw = np.array(P.geom.dcarea, dtype=float)
    for st in m.periodic_sets:
        aw[st] /= len(st)
    fm, sm, m2 = b.moments(0, extras=extras)
    rho = p / (R * T)
    more = [rho, np.sqrt(u * u + v * v) / np.sqrt(gamma * p / rho), np.log(p) - gamma * np.log(rho)]
    y = np.concatenate([x] + [more[i][:, :, None] for i in range(3) if extras >> i & 1], axis=2)
    big = np.abs(y).max(axis=(0, 1))
    eps = 2.0 ** -52
    assert fm.shape == y.shape[1:]
    assert np.all(np.abs(fm - y.mean(0)) <= 16 * eps * big)
    assert np.all(np.abs(sm - (y ** 2).sum(0)) <= 16 * S * eps * big ** 2)
    assert np.all(np.abs(m2 - ((y - y.mean(0)) ** 2).sum(0)) <= 16 * S * eps * big ** 2)
    q = np.stack([(0.5 * rho * v * v * aw).sum(1), (0.5 * rho * u * u * aw).sum(1),
                  (-rho * more[2] / (gamma - 1.0) * aw).sum(1)], axis=1)
    mag = np.stack([(0.5 * rho * v * v * aw).sum(1), (0.5 * rho * u * u * aw).sum(1),
                    (np.abs(rho * more[2]) / (gamma - 1.0) * aw).sum(1)], axis=1)
    assert np.all(np.abs(b.integrals(0) - q) <= 64 * m.n_vertex * eps * mag + 64 * eps)
