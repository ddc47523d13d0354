"""New gas constants on a handle that holds a state.

tg_update_parameters leaves the state -- temperature, pressure, velocity -- as it is.  The
next steps must be those of a handle created with the new constants and given that state:
the density the fluxes and the update read is p / (R T) of the new gas, not of the gas the
state came with.  The same bits, as for any other parameter.
"""
import numpy as np
import pytest

from tensum_b200 import abi, cases, gpu, preproc

pytestmark = pytest.mark.gpu

GASES = [dict(gas_const=1.25), dict(gamma=1.3), dict(gas_const=0.7, gamma=1.6)]


def _cfg(flux, recon, **gas):
    return dict(flux=flux, reconstruct=recon, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)}, final_time=1e9,
                time_stamps=1, **gas)


@pytest.mark.parametrize("gas", GASES)
@pytest.mark.parametrize("flux,recon", [("kepes_tecno_roe", "minmod"), ("kepec", "first"), ("roe_ec", "first")])
@pytest.mark.parametrize("steps", [0, 5])
def test_a_state_keeps_its_primitive_variables(flux, recon, gas, steps):
    m = cases.kh_mesh(33, 2)
    g = preproc.preprocess(m)
    a = gpu.Solver(abi.Problem(g, _cfg(flux, recon)))
    a.set_state(cases.kh_ic(m.coords, *cases.kh_coefficients(2)))
    if steps:
        a.step(steps)
    state = a.get_state()
    Q = abi.Problem(g, _cfg(flux, recon, **gas))
    a.update_parameters(Q)
    assert np.array_equal(a.get_state(), state)
    b = gpu.Solver(Q)
    b.set_state(state)
    assert np.array_equal(a.residual(), b.residual())
    assert np.array_equal(a.gradients(), b.gradients())
    ia, ib = a.step(4), b.step(4)
    assert ia[1] == ib[1]                          # the last dt
    assert np.array_equal(a.get_state(), b.get_state())
