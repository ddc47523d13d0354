"""The tiled stage kernels at the edges of their tiling, against the oracle.

A CTA owns up to 128 vertices of a tile, walks several tiles where a mesh has more than
the grid holds at once, and reads the next tile behind the current one.  The sizes here are
the smallest mesh (one partly filled tile), one tile and a remainder of a few vertices,
and a mesh whose tile count is neither below nor a multiple of any kernel's grid
(148 SMs times 4 to 6 CTAs).  The residual (src/fv.cc:1467-1494) and the state, clock and
dt after three steps (a cold one, then two that take dt from the previous step's last
update) at 1e-12 and 1e-10, the bounds of the parity cases.
"""
import numpy as np
import pytest

from tests.helpers import rel_l2
from tensum_b200 import abi, cases, gpu, preproc
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 12, 300])
@pytest.mark.parametrize("flux,recon,scheme", [("kepes_tecno_roe", "minmod", "ssprk3"), ("kepec", "first", "ssprk3"),
                                               ("kep", "first", "rk4"), ("roe_ec", "first", "ssprk3")])
def test_tile_edges(n, flux, recon, scheme):
    m = cases.kh_mesh(n, 3)
    cfg = dict(flux=flux, reconstruct=recon, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)}, final_time=1e9,
               time_stamps=1, time_scheme=scheme)
    P = abi.Problem(preproc.preprocess(m), cfg)
    prim = cases.kh_ic(m.coords, *cases.kh_coefficients(3))
    s, o = gpu.Solver(P), O.Oracle(P)
    s.set_state(prim)
    o.set_prim(prim)
    assert rel_l2(s.residual(), o.residual()[0]) < 1e-12
    s.set_state(prim)
    o.set_prim(prim)
    a, b = s.step(3), o.step(3)[1]
    assert rel_l2(s.get_state(), o.get_prim()) < 1e-10
    assert np.allclose(a[:2], b[:2], rtol=1e-12, atol=0)
