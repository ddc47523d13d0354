"""Meshes on which every pass of a step walks several tiles per CTA, against the oracle.

The tile size follows the mesh, so a mesh takes more than one round of CTAs only past some
size: of 400 x 400 vertices the central fluxes make 1667 tiles of 96 for 888 CTAs (740 in the
last update), TeCNO-Roe 1250 of 128 for 592.  Neither is a multiple of its grid, so CTAs that
walk one tile fewer than others, the other half of the double-buffered lists and the restaged
normals are all taken in each mode: the residual, a step's earlier updates and its last one.
The residual (src/fv.cc:1467-1494) and the state, clock and dt after three steps at 1e-12 and
1e-10, the bounds of the parity cases.
"""
import numpy as np
import pytest

from tests.helpers import rel_l2
from tensum_b200 import abi, cases, gpu, preproc
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    m = cases.kh_mesh(400, 3)
    return m, preproc.preprocess(m)


@pytest.mark.parametrize("flux,recon,scheme", [("kepes_tecno_roe", "minmod", "ssprk3"), ("kepec", "first", "ssprk3"),
                                               ("kep", "first", "rk4"), ("roe_ec", "first", "ssprk3")])
def test_several_tiles_per_block(mesh, flux, recon, scheme):
    m, pre = mesh
    cfg = dict(flux=flux, reconstruct=recon, boundary={t: ("periodic", {}) for t in (1, 2, 3, 4)}, final_time=1e9,
               time_stamps=1, time_scheme=scheme)
    P = abi.Problem(pre, cfg)
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
