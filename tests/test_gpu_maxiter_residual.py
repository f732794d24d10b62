"""A plain FP64 solve that stops by maxiter reports the true residual: with a tolerance that cannot be met the recursion's
residual falls on (0.03 to 0.1 per V-cycle with constant coefficients), the true one stays at its rounding."""
import ctypes

import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, _abi, make_options
from incflo_gb300.projection import array4
from tests.helpers import N, P, cuda, face_fields, nodal_case

pytestmark = pytest.mark.gpu

# |b - A phi| is formed in FP64 from terms of the size of b: on thousands of points its largest value is a good part of a unit of
# rounding, 1.1e-16 |b|. The recursion gets to 1e-19 and less.
FLOOR, MAXITER = 1e-18, 24


@pytest.mark.parametrize("bc", [(P, P, N), (N, N, N)], ids=["periodic-xy", "walls"])
def test_nodal(gpu_lib, bc):
    n = (32, 24, 16)
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, bc, bc, seed=2, sigma_range=(1.0, 1.0))
    proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(n, (0, 0, 0), ext),
                          options=make_options(0, mg_rtol=1e-60, mg_atol=0.0, maxiter=MAXITER))
    proj.setDomainBC(bc, bc)
    plan, lib, st = proj._plan(), _abi.load(), _abi.Stats()
    _abi.check(lib.gbp_nodal_set_sigma(plan.ptr, ctypes.byref(array4(proj.sigma)), 0.0), "set_sigma")
    assert lib.gbp_nodal_project(plan.ptr, ctypes.byref(array4(proj.vel, 1)), None, None, 0,
                                 ctypes.byref(st)) == _abi.GBP_NOT_CONVERGED
    assert st.vcycles == MAXITER and st.status == _abi.GBP_NOT_CONVERGED
    assert FLOOR <= st.final_rel_resid <= 1e-11


@pytest.mark.parametrize("bc", [(P, P, N), (N, N, N)], ids=["periodic-xy", "walls"])
def test_mac(gpu_lib, bc):
    n = (32, 24, 16)
    ext = tuple(v / n[0] for v in n)
    g = O.Grid(n, hi=ext, bclo=bc, bchi=bc)
    rng = np.random.default_rng(2)
    beta = [cuda(np.ones(g.face_shape(d))) for d in range(3)]
    u = [cuda(x) for x in face_fields(g, rng)]
    mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, mg_rtol=1e-60, mg_atol=0.0, maxiter=MAXITER))
    mp.initProjector(beta=beta)
    mp.setDomainBC(bc, bc)
    mp._ensure()
    st = _abi.Stats()
    assert _abi.load().gbp_mac_project(mp.plan.ptr, *(ctypes.byref(array4(x)) for x in u), None, 0,
                                       ctypes.byref(st)) == _abi.GBP_NOT_CONVERGED
    assert st.vcycles == MAXITER and st.status == _abi.GBP_NOT_CONVERGED
    assert FLOOR <= st.final_rel_resid <= 1e-11
