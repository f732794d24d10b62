"""Singular systems run on below their rounding: the constant that the rounding errors of the residual sum up to stays in it, and
nothing may grow from it. A tolerance that cannot be met ends at maxiter with the solution of a solve that met its own."""
import ctypes

import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, _abi, eb, make_options
from incflo_gb300.projection import array4
from tests.helpers import N, P, cuda, face_fields, nodal_case, rel_l2

pytestmark = pytest.mark.gpu

N3 = (32, 24, 16)
EXT = tuple(v / N3[0] for v in N3)
BCS = [(P, P, N), (P, P, P), (N, N, N)]
sides = pytest.mark.parametrize("bc", BCS, ids=["periodic-xy", "periodic", "walls"])
FORMS = [dict(precision="fp64", maxiter=40), dict(precision="mixed", maxiter=12),
         dict(precision="mixed", maxiter=12, ir_inner_cycles=20)]
forms = pytest.mark.parametrize("form", FORMS, ids=["fp64", "mixed", "mixed-20"])


def _nodal(bc, **opt):
    _, sigma, vel = nodal_case(N3, EXT, bc, bc, seed=2, sigma_range=(1.0, 1.0))
    proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(N3, (0, 0, 0), EXT), options=make_options(0, mg_atol=0.0, **opt))
    proj.setDomainBC(bc, bc)
    plan, lib, st = proj._plan(), _abi.load(), _abi.Stats()
    phi = cuda(np.zeros([v + 1 for v in reversed(N3)]))
    _abi.check(lib.gbp_nodal_set_sigma(plan.ptr, ctypes.byref(array4(proj.sigma)), 0.0), "set_sigma")
    rc = lib.gbp_nodal_project(plan.ptr, ctypes.byref(array4(proj.vel, 1)), ctypes.byref(array4(phi)), None, 0, ctypes.byref(st))
    return rc, st, phi.cpu().numpy()


def _mac(bc, cut=False, **opt):
    g = O.Grid(N3, hi=EXT, bclo=bc, bchi=bc)
    rng = np.random.default_rng(2)
    beta = [cuda(np.ones(g.face_shape(d))) for d in range(3)]
    u = [cuda(x) for x in face_fields(g, rng)]
    mp = MacProjector(Geometry(N3, (0, 0, 0), EXT), options=make_options(1, mg_atol=0.0, **opt))
    mp.initProjector(beta=beta)
    mp.setDomainBC(bc, bc)
    if cut:
        geo = eb.cylinder(N3, (0, 0, 0), EXT, (0.5, 0.4, 0.0), 0.2)
        mp.setEB(cuda(geo["vfrac"]), [cuda(geo[k]) for k in ("apx", "apy", "apz")],
                 [cuda(np.moveaxis(geo[k], -1, 0)) for k in ("fcx", "fcy", "fcz")])
    mp._ensure()
    st, phi = _abi.Stats(), cuda(np.zeros(g.cell_shape))
    rc = _abi.load().gbp_mac_project(mp.plan.ptr, *(ctypes.byref(array4(x)) for x in u), ctypes.byref(array4(phi)), 0,
                                     ctypes.byref(st))
    return rc, st, phi.cpu().numpy()


def _check(solve, form):
    rc, st, phi = solve(mg_rtol=1e-60, **form)
    assert rc == _abi.GBP_NOT_CONVERGED and st.final_rel_resid <= 1e-13  # rounding, 1e-16, with three digits to spare
    rc, st, ref = solve(mg_rtol=1e-12, precision="fp64")
    assert rc == _abi.GBP_OK and rel_l2(phi, ref) <= 1e-9


@forms
@sides
def test_nodal(gpu_lib, bc, form):
    _check(lambda **o: _nodal(bc, **o), form)


@forms
@sides
def test_mac(gpu_lib, bc, form):
    _check(lambda **o: _mac(bc, **o), form)


@forms
def test_mac_cut_cells(gpu_lib, form):
    _check(lambda **o: _mac((P, N, P), cut=True, **o), form)


@pytest.mark.parametrize("solve", [_nodal, _mac], ids=["nodal", "mac"])
@sides
def test_strong_vcycles(gpu_lib, bc, solve):
    """Eight sweeps before and after: an FP32 inner solve goes below its rounding with its 5 V-cycles, and the refinement still
    gains what it delivers (1e-6 and more, as with two sweeps): two steps from 1 to 1e-11."""
    rc, st, _ = solve(bc, precision="mixed", mg_rtol=1e-11, num_pre_smooth=8, num_post_smooth=8)
    assert rc == _abi.GBP_OK and st.outer_iters <= 3
