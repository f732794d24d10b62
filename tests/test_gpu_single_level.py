"""Hierarchies of one level (a direction that does not coarsen): their V-cycle is the coarsest level's solve. A dense inverse
leaves rounding, so a plain solve takes one and a mixed one an FP32 rounding (1e-7) per step, two from 1 to 1e-11 (three with its
error constants); conjugate gradients to bottom_rtol = 1e-4 three to four."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, make_options
from tests.helpers import D, N, P, cuda, face_fields, nodal_case, rel_l2, unique_nodes

pytestmark = pytest.mark.gpu

# unknowns of the nodal and the MAC system: up to 112 (dense) and beyond
CASES = [((2, 2, 2), (N, N, N), (N, N, N), True, True), ((2, 2, 2), (P, P, N), (P, P, N), True, True),
         ((4, 4, 2), (P, P, P), (P, P, P), True, True), ((4, 2, 6), (N, D, P), (N, N, P), True, True),
         ((2, 32, 2), (N, N, N), (N, N, N), False, False), ((2, 6, 10), (P, N, D), (P, N, N), False, False)]
cases = pytest.mark.parametrize("n,lo,hi,dense_nodal,dense_mac", CASES,
                                ids=["x".join(map(str, c[0])) + "-" + "".join(map(str, c[1])) for c in CASES])


def _most(dense, precision):
    return (1 if precision == "fp64" else 3) if dense else 4


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@cases
def test_nodal(gpu_lib, n, lo, hi, dense_nodal, dense_mac, precision):
    ext = tuple(v / n[0] for v in n)
    g, sigma, vel = nodal_case(n, ext, lo, hi, seed=8)
    _, phi_or, _, _ = O.nodal_project(g, sigma, vel, rtol=1e-13)
    proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(n, (0, 0, 0), ext), options=make_options(0, precision=precision))
    proj.setDomainBC(lo, hi)
    st = proj.project(rtol=1e-11, atol=0.0)
    assert st["status"] == 0 and st["vcycles"] <= _most(dense_nodal, precision), st
    assert rel_l2(unique_nodes(g, proj.getPhi().cpu().numpy()), phi_or) <= 1e-9


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@cases
def test_mac(gpu_lib, n, lo, hi, dense_nodal, dense_mac, precision):
    ext = tuple(v / n[0] for v in n)
    g = O.Grid(n, hi=ext, bclo=lo, bchi=hi)
    rng = np.random.default_rng(8)
    beta = [np.abs(b) + 0.5 for b in face_fields(g, rng, zero_neumann=False)]
    umac = face_fields(g, rng)
    _, phi_or, _ = O.mac_project(g, beta, umac, rtol=1e-13)
    mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, precision=precision))
    mp.initProjector(beta=[cuda(b) for b in beta])
    mp.setDomainBC(lo, hi)
    mp.setUMAC([cuda(u) for u in umac])
    phi = cuda(np.zeros(g.cell_shape))
    st = mp.project(rtol=1e-11, atol=0.0, phi=phi, phi_guess=False)
    assert st["status"] == 0 and st["vcycles"] <= _most(dense_mac, precision), st
    assert rel_l2(phi.cpu().numpy(), phi_or) <= 1e-9
