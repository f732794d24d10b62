"""FP32 solves inside FP64 refinement on the smallest grids, where a V-cycle is an exact solve or nearly: the inner solve
reaches its rounding after a V-cycle or two, and the refinement goes on as fast as on any other grid."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, make_options
from tests.helpers import N, P, cuda, face_fields, nodal_case

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2, 2), (4, 4, 2), (2, 6, 10), (4, 4, 4), (6, 6, 6), (8, 8, 8)]
BCS = {"walls": (N, N, N), "periodic-xy": (P, P, N), "periodic": (P, P, P)}
grids = pytest.mark.parametrize("n", GRIDS, ids=["x".join(map(str, n)) for n in GRIDS])
sides = pytest.mark.parametrize("bc", list(BCS.values()), ids=list(BCS))

# A step of refinement reduces the residual by 1e-5 to 1e-7 with its (at most 5) V-cycles: two steps and a third one of a
# V-cycle or two from 1 to 1e-11
MOST = 12


@grids
@sides
def test_mac(gpu_lib, n, bc):
    g = O.Grid(n, hi=tuple(v / n[0] for v in n), bclo=bc, bchi=bc)
    for seed in range(6):
        rng = np.random.default_rng(seed)
        beta = [np.abs(b) + 0.5 for b in face_fields(g, rng, zero_neumann=False)]
        umac = face_fields(g, rng)
        mp = MacProjector(Geometry(n, (0, 0, 0), tuple(v / n[0] for v in n)), options=make_options(1, precision="mixed"))
        mp.initProjector(beta=[cuda(b) for b in beta])
        mp.setDomainBC(bc, bc)
        mp.setUMAC([cuda(u) for u in umac])
        st = mp.project(rtol=1e-11, atol=0.0)
        assert st["status"] == 0 and st["vcycles"] <= MOST, (seed, st)


@grids
@sides
def test_nodal(gpu_lib, n, bc):
    ext = tuple(v / n[0] for v in n)
    for seed in range(6):
        _, sigma, vel = nodal_case(n, ext, bc, bc, seed=seed)
        proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(n, (0, 0, 0), ext),
                              options=make_options(0, precision="mixed"))
        proj.setDomainBC(bc, bc)
        st = proj.project(rtol=1e-11, atol=0.0)
        assert st["status"] == 0 and st["vcycles"] <= MOST, (seed, st)
