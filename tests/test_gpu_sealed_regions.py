"""Cut-cell MAC projections whose fluid falls into two regions with covered cells between them: each closed region has its own
constant, and the coarsest operator a null space of two dimensions. Both precisions reach the tolerance as on one region (9 to
14 V-cycles; 24 allowed), and the divergence is gone from either side."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, make_options
from tests.helpers import D, N, P, cuda, face_fields

pytestmark = pytest.mark.gpu

BCS = {"closed": ((N, P, N), (N, P, N)), "one-open": ((N, N, N), (D, N, N))}
CASES = [((32, 16, 16), (15, 17)), ((32, 16, 16), (14, 18)), ((48, 24, 40), (22, 26)), ((48, 24, 40), (12, 15)),
         ((64, 32, 32), (16, 19))]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bc", list(BCS.values()), ids=list(BCS))
@pytest.mark.parametrize("n,wall", CASES, ids=["x".join(map(str, c[0])) + f"-{c[1][0]}" for c in CASES])
def test_two_regions(gpu_lib, n, wall, bc, precision):
    ext = tuple(v / n[1] for v in n)
    g = O.Grid(n, hi=ext, bclo=bc[0], bchi=bc[1])
    a, b = wall  # covered cells a .. b - 1 along x
    vf = np.ones(g.cell_shape)
    vf[:, :, a:b] = 0.0
    ap = [np.ones(g.face_shape(d)) for d in range(3)]
    ap[0][:, :, a:b + 1] = 0.0
    ap[1][:, :, a:b] = 0.0
    ap[2][:, :, a:b] = 0.0
    u = face_fields(g, np.random.default_rng(3))
    u[0][:, :, a:b + 1] = 0.0
    mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, precision=precision))
    mp.initProjector(beta=1.0)
    mp.setDomainBC(*bc)
    mp.setEB(cuda(vf), [cuda(x) for x in ap], [cuda(np.zeros((2,) + x.shape)) for x in ap])
    ut = [cuda(x) for x in u]
    mp.setUMAC(ut)
    st = mp.project(rtol=1e-11, atol=0.0, phi=cuda(np.zeros(g.cell_shape)), phi_guess=False)
    assert st["status"] == 0 and st["vcycles"] <= 24

    def div(f):
        d = sum(np.diff(f[k] * ap[k], axis=2 - k) / (ext[k] / n[k]) for k in range(3))
        return np.abs(d[vf > 0]).max()

    assert div([x.cpu().numpy() for x in ut]) <= 1e-9 * div(u)
