"""Cut-cell MAC projections whose operator is far from symmetric: the centroids of all cut faces lie off the face centre by 0.4
of a face, on one side. Conjugate gradients stagnate on it; stationary V-cycles take 26 from 1 to 1e-11 on these grids, and the
solve finds them after a window or two of V-cycles without success."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, eb, make_options
from oracle.eb_mac import EBMac
from tests.helpers import D, N, P, cuda, face_fields, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bc", [((N, N, P), (D, N, P)), ((P, N, P), (P, N, P))], ids=["outflow", "singular"])
def test_skewed_face_centroids(gpu_lib, bc, precision):
    n, ext = (64, 16, 8), (4.0, 1.0, 0.5)
    geo = dict(eb.cylinder(n, (0, 0, 0), ext, (1.03, 0.47, 0.0), 0.33))
    for k in ("fcx", "fcy", "fcz"):
        cut = np.abs(geo[k]).sum(-1, keepdims=True) > 0
        geo[k] = np.where(cut, 0.4, 0.0) * np.ones(geo[k].shape)
    g = O.Grid(n, hi=ext, bclo=bc[0], bchi=bc[1])
    rng = np.random.default_rng(4)
    beta = [0.5 + np.abs(b) for b in face_fields(g, rng, zero_neumann=False)]
    umac = face_fields(g, rng)
    mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, precision=precision, maxiter=100))
    mp.initProjector(beta=[cuda(b) for b in beta])
    mp.setDomainBC(*bc)
    mp.setEB(cuda(geo["vfrac"]), [cuda(geo[k]) for k in ("apx", "apy", "apz")],
             [cuda(np.moveaxis(geo[k], -1, 0)) for k in ("fcx", "fcy", "fcz")])
    mp.setUMAC([cuda(u) for u in umac])
    phi = cuda(np.zeros(g.cell_shape))
    st = mp.project(rtol=1e-11, atol=0.0, phi=phi, phi_guess=False)
    assert st["status"] == 0 and st["vcycles"] <= 2 * 26
    m = EBMac(n, [ext[d] / n[d] for d in range(3)], *bc, geo["vfrac"], [geo[k] for k in ("apx", "apy", "apz")],
              [geo[k] for k in ("fcx", "fcy", "fcz")], beta)
    assert rel_l2(phi.cpu().numpy(), m.project(umac)[1]) <= 1e-8
