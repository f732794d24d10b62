"""stats.kernel_launches: the kernels a projection ran, counted by hand on small grids (levels of 8, 4 and 2 cells per
direction, or one level of 2), with captured steps and without."""
import numpy as np
import pytest

from incflo_gb300 import Geometry, MacProjector, apply_nodal_projection, make_options
from tests.helpers import N, P, cuda, face_fields
import oracle as O

pytestmark = pytest.mark.gpu

BC = (P, P, N)
VECTORS = 5  # beta, direction, operator, alpha, update


@pytest.mark.parametrize("graphs", [1, 0], ids=["graphs", "direct"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2, 8])
def test_mac(gpu_lib, n, precision, graphs):
    g = O.Grid((n,) * 3, bclo=BC, bchi=BC)
    rng = np.random.default_rng(3)
    umac = face_fields(g, rng)
    mp = MacProjector(Geometry((n,) * 3), options=make_options(1, precision=precision, use_graphs=graphs))
    mp.initProjector(beta=1.0)
    mp.setDomainBC(BC, BC)
    phi = cuda(np.zeros(g.cell_shape))
    for first in (True, False):
        mp.setUMAC([cuda(u) for u in umac])
        st = mp.project(rtol=1e-11, atol=0.0, phi=phi, phi_guess=False)
        steps, v = st["outer_iters"] - 1, st["vcycles"]
        # right-hand side and its mean (sums, fold, subtraction), two norms' kernels; phi's mean, three corrections, phi out
        want = (1 + 3 + 2) + (3 + 3 + 1)
        if precision == "mixed":
            want += 3 * steps + v * (1 + (VECTORS if n > 2 else 0))  # to FP32, from FP32, residual; the cluster's V-cycle
        elif n == 2:
            want += 3 * steps
        else:
            want += v * (2 * 9 + 1 + VECTORS) + 1  # two levels of 8 half sweeps and a residual, the bottom; the true residual
        if precision == "fp64" and first:
            want += st["num_levels"]  # the reciprocal diagonals
        assert st["kernel_launches"] == want, (st, want)


@pytest.mark.parametrize("graphs", [1, 0], ids=["graphs", "direct"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2, 8])
def test_nodal(gpu_lib, n, precision, graphs):
    rng = np.random.default_rng(3)
    vel = np.zeros((3,) + (n + 2,) * 3)
    vel[:, 1:-1, 1:-1, 1:-1] = rng.standard_normal((3,) + (n,) * 3)
    rho = cuda(1.0 + rng.random((n,) * 3))
    gp, p = cuda(np.zeros((3,) + (n,) * 3)), cuda(np.zeros((n + 1,) * 3))
    opt = make_options(0, precision=precision, use_graphs=graphs, mg_rtol=1e-11, mg_atol=0.0)
    st = apply_nodal_projection(Geometry((n,) * 3), BC, BC, cuda(vel), rho, gp, p, options=opt)
    steps, v = st["outer_iters"] - 1, st["vcycles"]
    # sigma on every level, the bottom's rows and inverse; right-hand side, its mean (two); phi's mean, phi out, correction
    want = st["num_levels"] + 2 + 1 + 2 + 3 + 1 + 1
    if precision == "mixed":
        # the first right-hand side; per step the correction, the residual and the next right-hand side
        want += 1 + 3 * steps + v * (1 + (VECTORS if n > 2 else 0))
    elif n == 2:
        want += 3 * steps
    else:
        want += v * (1 + VECTORS) + 1
    assert st["kernel_launches"] == want, (st, want)
