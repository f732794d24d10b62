"""Coefficients beyond the everyday ones: of the other sign, zero, NaN, infinite. What a call accepts, what it refuses and
with which status does not depend on how the coarsest level is solved."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, LPInfo, MacProjector, NodalProjector, _abi, make_options
from tests.helpers import D, N, P, cuda, face_fields, nodal_case, rel_l2

pytestmark = pytest.mark.gpu

# coarsest levels of 27 nodes (dense inverse), 96 (the same, several entries per thread), 125 and 216 (conjugate gradients)
SIZES = [(16, 16, 16), (24, 24, 40), (32, 32, 32), (20, 20, 20)]
BCS = [((N, N, N), (N, N, N)), ((N, D, P), (N, N, P))]
ids = dict(argnames="n", argvalues=SIZES, ids=["x".join(map(str, n)) for n in SIZES])


def _solve(n, lo, hi, sigma, vel, precision, rtol=1e-11):
    ext = tuple(v / n[0] for v in n)
    info = LPInfo()
    if n == (32, 32, 32):
        info.setMaxCoarseningLevel(3)  # 4^3 cells
    vt = cuda(vel)
    proj = NodalProjector(vt, cuda(sigma), Geometry(n, (0, 0, 0), ext), info=info,
                          options=make_options(0, precision=precision))
    proj.setDomainBC(lo, hi)
    st = proj.project(rtol=rtol, atol=0.0)
    return st, proj.getPhi().cpu().numpy(), vt.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lo,hi", BCS, ids=["singular", "outflow"])
@pytest.mark.parametrize("n", SIZES[:2], ids=ids["ids"][:2])
def test_negative_sigma(gpu_lib, n, lo, hi, precision):
    """-sigma gives -phi and the same velocity: the solve runs through negated numbers, and two solves to 1e-11 agree
    within 1e-9."""
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, lo, hi, seed=6)
    st, phi, v = _solve(n, lo, hi, sigma, vel, precision)
    sn, pn, vn = _solve(n, lo, hi, -sigma, vel, precision)
    assert st["status"] == 0 and sn["status"] == 0
    assert rel_l2(-pn, phi) <= 1e-9
    assert np.abs(vn - v).max() <= 1e-9 * np.abs(v).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lo,hi", BCS, ids=["singular", "outflow"])
@pytest.mark.parametrize(**ids)
def test_zero_sigma_is_refused(gpu_lib, n, lo, hi, precision):
    """The coarsest operator vanishes: refused as a bad argument when sigma is set, the velocity untouched."""
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, lo, hi, seed=6)
    with pytest.raises(_abi.ProjectionError, match="bad argument"):
        _solve(n, lo, hi, 0.0 * sigma, vel, precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
@pytest.mark.parametrize(**ids)
def test_non_finite_sigma(gpu_lib, n, value, precision):
    """One non-finite cell: the solve reports a residual that is not a number, not a bad argument."""
    lo, hi = BCS[0]
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, lo, hi, seed=6)
    bad = sigma.copy()
    bad[3, 4, 5] = value
    with pytest.raises(_abi.ProjectionError, match="NaN"):
        _solve(n, lo, hi, bad, vel, precision)
    # and leaves nothing behind in the plan, which the next projector of this geometry uses
    assert _solve(n, lo, hi, sigma, vel, precision)[0]["status"] == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lo,hi", BCS, ids=["singular", "outflow"])
@pytest.mark.parametrize(**ids)
def test_negative_sigma_takes_the_same_vcycles(gpu_lib, n, lo, hi, precision):
    """Every number of the solve is the negated one of the positive solve or the same."""
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, lo, hi, seed=6)
    st, phi, _ = _solve(n, lo, hi, sigma, vel, precision)
    sn, pn, _ = _solve(n, lo, hi, -sigma, vel, precision)
    assert st["status"] == 0 and sn["status"] == 0 and sn["vcycles"] == st["vcycles"]
    assert rel_l2(-pn, phi) <= 1e-9


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("hi_z", [N, D], ids=["singular", "outflow"])
@pytest.mark.parametrize("n", [(16, 16, 16), (24, 24, 40), (20, 20, 20)], ids=["16x16x16", "24x24x40", "20x20x20"])
def test_negative_beta_takes_the_same_vcycles(gpu_lib, n, hi_z, precision):
    """The same for the MAC projection (coarsest levels of 8, 45 and 125 cells)."""
    lo, hi = (P, P, N), (P, P, hi_z)
    ext = tuple(v / n[0] for v in n)
    g = O.Grid(n, hi=ext, bclo=lo, bchi=hi)
    rng = np.random.default_rng(9)
    beta = [np.abs(b) + 0.2 for b in face_fields(g, rng, zero_neumann=False)]
    umac = face_fields(g, rng)
    res = []
    for s in (1.0, -1.0):
        mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, precision=precision))
        mp.initProjector(beta=[cuda(s * b) for b in beta])
        mp.setDomainBC(lo, hi)
        mp.setUMAC([cuda(u) for u in umac])
        phi = cuda(np.zeros(g.cell_shape))
        st = mp.project(rtol=1e-11, atol=0.0, phi=phi, phi_guess=False)
        assert st["status"] == 0
        res.append((st["vcycles"], s * phi.cpu().numpy()))
    assert res[1][0] == res[0][0] and rel_l2(res[1][1], res[0][1]) <= 1e-9
