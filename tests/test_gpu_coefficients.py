"""Coefficients beyond the everyday ones: of the other sign, zero, NaN, infinite. What a call accepts, what it refuses and
with which status does not depend on how the coarsest level is solved."""
import numpy as np
import pytest

from incflo_gb300 import Geometry, LPInfo, NodalProjector, _abi, make_options
from tests.helpers import D, N, P, cuda, nodal_case, rel_l2

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
