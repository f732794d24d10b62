"""Level kernels of the nodal and MAC hierarchies at the sizes where their tiles, seams and dispatch rules change,
against the CPU oracle: phi within 1e-9 (relative L2) of the oracle's at rtol 1e-12, as in test_gpu_nodal.py."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, NodalProjector, make_options
from tests.helpers import D, I, N, P, cuda, nodal_case, rel_l2, unique_nodes

pytestmark = pytest.mark.gpu


def _nodal(n, lo, hi, precision, ext=None, seed=1):
    ext = ext or tuple(v / n[0] for v in n)
    g, sigma, vel = nodal_case(n, ext, lo, hi, seed=seed)
    vel_or, phi_or, _, st_or = O.nodal_project(g, sigma, vel, rtol=1e-13)
    vt = cuda(vel)
    proj = NodalProjector(vt, cuda(sigma), Geometry(n, (0, 0, 0), ext), options=make_options(0, precision=precision))
    proj.setDomainBC(lo, hi)
    st = proj.project(rtol=1e-12, atol=0.0)
    assert st["status"] == 0 and st["final_rel_resid"] <= 1e-12
    assert rel_l2(unique_nodes(g, proj.getPhi().cpu().numpy()), phi_or) <= 1e-9
    scale = np.abs(vel_or[:, 1:-1, 1:-1, 1:-1]).max()
    assert np.abs(vt.cpu().numpy()[:, 1:-1, 1:-1, 1:-1] - vel_or[:, 1:-1, 1:-1, 1:-1]).max() <= 1e-9 * scale


@pytest.mark.parametrize("n,lo,hi", [
    ((48, 48, 48), (P, P, P), (P, P, P)),    # the smallest level of the shared-sum FP64 sweep
    ((72, 56, 40), (N, D, P), (I, N, P)),    # tiles of 32 x 8 with remainders, z chunks with a remainder
    ((128, 32, 32), (P, N, N), (P, N, D)),
], ids=["48", "72x56x40", "128x32x32"])
def test_fp64_sweep_tiles(gpu_lib, n, lo, hi):
    _nodal(n, lo, hi, "fp64")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi", [
    ((4, 4, 4), (P, P, P), (P, P, P)),       # a 2-cell periodic level: node 1 aliases to both sides
    ((12, 6, 10), (P, P, P), (P, P, P)),     # 3- and 5-cell periodic levels
    ((8, 12, 4), (P, N, P), (P, D, P)),
], ids=["4", "12x6x10", "8x12x4"])
def test_periodic_seams_of_small_levels(gpu_lib, n, lo, hi, precision):
    _nodal(n, lo, hi, precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ext,lo,hi", [
    ((34, 24, 40), (1.0, 24 * 0.8 / 34, 40 * 1.25 / 34), (P, P, N), (P, P, N)),  # rows end inside a 16-byte vector
    ((32, 32, 24), (1.0, 0.8, 0.9375), (D, N, P), (N, I, P)),
], ids=["34x24x40", "32x32x24"])
def test_accelerated_vcycles_on_stretched_cells(gpu_lib, n, ext, lo, hi, precision):
    """Cells of aspect 1 : 0.8 : 1.25: stationary V(2,2) cycles need 38 for 1e-11, accelerated ones 16."""
    _nodal(n, lo, hi, precision, ext=ext)
    proj = NodalProjector(*(cuda(a) for a in nodal_case(n, ext, lo, hi, seed=1)[:0:-1]), Geometry(n, (0, 0, 0), ext),
                          options=make_options(0, precision=precision))
    proj.setDomainBC(lo, hi)
    assert proj.project(rtol=1e-11, atol=0.0)["vcycles"] <= 24
