"""Level kernels of the nodal and MAC hierarchies at the sizes where their tiles, seams and dispatch rules change,
against the CPU oracle: phi within 1e-9 (relative L2) of the oracle's at rtol 1e-12, as in test_gpu_nodal.py."""
import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, make_options
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


# coarsest levels of 65 to several thousand unknowns (cell counts with odd factors): the cluster's conjugate
# gradients, with rows that leave lanes, warps and whole CTAs idle, and with coefficients kept in shared memory or not
BOTTOMS = [
    ((24, 20, 36), (P, N, P), (P, N, P)),     # singular
    ((40, 56, 24), (N, D, P), (I, N, P)),
    ((26, 22, 34), (P, P, D), (P, P, N)),     # 13 x 11 x 17 cells
    ((42, 38, 50), (N, N, N), (N, N, N)),     # 21 x 19 x 25 cells: coefficients from L2
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi", BOTTOMS, ids=["x".join(map(str, c[0])) for c in BOTTOMS])
def test_cluster_bottom_solve_nodal(gpu_lib, n, lo, hi, precision):
    _nodal(n, lo, hi, precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi", BOTTOMS, ids=["x".join(map(str, c[0])) for c in BOTTOMS])
def test_cluster_bottom_solve_mac(gpu_lib, n, lo, hi, precision):
    lo, hi = ([N if b == I else b for b in s] for s in (lo, hi))
    g = O.Grid(n, hi=tuple(v / n[0] for v in n), bclo=lo, bchi=hi)
    rng = np.random.default_rng(3)
    beta = [rng.uniform(0.3, 1.0, g.face_shape(d)) for d in range(3)]
    u = [rng.standard_normal(g.face_shape(d)) for d in range(3)]
    for d in range(3):  # one value per periodic face, none through walls
        ax = 2 - d
        first, last = [slice(None)] * 3, [slice(None)] * 3
        first[ax], last[ax] = 0, -1
        for f in (beta[d], u[d]):
            if lo[d] == P:
                f[tuple(last)] = f[tuple(first)]
        if lo[d] == N:
            u[d][tuple(first)] = 0.0
        if hi[d] == N:
            u[d][tuple(last)] = 0.0
    un, phi_or, st_or = O.mac_project(g, beta, u, rtol=1e-13)
    mp = MacProjector(Geometry(n, (0, 0, 0), tuple(v / n[0] for v in n)), options=make_options(1, precision=precision))
    mp.initProjector(beta=[cuda(b) for b in beta])
    mp.setDomainBC(lo, hi)
    ut, phi = [cuda(x) for x in u], cuda(np.zeros(g.cell_shape))
    mp.setUMAC(ut)
    st = mp.project(rtol=1e-12, atol=0.0, phi=phi, phi_guess=False)
    assert st["status"] == 0 and rel_l2(phi.cpu().numpy(), phi_or) <= 1e-9


# levels that one thread-block cluster cycles in shared memory: fewer planes than CTAs, planes that do not split evenly,
# levels with one CTA's worth of points at once, periodic and bounded in z
TAILS = [((16, 32, 8), (P, N, P), (P, D, P)), ((8, 12, 64), (N, P, P), (N, P, P)), ((32, 16, 56), (D, N, N), (N, I, N))]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi", TAILS, ids=["x".join(map(str, c[0])) for c in TAILS])
def test_cluster_tail(gpu_lib, n, lo, hi, precision):
    _nodal(n, lo, hi, precision)
    test_cluster_bottom_solve_mac(gpu_lib, n, lo, hi, precision)


@pytest.mark.parametrize("n,lo,hi", [((128, 128, 72), (P, P, N), (P, P, N)), ((144, 100, 96), (N, D, P), (I, N, P))],
                         ids=["128x128x72", "144x100x96"])
def test_relaxed_vcycles(gpu_lib, n, lo, hi):
    """FP32 V-cycles from the current iterate with Chebyshev weights (whole-row levels): the FP64 solve's phi within twice
    the 1e-9 that either may be off, in at most a V-cycle more per refinement step than accelerated FP64 V-cycles."""
    ext = tuple(v / n[0] for v in n)
    g, sigma, vel = nodal_case(n, ext, lo, hi, seed=2)
    phi, st = {}, {}
    for p in ("fp64", "mixed"):
        proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(n, (0, 0, 0), ext), options=make_options(0, precision=p))
        proj.setDomainBC(lo, hi)
        st[p] = proj.project(rtol=1e-12, atol=0.0)
        assert st[p]["status"] == 0 and st[p]["final_rel_resid"] <= 1e-12
        phi[p] = unique_nodes(g, proj.getPhi().cpu().numpy())
    assert rel_l2(phi["mixed"], phi["fp64"]) <= 2e-9
    assert st["mixed"]["vcycles"] <= st["fp64"]["vcycles"] + st["mixed"]["outer_iters"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi", [((48, 24, 48), (N, N, N), (N, N, N)), ((56, 32, 16), (N, P, D), (D, P, N))],
                         ids=["48x24x48", "56x32x16"])
def test_dense_bottoms(gpu_lib, n, lo, hi, precision):
    """Dense inverses of several entries per thread (108 and 112 cells), singular and not, and nodal bottoms beside them."""
    test_cluster_bottom_solve_mac(gpu_lib, n, lo, hi, precision)
    _nodal(n, lo, hi, precision)
