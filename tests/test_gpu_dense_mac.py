"""Cell-centred hierarchies whose coarsest level has 113 to 127 cells (5^3 of 20^3, 40^3, ... among them): dense inverses with up
to eight entries per thread, behind the cluster's small levels where those fit beside the inverse."""
import ctypes

import numpy as np
import pytest

import oracle as O
from incflo_gb300 import Geometry, MacProjector, _abi, make_options
from tests.helpers import D, I, N, P, cuda, face_fields
from tests.test_gpu_level_kernels import test_cluster_bottom_solve_mac as _mac

pytestmark = pytest.mark.gpu

# 5 x 5 x 5 cells, 14 x 3 x 3, 6 x 7 x 3, 2 x 7 x 9 of one level; singular and not
CASES = [((20, 20, 20), (N, N, N), (N, N, N)), ((20, 20, 20), (P, N, D), (P, N, N)), ((28, 6, 6), (P, N, N), (P, N, N)),
         ((12, 14, 6), (N, D, P), (I, N, P)), ((2, 7, 9), (P, N, N), (P, N, N))]
cases = pytest.mark.parametrize("n,lo,hi", CASES, ids=["x".join(map(str, c[0])) + "-" + "".join(map(str, c[1])) for c in CASES])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@cases
def test_projection(gpu_lib, n, lo, hi, precision):
    _mac(gpu_lib, n, lo, hi, precision)


@pytest.mark.parametrize("n", [(20, 20, 20), (28, 6, 6)], ids=["20", "28x6x6"])
def test_cluster_vcycle(gpu_lib, n):
    """One V-cycle through the cluster against the per-level launches, as in test_gpu_mac.py."""
    bc = (P, P, N) if n[0] == 20 else (N, N, N)
    g = O.Grid(n, hi=tuple(v / n[0] for v in n), bclo=bc, bchi=bc)
    rng = np.random.default_rng(5)
    mp = MacProjector(Geometry(n, (0, 0, 0), tuple(v / n[0] for v in n)), options=make_options(1, precision="mixed"))
    mp.initProjector(beta=[cuda(np.abs(b) + 0.2) for b in face_fields(g, rng, zero_neumann=False)])
    mp.setDomainBC(bc, bc)
    mp.setUMAC([cuda(u) for u in face_fields(g, rng)])
    assert mp.project(rtol=1e-11, atol=0.0)["status"] == 0
    diff = ctypes.c_double(-1.0)
    _abi.check(_abi.load().gbp_plan_check_coarse_cycle(mp.plan.ptr, ctypes.byref(diff)), "check_coarse_cycle")
    assert 0.0 <= diff.value <= 1e-5
