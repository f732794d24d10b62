"""Dense coarsest levels of 65 to 112 unknowns behind the cluster's small levels, singular ones above all: one V-cycle
through the cluster kernel against the per-level launches, as in test_gpu_nodal.py. A coarsest level solved for another
right-hand side differs by O(1); the summation order differs by FP32 rounding over some 10 passes (1e-5)."""
import ctypes

import pytest

from incflo_gb300 import Geometry, NodalProjector, _abi, make_options
from tests.helpers import D, N, P, cuda, nodal_case

pytestmark = pytest.mark.gpu

CASES = [
    ((24, 24, 40), (N, N, N), (N, N, N)),   # 4 x 4 x 6 nodes
    ((24, 24, 72), (P, P, P), (P, P, P)),   # 3 x 3 x 9
    ((56, 16, 32), (P, P, N), (P, P, N)),   # 7 x 2 x 5
    ((16, 16, 88), (N, N, N), (N, N, N)),   # 3 x 3 x 12: 108
    ((40, 40, 24), (P, P, N), (P, P, N)),   # 5 x 5 x 4: 100
    ((24, 24, 24), (N, N, N), (N, N, N)),   # 4 x 4 x 4: 64, the former limit
    ((24, 24, 40), (N, D, P), (N, N, P)),   # 4 x 4 x 5: 80, not singular
]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,lo,hi", CASES, ids=["x".join(map(str, c[0])) + "-" + "".join(map(str, c[1])) for c in CASES])
def test_cluster_vcycle_over_dense_bottoms(gpu_lib, n, lo, hi, precision):
    ext = tuple(v / n[0] for v in n)
    _, sigma, vel = nodal_case(n, ext, lo, hi, seed=4)
    proj = NodalProjector(cuda(vel), cuda(sigma), Geometry(n, (0, 0, 0), ext), options=make_options(0, precision=precision))
    proj.setDomainBC(lo, hi)
    assert proj.project(rtol=1e-11, atol=0.0)["status"] == 0
    diff = ctypes.c_double(-1.0)
    _abi.check(_abi.load().gbp_plan_check_coarse_cycle(proj._plan().ptr, ctypes.byref(diff)), "check_coarse_cycle")
    assert 0.0 <= diff.value <= 1e-5
