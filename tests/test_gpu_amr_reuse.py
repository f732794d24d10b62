"""One two-level projector over several densities: its captured step is replayed, so everything that depends on the
density has to be renewed outside of it. The second projection of a kept projector agrees with a fresh projector's."""
import numpy as np
import pytest
import torch

from incflo_gb300 import AmrNodalProjector, Geometry, make_options
from tests.helpers import N, P, cuda, rel_l2

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def _density(n, z0):
    """1 -> 3 across an interface two coarse cells wide at height z0 (of a unit box), rippled along x and y"""
    x, y, z = ((np.arange(v) + 0.5) / v for v in n)
    hxy = z0 + 0.05 * np.cos(2 * np.pi * x)[None, :] * np.cos(2 * np.pi * y)[:, None]
    return 2.0 + np.tanh((z[:, None, None] - hxy[None]) * 24.0)


def _apply(proj, nc, box, z0, vel_c, vel_f):
    nf = [2 * v for v in nc]
    lo, hi = box
    rho_f = _density(nf, z0)[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]
    vc, vf = cuda(vel_c), [cuda(vel_f)]
    pc = torch.zeros((nc[2] + 1, nc[1] + 1, nc[0] + 1), dtype=torch.float64, device="cuda")
    pf = [torch.zeros([hi[d] - lo[d] + 2 for d in (2, 1, 0)], dtype=torch.float64, device="cuda")]
    st = proj.apply(vc, cuda(_density(nc, z0)), torch.zeros_like(vc), pc, vf, [cuda(rho_f)],
                    [torch.zeros_like(v) for v in vf], pf, scaling_factor=1.0)
    return st, pc.cpu().numpy(), pf[0].cpu().numpy(), vc.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,box", [
    ((48, 48, 48), ((0, 0, 32), (95, 95, 63))),  # both levels have the shared-sum FP64 sweep (100 000 nodes and more)
    ((32, 32, 32), ((0, 0, 16), (63, 63, 47))),  # the fine level alone
], ids=["base-48", "base-32"])
def test_moved_density_on_a_kept_projector(gpu_lib, nc, box, precision):
    """The interface moves by two coarse cells; velocity, and with it the right-hand side and its power-of-two scale, stay.
    Two solves to a relative residual of 1e-11 agree within 1e-9, and start and right-hand side are the same, so that the
    V-cycle counts differ by a step's worth of rounding at most."""
    lo, hi = box
    rng = np.random.default_rng(3)
    vel_c = rng.standard_normal((3, nc[2], nc[1], nc[0]))
    sl = tuple(slice(lo[d] // 2, (hi[d] + 1) // 2) for d in (2, 1, 0))
    vel_f = vel_c[(slice(None),) + sl].repeat(2, 1).repeat(2, 2).repeat(2, 3)

    def projector():
        return AmrNodalProjector(Geometry(nc), (P, P, N), (P, P, N), [box],
                                 options=make_options(0, precision=precision, mg_rtol=RTOL, mg_atol=0.0))

    kept = projector()
    shift = 2.0 / nc[2]
    for z0 in (0.5, 0.5 + shift, 0.5 - shift):
        st, pc, pf, vc = _apply(kept, nc, box, z0, vel_c, vel_f)
        ref, rc, rf, rv = _apply(projector(), nc, box, z0, vel_c, vel_f)
        assert ref["status"] == 0 and ref["final_rel_resid"] <= RTOL
        assert st["status"] == 0 and st["final_rel_resid"] <= RTOL
        assert abs(st["vcycles"] - ref["vcycles"]) <= 2
        assert rel_l2(pc, rc) <= 1e-9 and rel_l2(pf, rf) <= 1e-9
        assert np.abs(vc - rv).max() <= 1e-9 * np.abs(rv).max()
