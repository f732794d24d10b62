"""Device memory of the plans: the mixed form holds nothing that only the plain form reads, the plain form's own arrays are
reserved when it is chosen, and a plan without the memory for them solves all the same."""
import gc

import numpy as np
import pytest
import torch

import oracle as O
from incflo_gb300 import Geometry, MacProjector, NodalProjector, _abi, make_options
from tests.helpers import D, N, P, cuda, face_fields, nodal_case, rel_l2

pytestmark = pytest.mark.gpu

LO, HI = (N, D, P), (N, N, P)


def _padded(n, nodal, wide=True):
    """elements of a level's padded array: rows of n + 7 rounded up to 8; n + 3 (nodal) or n + 2 (cells) rows and planes. wide:
    nodal levels of 2^20 nodes with x walls have room for the four columns of a row's last thread"""
    e = 3 if nodal else 2
    row = -(-(n[0] + 7) // 8) * 8
    if nodal and wide and (n[0] + 1) * (n[1] + 1) * n[2] >= 1 << 20:
        row = max(row, -(-(4 * -(-(n[0] + 1) // 4) + 5) // 8) * 8)
    return row * (n[1] + e) * (n[2] + e)


def _levels(n):
    out = [tuple(n)]
    while all(v % 2 == 0 and v >= 4 for v in out[-1]):
        out.append(tuple(v // 2 for v in out[-1]))
    return out


class Nodal:
    def __init__(self, n, precision, create=True):
        ext = tuple(v / n[0] for v in n)
        _, self.sigma, self.vel = nodal_case(n, ext, LO, HI, seed=5)
        self.proj = NodalProjector(cuda(self.vel), cuda(self.sigma), Geometry(n, (0, 0, 0), ext),
                                   options=make_options(0, precision=precision))
        self.proj.setDomainBC(LO, HI)
        if create:
            self.create()

    def create(self):
        self.proj._plan()

    def bytes(self):
        return _abi.load().gbp_plan_device_bytes(self.proj._plan().ptr)

    def solve(self, precision):
        self.proj.vel = cuda(self.vel)
        self.proj.options = make_options(0, precision=precision)
        st = self.proj.project(rtol=1e-11, atol=0.0)
        return st, self.proj.getPhi().cpu().numpy()

    # per level: sigma and four vectors in FP64 and in FP32, a mask byte; on level 0: phi, right-hand side, residual and four
    # weights of the FP64 residual
    @staticmethod
    def most(n, wide=True):
        p = [_padded(v, True, wide) for v in _levels(n)]
        return 61 * sum(p) + (3 + 4) * 8 * p[0]


class Mac:
    def __init__(self, n, precision, create=True):
        ext = tuple(v / n[0] for v in n)
        g = O.Grid(n, hi=ext, bclo=LO, bchi=HI)
        rng = np.random.default_rng(5)
        beta = [cuda(np.abs(b) + 0.5) for b in face_fields(g, rng, zero_neumann=False)]
        self.umac, self.shape = face_fields(g, rng), g.cell_shape
        self.mp = MacProjector(Geometry(n, (0, 0, 0), ext), options=make_options(1, precision=precision))
        self.mp.initProjector(beta=beta)
        self.mp.setDomainBC(LO, HI)
        if create:
            self.create()

    def create(self):
        self.mp._ensure()

    def bytes(self):
        return _abi.load().gbp_plan_device_bytes(self.mp.plan.ptr)

    def solve(self, precision):
        self.mp.options = make_options(1, precision=precision)
        self.mp.setUMAC([cuda(u) for u in self.umac])
        phi = cuda(np.zeros(self.shape))
        st = self.mp.project(rtol=1e-11, atol=0.0, phi=phi, phi_guess=False)
        return st, phi.cpu().numpy()

    # per level: three face coefficients and three vectors in FP64 and in FP32; on level 0: phi, right-hand side, residual
    @staticmethod
    def most(n, wide=True):
        p = [_padded(v, False) for v in _levels(n)]
        return 72 * sum(p) + 3 * 8 * p[0]


@pytest.fixture(autouse=True)
def _fresh_plans():
    NodalProjector._plans.clear()
    yield
    NodalProjector._plans.clear()


@pytest.mark.parametrize("plan", [Nodal, Mac])
@pytest.mark.parametrize("n", [(64, 48, 56), (128, 96, 96)], ids=["64x48x56", "128x96x96"])
def test_mixed_plan_holds_no_plain_arrays(gpu_lib, plan, n):
    """(coarsest-level rows, tables and partial sums, alignment: 4 MB)"""
    p = plan(n, "mixed")
    assert p.bytes() <= plan.most(n) + (4 << 20)


@pytest.mark.parametrize("plan", [Nodal, Mac])
@pytest.mark.parametrize("n", [(48, 48, 48), (40, 24, 36)], ids=["48", "40x24x36"])
def test_changing_form(gpu_lib, plan, n):
    """mixed, plain, mixed, plain on one plan: the solutions of plans that never changed. Solves to 1e-11: within 1e-9."""
    ref = {f: plan(n, f).solve(f)[1] for f in ("mixed", "fp64")}
    NodalProjector._plans.clear()
    p = plan(n, "mixed")
    for f in ("mixed", "fp64", "mixed", "fp64", "fp64", "mixed"):
        st, phi = p.solve(f)
        assert st["status"] == 0 and rel_l2(phi, ref[f]) <= 1e-9


def _solve_with_room(plan, n, precision, room):
    """a plan made and used on a device with `room` bytes left (and a pool of torch's own for the solve's tensors)"""
    NodalProjector._plans.clear()
    gc.collect()  # no plan of an earlier test goes while the device is full
    torch.cuda.synchronize()
    p = plan(n, precision, create=False)
    hold = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    del hold
    fill = []
    while torch.cuda.mem_get_info()[0] > room + (8 << 20):
        fill.append(torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda"))
    try:
        p.create()
        return (p.bytes(),) + p.solve(precision)
    finally:
        del fill
        torch.cuda.empty_cache()


@pytest.mark.parametrize("plan", [Nodal, Mac])
def test_plain_form_without_its_arrays(gpu_lib, plan):
    """Room for a plan's basic arrays and half of the plain form's own: the plain form runs without them, as stationary V-cycles
    (12 to 14 of them from 1 to 1e-11 on smooth coefficients; 40 allowed)."""
    n = (256, 256, 128)
    p = plan(n, "fp64")
    full, phi = p.bytes(), p.solve("fp64")[1]
    del p
    base = plan.most(n)
    assert full - base > 128 << 20
    held, st, got = _solve_with_room(plan, n, "fp64", base + (full - base) // 2)
    assert held <= base + (4 << 20)
    assert st["status"] == 0 and st["vcycles"] <= 40 and rel_l2(got, phi) <= 1e-9


def test_nodal_plan_with_short_rows(gpu_lib):
    """Room for the basic arrays with rows as short as they can be, and half of what the whole-row sweeps want beyond that."""
    n = (256, 256, 128)
    phi = Nodal(n, "mixed").solve("mixed")[1]
    short, wide = Nodal.most(n, wide=False), Nodal.most(n)
    assert wide - short > 24 << 20
    held, st, got = _solve_with_room(Nodal, n, "mixed", (short + wide) // 2)
    assert held <= short + (4 << 20)
    assert st["status"] == 0 and st["vcycles"] <= 40 and rel_l2(got, phi) <= 1e-9
