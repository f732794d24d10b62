"""The projections, diffusion solve and network step that a flow solver asks of this library, as measured cases.

Every case is one call of a public entry point on fields resident on the GPU, at the sizes of this repository's
configurations, tests and benchmark:

  nodal      apply_nodal_projection: the cell velocity, gp and p_nd of one level (gp is added back first)
  mac        MacProjector: new face coefficients, then the face velocities and phi
  eb_nodal   apply_nodal_projection with cut cells (a cylinder across a channel)
  eb_mac     MacProjector with cut cells
  amr        AmrNodalProjector: base level and a tagged fine level of ratio 2 in many boxes
  tensor     TensorOp: the implicit velocity diffusion of a channel
  unet       Surrogate: loss and gradients of one pair, then the prediction of the warm-start network

The projections overwrite their velocity; a time step writes a new one before each of them, so a pass starts by
copying it in. Plans, projectors and cut-cell geometry are kept from one step to the next, as a program does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from incflo_gb300 import AmrNodalProjector, Geometry, MacProjector, apply_nodal_projection, eb, make_options, synth
from incflo_gb300.diffusion import TensorOp
from incflo_gb300.surrogate import Surrogate

P, D, N, I = 0, 1, 2, 3
CODE = {"p": P, "d": D, "n": N, "i": I}
F64 = dict(dtype=torch.float64, device="cuda")


def listed():
    return [
        # the smallest grids in use (unit problems, coarse regression runs): launches and read-backs count
        dict(name="nodal-16", kind="nodal", nx=16, ny=16, nz=16, lo="ppn", hi="ppn", hy=1.0, hz=1.0, rho="interface",
             precision="fp64", rtol=1e-11),
        # the single-level Taylor-Green configuration with incflo's own precision and tolerances
        dict(name="nodal-tg-64", kind="nodal", nx=64, ny=64, nz=64, lo="ppp", hi="ppp", hy=1.0, hz=1.0, rho="one",
             precision="fp64", rtol=1e-11),
        dict(name="mac-tg-64", kind="mac", nx=64, ny=64, nz=64, lo="ppp", hi="ppp", hy=1.0, hz=1.0, rho="one",
             precision="fp64", rtol=1e-11),
        # a box that is no power of two, between an inflow and an outflow, with walls
        dict(name="nodal-ragged", kind="nodal", nx=144, ny=80, nz=112, lo="inn", hi="dnn", hy=1.0, hz=1.0,
             rho="interface", precision="mixed", rtol=1e-11),
        # the variable-density benchmark: the chosen form, the plain form, and its MAC projection
        dict(name="nodal-256", kind="nodal", nx=256, ny=256, nz=256, lo="ppn", hi="ppn", hy=1.0, hz=1.0,
             rho="interface", precision="mixed", rtol=1e-10),
        dict(name="nodal-256-fp64", kind="nodal", nx=256, ny=256, nz=256, lo="ppn", hi="ppn", hy=1.0, hz=1.0,
             rho="interface", precision="fp64", rtol=1e-10),
        dict(name="mac-256", kind="mac", nx=256, ny=256, nz=256, lo="ppn", hi="ppn", hy=1.0, hz=1.0, rho="interface",
             precision="mixed", rtol=1e-10),
        # flow past a cylinder: cut cells
        dict(name="eb-nodal", kind="eb_nodal", ny=64, precision="mixed", rtol=1e-11),
        dict(name="eb-mac", kind="eb_mac", ny=64, precision="mixed", rtol=1e-11),
        # two levels, the fine one tagged around the interface
        dict(name="amr-256", kind="amr", nx=256, precision="mixed", rtol=1e-10),
        # implicit viscous step of a channel
        dict(name="tensor-channel", kind="tensor", nx=256, ny=128, nz=128, precision="mixed", rtol=1e-10),
        # training and inference of the warm-start network at its training size
        dict(name="unet-128", kind="unet", nx=128, ny=128, nz=128),
    ]


def _size(rng, most):
    """2^k m with k >= 3 (the default blocking factor) and m odd, spread over the logarithm"""
    sizes = [m << k for k in range(3, 9) for m in (1, 3, 5, 7, 9, 11, 13) if 16 <= m << k <= most]
    t = math.exp(rng.uniform(math.log(16), math.log(most)))
    return min(sizes, key=lambda s: (abs(math.log(s / t)), s))


def draw(rng):
    """the same calls over their range, at the library's default tolerance"""
    kind = rng.choice(["nodal", "nodal", "nodal", "mac", "mac", "eb_nodal", "eb_mac", "amr", "tensor", "unet"])
    if kind in ("nodal", "mac"):
        precision = rng.choice(["fp64", "mixed"])
        most = 128 if precision == "fp64" else 256
        n = [_size(rng, most) for _ in range(3)]
        lo, hi = rng.choice([("ppp", "ppp"), ("ppn", "ppn"), ("inn", "dnn"), ("ipp", "dpp"), ("nnn", "nnn"), ("pnp", "pnp")])
        hy, hz = rng.choice([(1.0, 1.0), (1.0, 1.0), (0.8, 1.25)])
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], lo=lo, hi=hi, hy=hy, hz=hz,
                    rho=rng.choice(["interface", "one"]), precision=precision, rtol=1e-11)
    if kind in ("eb_nodal", "eb_mac"):
        return dict(kind=kind, ny=rng.choice([16, 24, 32, 40, 48, 64]), precision=rng.choice(["fp64", "mixed"]),
                    rtol=1e-11)
    if kind == "amr":
        return dict(kind=kind, nx=rng.choice([64, 96, 128, 160]), precision="mixed", rtol=1e-11)
    if kind == "tensor":
        n = [_size(rng, 128) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], precision=rng.choice(["fp64", "mixed"]),
                    rtol=1e-11)
    n = [8 * rng.randint(2, 16) for _ in range(3)]
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2])


# ------------------------------------------------------------------------------------------------ inputs
def _grid(case):
    """cells, spacing, boundary types of both sides"""
    k = case["kind"]
    if k in ("eb_nodal", "eb_mac"):
        m = case["ny"]
        n = (4 * m, m, m)
        return n, (1.0 / m,) * 3, (I, N, P), (D, N, P)
    if k == "amr":
        n = (case["nx"],) * 3
        return n, (1.0 / n[0],) * 3, (P, P, N), (P, P, N)
    n = (case["nx"], case["ny"], case["nz"])
    if k == "tensor":
        return n, (1.0 / n[1],) * 3, (P, D, P), (P, D, P)
    h = 1.0 / n[0]
    return (n, (h, h * case["hy"], h * case["hz"]), tuple(CODE[c] for c in case["lo"]),
            tuple(CODE[c] for c in case["hi"]))


def _geom(n, h):
    return Geometry(n, (0.0, 0.0, 0.0), tuple(n[d] * h[d] for d in range(3)))


def _options(case, kind):
    return make_options(kind, precision=case["precision"], mg_rtol=case["rtol"], mg_atol=0.0)


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _random_field(n, g):
    """three components of a Gaussian random field with energy spectrum k^-2, zero mean, unit RMS"""
    k = [torch.fft.fftfreq(n[d], **F64) * n[d] for d in (2, 1)] + [torch.fft.rfftfreq(n[0], **F64) * n[0]]
    kk = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    amp = torch.where(kk > 0, kk.clamp(min=1.0) ** -1.0, torch.zeros_like(kk))
    v = torch.empty((3, n[2], n[1], n[0]), **F64)
    for c in range(3):
        w = torch.randn((n[2], n[1], n[0]), generator=g, **F64)
        v[c] = torch.fft.irfftn(torch.fft.rfftn(w) * amp, s=(n[2], n[1], n[0]))
    v -= v.mean(dim=(1, 2, 3), keepdim=True)
    return v / (v * v).sum(dim=0).mean().sqrt()


def _density(case, n, h, seed):
    """1, or 1 -> 3 across a tanh interface two cells wide, displaced by cosine modes"""
    if case["rho"] == "one":
        return torch.ones((n[2], n[1], n[0]), **F64)
    hxy = torch.from_numpy(synth.interface_height(n, seed)).to(**F64)
    z = (torch.arange(n[2], **F64) + 0.5) / n[2]
    return 2.0 + torch.tanh((z[:, None, None] - hxy[None]) * n[2] / 2.0)


def _velocity(n, h, lo, hi, seed):
    """random field, on an all-periodic box with the Taylor-Green vortex, behind an inflow with the mean stream"""
    v = _random_field(n, _generator(seed))
    if all(b == P for b in lo):
        x, y, z = (2.0 * math.pi * (torch.arange(n[d], **F64) + 0.5) / n[d] for d in range(3))
        x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
        v *= 1e-2
        v[0] += torch.sin(x) * torch.cos(y) * torch.cos(z)
        v[1] -= torch.cos(x) * torch.sin(y) * torch.cos(z)
    if I in lo:
        v *= 0.1
        v[0] += 1.0
    return v


def _faces(v, n, lo, hi):
    """cell velocity averaged to the faces: wrapped on periodic sides, 0 on walls, 1 on an inflow, the cell's else"""
    out = []
    for d in range(3):
        ax = 2 - d
        c = v[d]
        first, last = c.narrow(ax, 0, 1), c.narrow(ax, n[d] - 1, 1)
        mid = 0.5 * (c.narrow(ax, 1, n[d] - 1) + c.narrow(ax, 0, n[d] - 1))
        ends = []
        for b, own, other in ((lo[d], first, last), (hi[d], last, first)):
            ends.append(0.5 * (own + other) if b == P else torch.zeros_like(own) if b == N
                        else torch.ones_like(own) if b == I else own)
        out.append(torch.cat([ends[0], mid, ends[1]], dim=ax).contiguous())
    return out


def _face_beta(rho, n, lo):
    out = []
    for d in range(3):
        ax = 2 - d
        first, last = rho.narrow(ax, 0, 1), rho.narrow(ax, n[d] - 1, 1)
        mid = 0.5 * (rho.narrow(ax, 1, n[d] - 1) + rho.narrow(ax, 0, n[d] - 1))
        a, b = (0.5 * (first + last),) * 2 if lo[d] == P else (first, last)
        out.append((1.0 / torch.cat([a, mid, b], dim=ax)).contiguous())
    return out


_kept: dict = {}


def _keep(case, what, make):
    """what a program makes once and uses in every step; the last two kinds of case stay"""
    key = (tuple(sorted((k, v) for k, v in case.items() if k != "name")), what)
    if key not in _kept:
        while len(_kept) >= 4:
            _kept.pop(next(iter(_kept)))
        _kept[key] = make()
    return _kept[key]


CENTER, RADIUS, SMALL = (1.0, 0.5, 0.0), 0.125, 1e-4


def _cut_nodal(n, h):
    ext = tuple(n[d] * h[d] for d in range(3))
    m = eb.cylinder_moments(n, (0, 0, 0), ext, CENTER, RADIUS, small_volfrac=SMALL)
    return torch.from_numpy(eb.moments_components(m)).cuda()


def _cut_mac(n, h):
    ext = tuple(n[d] * h[d] for d in range(3))
    geo = eb.cylinder(n, (0, 0, 0), ext, CENTER, RADIUS, small_volfrac=SMALL)
    ap = [torch.from_numpy(geo[k]).cuda() for k in ("apx", "apy", "apz")]
    fc = [torch.from_numpy(np.ascontiguousarray(np.moveaxis(geo[k], -1, 0))).cuda() for k in ("fcx", "fcy", "fcz")]
    return torch.from_numpy(geo["vfrac"]).cuda(), ap, fc


def _amr_layout(case, n):
    """fine boxes around the interface and where the reference field's vorticity is high"""
    hxy = torch.from_numpy(synth.interface_height(n, 2)).to(**F64)
    z = (torch.arange(n[2], **F64) + 0.5) / n[2]
    dist = z[:, None, None] - hxy[None]
    v = _random_field(n, _generator(3)) * torch.exp(-(dist / 0.1) ** 2)
    rot = [torch.roll(v[a], -1, 3 - b - 1) - torch.roll(v[a], 1, 3 - b - 1) - torch.roll(v[b], -1, 3 - a - 1)
           + torch.roll(v[b], 1, 3 - a - 1) for a, b in ((2, 1), (0, 2), (1, 0))]
    om = (rot[0] ** 2 + rot[1] ** 2 + rot[2] ** 2).sqrt()
    high = om > torch.kthvalue(om.reshape(-1), int(0.9 * om.numel())).values
    band = dist.abs() <= 0.1
    return synth.tag_and_box((band | (high & (dist.abs() <= 0.2))).cpu().numpy(), 32, 64), dist


def _prepare_amr(case, seed):
    n, h, lo, hi = _grid(case)
    boxes, dist = _keep(case, "layout", lambda: _amr_layout(case, n))
    proj = _keep(case, "projector", lambda: AmrNodalProjector(_geom(n, h), lo, hi, boxes, options=_options(case, 0)))
    vel = (_random_field(n, _generator(seed)) * torch.exp(-(dist / 0.1) ** 2)).contiguous()
    rho = 2.0 + torch.tanh(dist * n[2] / 2.0)
    nf = tuple(2 * v for v in n)
    hf = torch.from_numpy(synth.interface_height(nf, 2)).to(**F64)
    zf = (torch.arange(nf[2], **F64) + 0.5) / nf[2]
    size = [tuple(b[1][d] - b[0][d] + 1 for d in (2, 1, 0)) for b in boxes]
    cells = [int(np.prod(s)) for s in size]
    nodes = [int(np.prod([v + 1 for v in s])) for s in size]
    # the fine level's FABs lie one behind the other in one allocation per field
    vel_f, rho_f = torch.empty(3 * sum(cells), **F64), torch.empty(sum(cells), **F64)
    s = dict(case=case, proj=proj, vel0=vel, vel=vel.clone(), rho=rho, gp=torch.zeros_like(vel),
             p=torch.zeros((n[2] + 1, n[1] + 1, n[0] + 1), **F64), vel_f0=vel_f, rho_f=rho_f,
             gp_f=torch.zeros_like(vel_f), p_f=torch.zeros(sum(nodes), **F64))

    def fabs(flat, comps, counts, shape):
        out, at = [], 0
        for c, sh in zip(counts, shape):
            out.append(flat[at:at + comps * c].view((comps,) + sh if comps > 1 else sh))
            at += comps * c
        return out

    for v, r, (blo, bhi) in zip(fabs(vel_f, 3, cells, size), fabs(rho_f, 1, cells, size), boxes):
        sl = tuple(slice(blo[d] // 2, (bhi[d] + 1) // 2) for d in (2, 1, 0))
        v.copy_(vel[(slice(None),) + sl].repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3))
        f = tuple(slice(blo[d], bhi[d] + 1) for d in (2, 1, 0))
        r.copy_(2.0 + torch.tanh((zf[f[0], None, None] - hf[None, f[1], f[2]]) * nf[2] / 2.0))
    s["vel_f"] = vel_f.clone()
    s["fabs"] = [fabs(s["vel_f"], 3, cells, size), fabs(rho_f, 1, cells, size), fabs(s["gp_f"], 3, cells, size),
                 fabs(s["p_f"], 1, nodes, [tuple(v + 1 for v in q) for q in size])]
    return s


def _tensor_fields(case, seed):
    n, h, lo, hi = _grid(case)
    g = _generator(seed)
    shape = (n[2], n[1], n[0])
    rho = 1.0 + torch.rand(shape, generator=g, **F64)
    eta = 0.01 * (1.0 + torch.rand(shape, generator=g, **F64))
    v = torch.zeros((3, n[2] + 2, n[1] + 2, n[0] + 2), **F64)
    v[:, 1:-1, 1:-1, 1:-1] = torch.randn((3,) + shape, generator=g, **F64)
    v[0, 1:-1, -1, 1:-1] = 1.0  # moving upper wall
    return n, h, rho, eta, v


def _tensor_op(case, n, h):
    op = TensorOp(_geom(n, h), options=_options(case, 1))
    op.setDomainBC([[P, D, P]] * 3, [[P, D, P]] * 3)
    op.setScalars(1.0, 0.5 * h[0])
    return op


def prepare(case, seed):
    kind = case["kind"]
    if kind == "amr":
        return _prepare_amr(case, seed)
    if kind == "unet":
        n = (case["nx"], case["ny"], case["nz"])
        g = _generator(seed)
        x = torch.zeros((n[2] + 2, n[1] + 2, n[0] + 2, 16), dtype=torch.bfloat16, device="cuda")
        x[1:-1, 1:-1, 1:-1, :3] = torch.randn((n[2], n[1], n[0], 3), generator=g, device="cuda").bfloat16()
        t = torch.zeros((n[2] + 2, n[1] + 2, n[0] + 2), dtype=torch.float32, device="cuda")
        t[1:-1, 1:-1, 1:-1] = torch.randn((n[2], n[1], n[0]), generator=g, device="cuda")
        net = _keep(case, "network", lambda: Surrogate(seed=5))
        return dict(case=case, net=net, x=x.reshape(-1, 16), t=t.reshape(-1), n=n)
    if kind == "tensor":
        n, h, rho, eta, v = _tensor_fields(case, seed)
        op = _keep(case, "operator", lambda: _tensor_op(case, n, h))
        rhs = (rho[None] * v[:, 1:-1, 1:-1, 1:-1]).contiguous()
        return dict(case=case, op=op, rho=rho, eta=eta, vel0=v, vel=v.clone(), rhs=rhs)
    n, h, lo, hi = _grid(case)
    if kind in ("eb_nodal", "eb_mac"):
        v = 1e-3 * (2.0 * torch.rand((3, n[2], n[1], n[0]), generator=_generator(seed), **F64) - 1.0)
        v[0] += 1.0
        rho = torch.ones((n[2], n[1], n[0]), **F64)
    else:
        v, rho = _velocity(n, h, lo, hi, seed), _density(case, n, h, seed)
    s = dict(case=case, geom=_geom(n, h), lo=lo, hi=hi)
    if kind in ("nodal", "eb_nodal"):
        vel = torch.zeros((3, n[2] + 2, n[1] + 2, n[0] + 2), **F64)
        vel[:, 1:-1, 1:-1, 1:-1] = v
        if lo[0] == I:
            vel[0, :, :, 0] = 1.0  # the inflow velocity in the ghost cells
        gp = torch.zeros((3, n[2], n[1], n[0]), **F64)
        if kind == "nodal":
            gp += 0.1 * _random_field(n, _generator(seed, 1))
        s |= dict(vel0=vel, vel=vel.clone(), rho=rho, gp0=gp, gp=gp.clone(), options=_options(case, 0),
                  p=torch.zeros((n[2] + 1, n[1] + 1, n[0] + 1), **F64), moments=None)
        if kind == "eb_nodal":
            s["moments"] = _keep(case, "cut", lambda: _cut_nodal(n, h))
        return s
    u = _faces(v, n, lo, hi)
    beta = 1.0 if kind == "eb_mac" or case["rho"] == "one" else _face_beta(rho, n, lo)

    def projector():
        mp = MacProjector(s["geom"], options=_options(case, 1))
        mp.initProjector(beta=beta)
        mp.setDomainBC(lo, hi)
        if kind == "eb_mac":
            mp.setEB(*_cut_mac(n, h))
        return mp

    return s | dict(mp=_keep(case, "projector", projector), beta=beta, u0=u, u=[x.clone() for x in u],
                    phi=torch.zeros((n[2], n[1], n[0]), **F64))


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind in ("nodal", "eb_nodal"):
        s["vel"].copy_(s["vel0"])
        s["gp"].copy_(s["gp0"])
        apply_nodal_projection(s["geom"], s["lo"], s["hi"], s["vel"], s["rho"], s["gp"], s["p"], options=s["options"],
                               set_inflow_bc=True, eb_moments=s["moments"])
        return dict(vel=s["vel"], gp=s["gp"], p=s["p"])
    if kind in ("mac", "eb_mac"):
        for a, b in zip(s["u"], s["u0"]):
            a.copy_(b)
        mp = s["mp"]
        if isinstance(s["beta"], float):
            mp.updateBeta(s["beta"])
        else:
            mp.updateCoeffs(s["beta"])
        mp.setUMAC(s["u"])
        mp.project(rtol=case["rtol"], atol=0.0, phi=s["phi"], phi_guess=False)
        return dict(u=s["u"], phi=s["phi"])
    if kind == "amr":
        s["vel"].copy_(s["vel0"])
        s["vel_f"].copy_(s["vel_f0"])
        s["gp"].zero_()
        s["gp_f"].zero_()
        v, r, g, p = s["fabs"]
        s["proj"].apply(s["vel"], s["rho"], s["gp"], s["p"], v, r, g, p)
        return dict(vel=s["vel"], gp=s["gp"], p=s["p"], vel_f=s["vel_f"], gp_f=s["gp_f"], p_f=s["p_f"])
    if kind == "tensor":
        op = s["op"]
        s["vel"].copy_(s["vel0"])
        op.setACoeffs(0, s["rho"])
        op.setShearViscosity(0, s["eta"])
        op.solve(s["vel"], s["rhs"], rtol=case["rtol"], atol=0.0)
        return s["vel"]
    loss = s["net"].train_pair(s["x"], s["t"], s["n"], s["n"], lr=0.0)
    return dict(loss=loss, grads=s["net"].grads(), out=s["net"].predict(s["x"], s["n"]))


def work(case):
    """Bytes of the fields that a call is given and returns, once each. Operations: for a solve one right-hand side,
    one application of the operator and one correction; for the network its convolutions."""
    kind = case["kind"]
    if kind == "unet":
        v = case["nx"] * case["ny"] * case["nz"]
        c = [16, 32, 64, 128]
        f = 0.0
        for lev in range(4):
            f += (27 * c[lev] * ((16 if lev == 0 else c[lev - 1]) + c[lev])) * v / 8 ** lev
        for lev in range(3):
            f += (27 * c[lev] * (c[lev + 1] + c[lev] + c[lev])) * v / 8 ** lev
        f += 16 * 16 * v
        # forward, the two gradients of training, and the forward of the prediction
        return dict(bytes=2.0 * v * 16 * 2 + 4 * v, flops=2.0 * f * 4)
    n, h, lo, hi = _grid(case)
    c = float(n[0]) * n[1] * n[2]
    if kind == "amr":
        c += 8.0 * 0.26 * c
    per = {"nodal": (3 + 3 + 1 + 3 + 3 + 1, 60), "eb_nodal": (3 + 1 + 3 + 3 + 1, 60), "amr": (3 + 1 + 3 + 3 + 1, 60),
           "mac": (3 + 3 + 3 + 1, 30), "eb_mac": (3 + 3 + 1, 30), "tensor": (3 + 1 + 1 + 3 + 3, 200)}[kind]
    return dict(bytes=8.0 * per[0] * c, flops=per[1] * c)


# ------------------------------------------------------------------------------------------------ 64-bit values
def _pairs(n, lo, hi, h, nodal):
    """1-D stiffness and mass of one direction (unique unknowns; Dirichlet nodes are left out by the mask)"""
    m = n if lo == P or not nodal else n + 1
    K, M = torch.zeros((m, m), **F64), torch.zeros((m, m), **F64)
    i = torch.arange(n, device="cuda")
    if nodal:
        j = (i + 1) % m
        one = torch.ones(n, **F64)
        for a, b, k, w in ((i, i, 1, 2), (j, j, 1, 2), (i, j, -1, 1), (j, i, -1, 1)):
            K.index_put_((a, b), k / h * one, accumulate=True)
            M.index_put_((a, b), w * h / 6.0 * one, accumulate=True)
        return K, M
    M += torch.eye(n, **F64) * h
    f = i if lo == P else i[:-1]
    j, one = (f + 1) % n, torch.ones(len(f), **F64) / h
    for a, b, k in ((f, f, 1), (j, j, 1), (f, j, -1), (j, f, -1)):
        K.index_put_((a, b), k * one, accumulate=True)
    for side, at in ((lo, 0), (hi, n - 1)):
        if side == D:
            K[at, at] += 2.0 / h
    return K, M


class _Separable:
    """the inverse of shift M x M x M + sum_d w_d (K_d with M elsewhere) by the directions' eigenvectors"""

    def __init__(self, n, h, lo, hi, nodal, weights=(1.0, 1.0, 1.0), shift=0.0):
        self.V, lam, self.free = [], [], []
        for d in range(3):
            K, M = _pairs(n[d], lo[d], hi[d], h[d], nodal)
            m = K.shape[0]
            free = torch.ones(m, dtype=torch.bool, device="cuda")
            if nodal:
                free[0] &= lo[d] != D
                free[-1] &= hi[d] != D
            L = torch.linalg.cholesky(M[free][:, free])
            A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, K[free][:, free], upper=False).T,
                                              upper=False)
            w, Q = torch.linalg.eigh(0.5 * (A + A.T))
            V = torch.zeros((m, len(w)), **F64)
            V[free] = torch.linalg.solve_triangular(L.T, Q, upper=True)
            self.V.append(V)
            lam.append(weights[d] * w)
            self.free.append(free)
        s = shift + lam[0][None, None, :] + lam[1][None, :, None] + lam[2][:, None, None]
        self.inv = torch.where(s > 1e-10 * s.max(), 1.0 / s.clamp(min=1e-300), torch.zeros_like(s))
        f = self.free
        self.mask = (f[2][:, None, None] & f[1][None, :, None] & f[0][None, None, :]).double()

    def __call__(self, r):
        V = self.V
        t = (r.reshape(-1, r.shape[2]) @ V[0]).view(r.shape[0], r.shape[1], -1)
        t = torch.matmul(V[1].T, t)
        t = (V[2].T @ t.reshape(t.shape[0], -1)).view(-1, t.shape[1], t.shape[2])
        t = t * self.inv
        t = (V[2] @ t.reshape(t.shape[0], -1)).view(-1, t.shape[1], t.shape[2])
        t = torch.matmul(V[1], t)
        return (t.reshape(-1, t.shape[2]) @ V[0].T).view(t.shape[0], t.shape[1], -1)


def _cg(A, b, Minv, rtol=3e-14, most=4000):
    """preconditioned conjugate gradients; on reaching rounding the last iterate"""
    x, r = torch.zeros_like(b), b.clone()
    z = Minv(r)
    p, rz = z.clone(), (r * z).sum()
    b2, best, stale = float((b * b).sum()), math.inf, 0
    for q in range(most):
        Ap = A(p)
        a = rz / (p * Ap).sum()
        x += a * p
        if q % 50 == 49:
            r = b - A(x)
        else:
            r -= a * Ap
        if q % 5 == 4:
            r2 = float((r * r).sum())
            if r2 <= rtol * rtol * b2:
                break
            stale = 0 if r2 < 0.5 * best else stale + 1
            best = min(best, r2)
            if stale > 200:
                break
        z = Minv(r)
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _split(t, ax):
    """sums and differences of neighbours along an axis"""
    n = t.shape[ax] - 1
    a, b = t.narrow(ax, 0, n), t.narrow(ax, 1, n)
    return a + b, b - a


def _join(s, d, ax):
    """the transpose of _split"""
    shape = list(s.shape)
    shape[ax] += 1
    out = torch.zeros(shape, **F64)
    n = s.shape[ax]
    out.narrow(ax, 0, n).add_(s).sub_(d)
    out.narrow(ax, 1, n).add_(s).add_(d)
    return out


class _Nodal:
    """div(sigma grad phi) on trilinear elements: on each cell the element matrix is diagonal in the sums and
    differences of the corner values along x, y and z (1-D mass s^2 h / 4 + d^2 h / 12, stiffness d^2 / h)"""

    def __init__(self, n, h, lo, hi, sigma):
        self.n, self.h, self.per, self.sigma = n, h, [b == P for b in lo], sigma
        V = h[0] * h[1] * h[2]
        self.V = V
        self.w = {}
        for m in range(1, 8):
            f = [(1.0 / 12.0 if (m >> d) & 1 else 0.25) for d in range(3)]
            self.w[m] = V * sum((1.0 / h[d] ** 2) * f[0] * f[1] * f[2] / f[d] for d in range(3) if (m >> d) & 1)

    def extend(self, t):
        for d in range(3):
            if self.per[d]:
                t = torch.cat([t, t.narrow(2 - d, 0, 1)], dim=2 - d)
        return t

    def fold(self, t):
        for d in range(3):
            if self.per[d]:
                k = self.n[d]
                t.narrow(2 - d, 0, 1).add_(t.narrow(2 - d, k, 1))
                t = t.narrow(2 - d, 0, k)
        return t

    def modes(self, phi):
        out = {0: self.extend(phi)}
        for d in range(3):
            out = {m | (q << d): v for m, t in out.items() for q, v in enumerate(_split(t, 2 - d))}
        return out

    def gather(self, modes):
        zero = None
        for d in (2, 1, 0):
            new = {}
            for m in {k & ~(1 << d) for k in modes}:
                s, t = modes.get(m), modes.get(m | (1 << d))
                zero = torch.zeros_like(s if s is not None else t)
                new[m] = _join(s if s is not None else zero, t if t is not None else zero, 2 - d)
            modes = new
        return self.fold(modes[0])

    def apply(self, phi):
        m = self.modes(phi)
        return self.gather({k: self.w[k] * self.sigma * m[k] for k in range(1, 8)})

    def divergence(self, vel):
        return self.gather({1 << d: vel[d] * (self.V / (4.0 * self.h[d])) for d in range(3)})

    def grad(self, phi):
        m = self.modes(phi)
        return torch.stack([m[1 << d] / (4.0 * self.h[d]) for d in range(3)])

    def dual(self):
        m = {0: torch.full((self.n[2], self.n[1], self.n[0]), self.V / 8.0, **F64)}
        return self.gather(m)


def _exact_nodal(case, seed):
    n, h, lo, hi = _grid(case)
    v, rho = _velocity(n, h, lo, hi, seed), _density(case, n, h, seed)
    gp = 0.1 * _random_field(n, _generator(seed, 1))
    sigma = 1.0 / rho
    op = _Nodal(n, h, lo, hi, sigma)
    v = v + sigma * gp
    b = op.divergence(v)
    if lo[0] == I:  # the unit inflow through the low x side
        s = torch.zeros((n[2], n[1]), **F64) + h[1] * h[2] / 4.0
        face = _join(_join(s, torch.zeros_like(s), 1), torch.zeros((n[2], n[1] + 1), **F64), 0)
        for d, ax in ((1, 1), (2, 0)):
            if op.per[d]:
                face.narrow(ax, 0, 1).add_(face.narrow(ax, n[d], 1))
                face = face.narrow(ax, 0, n[d])
        b[:, :, 0] += face
    pre = _Separable(n, h, lo, hi, True)
    vol = op.dual()
    singular = D not in lo + hi
    if singular:
        b -= vol * (b.sum() / vol.sum())
    b = b * pre.mask
    phi = _cg(lambda x: op.apply(x) * pre.mask, b, pre)
    if singular:
        phi = phi - (vol * phi).sum() / vol.sum()
    g = op.grad(phi)
    vel = torch.zeros((3, n[2] + 2, n[1] + 2, n[0] + 2), **F64)
    if lo[0] == I:
        vel[0, :, :, 0] = 1.0
    vel[:, 1:-1, 1:-1, 1:-1] = v - sigma * g
    return dict(vel=vel, gp=g, p=op.extend(phi))


class _Faces:
    """cell-centred fluxes: the differences of phi across the faces of each direction, and their divergence"""

    def __init__(self, n, h, lo, hi):
        self.n, self.h, self.lo, self.hi = n, h, lo, hi

    def diff(self, phi, d):
        ax, n = 2 - d, self.n[d]
        a, z = phi.narrow(ax, 0, 1), phi.narrow(ax, n - 1, 1)
        mid = phi.narrow(ax, 1, n - 1) - phi.narrow(ax, 0, n - 1)
        first = a - z if self.lo[d] == P else 2.0 * a if self.lo[d] == D else 0.0 * a
        last = a - z if self.lo[d] == P else -2.0 * z if self.hi[d] == D else 0.0 * z
        return torch.cat([first, mid, last], dim=ax) / self.h[d]

    def div(self, u):
        return sum((u[d].narrow(2 - d, 1, self.n[d]) - u[d].narrow(2 - d, 0, self.n[d])) / self.h[d] for d in range(3))


def _exact_mac(case, seed):
    n, h, lo, hi = _grid(case)
    v, rho = _velocity(n, h, lo, hi, seed), _density(case, n, h, seed)
    u, beta = _faces(v, n, lo, hi), _face_beta(rho, n, lo)
    f = _Faces(n, h, lo, hi)
    V = h[0] * h[1] * h[2]
    b = -V * f.div(u)
    singular = D not in lo + hi
    if singular:
        b -= b.mean()
    phi = _cg(lambda x: -V * f.div([beta[d] * f.diff(x, d) for d in range(3)]), b, _Separable(n, h, lo, hi, False))
    if singular:
        phi = phi - phi.mean()
    return dict(u=[u[d] - beta[d] * f.diff(phi, d) for d in range(3)], phi=phi)


def _exact_eb_nodal(case, seed):
    """the element matrices of the cut cells from the moments of their fluid part; conjugate gradients with the
    operator's diagonal"""
    n, h, lo, hi = _grid(case)
    M = _cut_nodal(n, h)
    v = 1e-3 * (2.0 * torch.rand((3, n[2], n[1], n[0]), generator=_generator(seed), **F64) - 1.0)
    v[0] += 1.0
    kap, V = M[0], h[0] * h[1] * h[2]
    regular = (kap >= 1.0 - 1e-12).double()
    cut = (kap > 1e-12) & (kap < 1.0 - 1e-12)
    Mc = M[:, cut]
    sgn = [[1.0 if (a >> d) & 1 else -1.0 for d in range(3)] for a in range(8)]
    K = torch.zeros((8, 8, Mc.shape[1]), **F64)
    G, Gc = torch.zeros((8, 3, Mc.shape[1]), **F64), torch.zeros((8, 3, Mc.shape[1]), **F64)
    cen = [Mc[k] / Mc[0] for k in (1, 3, 9)]
    step = (1, 3, 9)
    for a in range(8):
        for d in range(3):
            e, f = [t for t in range(3) if t != d]
            G[a, d] = sgn[a][d] / h[d] * V * (0.25 * Mc[0] + 0.5 * (sgn[a][e] * Mc[step[e]] + sgn[a][f] * Mc[step[f]])
                                              + sgn[a][e] * sgn[a][f] * Mc[step[e] + step[f]])
            Gc[a, d] = sgn[a][d] / h[d] * (0.5 + sgn[a][e] * cen[e]) * (0.5 + sgn[a][f] * cen[f])
            for b in range(8):
                ce = (0.25, 0.5 * (sgn[a][e] + sgn[b][e]), sgn[a][e] * sgn[b][e])
                cf = (0.25, 0.5 * (sgn[a][f] + sgn[b][f]), sgn[a][f] * sgn[b][f])
                K[a, b] += sgn[a][d] * sgn[b][d] / h[d] ** 2 * V * sum(
                    ce[p] * cf[q] * Mc[p * step[e] + q * step[f]] for p in range(3) for q in range(3))
    op = _Nodal(n, h, lo, hi, regular)
    kk, jj, ii = torch.nonzero(cut, as_tuple=True)
    wrap = [op.n[d] if op.per[d] else n[d] + 1 for d in range(3)]
    corner = torch.stack([((kk + (a >> 2)) % wrap[2] * wrap[1] + (jj + ((a >> 1) & 1)) % wrap[1]) * wrap[0]
                          + (ii + (a & 1)) % wrap[0] for a in range(8)])

    def apply(x):
        y = op.apply(x).contiguous()
        y.view(-1).index_add_(0, corner.reshape(-1), torch.einsum("abc,bc->ac", K, x.reshape(-1)[corner]).reshape(-1))
        return y * free

    shape = (wrap[2], wrap[1], wrap[0])
    fluid = _Nodal(n, h, lo, hi, None).gather({0: (kap > 1e-12).double()})
    free = (fluid > 0).double()
    free[:, :, -1] = 0.0  # the outflow
    k0 = V * sum(1.0 / h[d] ** 2 for d in range(3)) / 9.0
    diag = op.gather({0: regular * k0}).contiguous()
    diag.view(-1).index_add_(0, corner.reshape(-1), torch.stack([K[a, a] for a in range(8)]).reshape(-1))
    diag = torch.where(free > 0, 1.0 / diag.clamp(min=1e-300), torch.zeros_like(diag))
    b = op.divergence(v * regular).contiguous()
    vc = torch.stack([v[d][cut] for d in range(3)])
    b.view(-1).index_add_(0, corner.reshape(-1), torch.einsum("adc,dc->ac", G, vc).reshape(-1))
    s = torch.full((n[2], n[1]), h[1] * h[2] / 4.0, **F64)
    face = _join(_join(s, torch.zeros_like(s), 1), torch.zeros((n[2], n[1] + 1), **F64), 0)
    face[0] += face[n[2]]
    b[:, :, 0] += face[:n[2]]
    b = b * free
    phi = _cg(apply, b, lambda r: r * diag, most=6000).view(shape)
    g = op.grad(phi)
    gc = torch.einsum("adc,ac->dc", Gc, phi.reshape(-1)[corner])
    for d in range(3):
        g[d][cut] = gc[d]
    g = g * (kap > 1e-12)
    vel = torch.zeros((3, n[2] + 2, n[1] + 2, n[0] + 2), **F64)
    vel[0, :, :, 0] = 1.0
    vel[:, 1:-1, 1:-1, 1:-1] = v - g
    return dict(vel=vel, gp=g, p=op.extend(phi))


def _exact_eb_mac(case, seed):
    """fluxes at the centroids of the cut faces (bilinear in the neighbouring open faces); conjugate gradients on
    the face-centre fluxes inside a correction for the difference"""
    n, h, lo, hi = _grid(case)
    kap, ap, fc = _cut_mac(n, h)
    v = 1e-3 * (2.0 * torch.rand((3, n[2], n[1], n[0]), generator=_generator(seed), **F64) - 1.0)
    v[0] += 1.0
    u = _faces(v, n, lo, hi)
    f = _Faces(n, h, lo, hi)
    V = h[0] * h[1] * h[2]

    def shift(t, ax, d, s):
        """t at the neighbour one face towards s; 0 past a side that is not periodic"""
        r = torch.roll(t, -s, ax)
        if lo[d] != P:
            r.narrow(ax, t.shape[ax] - 1 if s > 0 else 0, 1).zero_()
        return r

    def centroid(df, d):
        ta, tb = [t for t in range(3) if t != d]
        a, cut = ap[d], ((ap[d] > 0) & (ap[d] < 1)).clone()
        if lo[d] != P:
            cut.narrow(2 - d, 0, 1).zero_()
            cut.narrow(2 - d, n[d], 1).zero_()
        oa, ob = fc[d][0], fc[d][1]
        out = df.clone()
        for sa in (1, -1):
            for sb in (1, -1):
                sel = cut & ((oa >= 0) == (sa > 0)) & ((ob >= 0) == (sb > 0))
                a1, a2 = shift(a, 2 - ta, ta, sa), shift(a, 2 - tb, tb, sb)
                a12 = shift(a1, 2 - tb, tb, sb)
                d1, d2 = shift(df, 2 - ta, ta, sa), shift(df, 2 - tb, tb, sb)
                d12 = shift(d1, 2 - tb, tb, sb)
                w1 = torch.where(a1 > 0, oa.abs(), torch.zeros_like(a))
                w2 = torch.where(a2 > 0, ob.abs(), torch.zeros_like(a))
                w2 = torch.where((w1 > 0) & (w2 > 0) & (a12 <= 0), torch.zeros_like(a), w2)
                val = (1 - w1) * (1 - w2) * df + w1 * (1 - w2) * d1 + (1 - w1) * w2 * d2 + w1 * w2 * d12
                out = torch.where(sel, val, out)
        return out

    open_ = [(a > 0).double() for a in ap]
    fluid = (kap > 0).double()

    def apply(x, exact):
        df = [f.diff(x, d) * open_[d] for d in range(3)]
        return -V * f.div([ap[d] * (centroid(df[d], d) if exact else df[d]) for d in range(3)]) * fluid

    diag = sum((V / h[d] ** 2) * (ap[d].narrow(2 - d, 1, n[d]) + ap[d].narrow(2 - d, 0, n[d])) for d in range(3))
    diag = torch.where(kap > 0, 1.0 / diag.clamp(min=1e-300), torch.zeros_like(kap))
    b = -V * f.div([ap[d] * u[d] for d in range(3)]) * fluid
    phi, r = torch.zeros_like(b), b.clone()
    b2 = float((b * b).sum())
    for _ in range(24):
        phi = phi + _cg(lambda x: apply(x, False), r, lambda t: t * diag, rtol=2e-2)
        r = b - apply(phi, True)
        if float((r * r).sum()) < 1e-26 * b2:
            break
    grad = [centroid(f.diff(phi, d) * open_[d], d) for d in range(3)]
    return dict(u=[u[d] - grad[d] for d in range(3)], phi=phi)


def _exact_tensor(case, seed):
    n, h, rho, eta, v = _tensor_fields(case, seed)
    beta = 0.5 * h[0]
    wall = [v[:, 1:-1, 0, 1:-1], v[:, 1:-1, -1, 1:-1]]
    ef = []
    for d in range(3):
        ax = 2 - d
        first, last = eta.narrow(ax, 0, 1), eta.narrow(ax, n[d] - 1, 1)
        mid = 0.5 * (eta.narrow(ax, 1, n[d] - 1) + eta.narrow(ax, 0, n[d] - 1))
        ends = (0.5 * (first + last),) * 2 if d != 1 else (first, last)
        ef.append(torch.cat([ends[0], mid, ends[1]], dim=ax))

    def apply(u, walls):
        w = torch.zeros((3, n[2] + 2, n[1] + 2, n[0] + 2), **F64)
        w[:, 1:-1, 1:-1, 1:-1] = u
        lo, hi = (wall[0], wall[1]) if walls else (0.0, 0.0)
        w[:, 1:-1, 0, 1:-1] = 2.0 * lo - u[:, :, 0]
        w[:, 1:-1, -1, 1:-1] = 2.0 * hi - u[:, :, -1]
        w[..., 0], w[..., -1] = w[..., -2].clone(), w[..., 1].clone()
        w[:, 0], w[:, -1] = w[:, -2].clone(), w[:, 1].clone()
        out = rho * u
        for d in range(3):
            def cells(s, e=None, t=0):
                sl = [slice(None)] + [slice(1, n[q] + 1) for q in (2, 1, 0)]
                sl[3 - d] = slice(s, s + n[d] + 1)
                if e is not None:
                    sl[3 - e] = slice(1 + t, 1 + t + n[e])
                return w[tuple(sl)]
            norm = (cells(1) - cells(0)) / h[d]
            tang = {e: (cells(0, e, 1) - cells(0, e, -1) + cells(1, e, 1) - cells(1, e, -1)) / (4.0 * h[e])
                    for e in range(3) if e != d}
            for c in range(3):
                if c == d:
                    fl = ef[d] * ((4.0 / 3.0) * norm[d] - (2.0 / 3.0) * sum(t[e] for e, t in tang.items()))
                else:
                    fl = ef[d] * (norm[c] + tang[c][d])
                out[c] -= beta * (fl.narrow(2 - d, 1, n[d]) - fl.narrow(2 - d, 0, n[d])) / h[d]
        return out

    zero = torch.zeros((3, n[2], n[1], n[0]), **F64)
    rhs = rho[None] * v[:, 1:-1, 1:-1, 1:-1] - apply(zero, True)
    V = h[0] * h[1] * h[2]
    pre = [_Separable(n, h, (P, D, P), (P, D, P), False, [0.015 * beta * (4.0 / 3.0 if c == d else 1.0) for d in range(3)],
                      1.5) for c in range(3)]

    def inverse(r):
        return torch.stack([pre[c](V * r[c]) / V for c in range(3)]) * V

    # stabilised biconjugate gradients (the wall rows are not symmetric)
    x, r = torch.zeros_like(rhs), rhs.clone()
    r0, p, b2 = r.clone(), r.clone(), float((rhs * rhs).sum())
    rho_k = (r0 * r).sum()
    for _ in range(200):
        y = inverse(p)
        q = apply(y, False)
        a = rho_k / (r0 * q).sum()
        s = r - a * q
        z = inverse(s)
        t = apply(z, False)
        w = (t * s).sum() / (t * t).sum()
        x = x + a * y + w * z
        r = s - w * t
        if float((r * r).sum()) < 1e-27 * b2:
            break
        new = (r0 * r).sum()
        p = r + (new / rho_k) * (a / w) * (p - w * q)
        rho_k = new
    out = v.clone()
    out[:, 1:-1, 1:-1, 1:-1] = x
    return out


def _exact_unet(case, seed):
    s = prepare(case, seed)
    n = s["n"]
    x = s["x"].view(n[2] + 2, n[1] + 2, n[0] + 2, 16)[1:-1, 1:-1, 1:-1].permute(3, 0, 1, 2)[None].double()
    t = s["t"].view(n[2] + 2, n[1] + 2, n[0] + 2)[1:-1, 1:-1, 1:-1].double()
    theta = torch.from_numpy(s["net"].params()).cuda().double()
    c = [16, 32, 64, 128]
    spec = []
    for lev in range(4):
        spec += [(16 if lev == 0 else c[lev - 1], c[lev], 3), (c[lev], c[lev], 3)]
    for lev in (2, 1, 0):
        spec += [(c[lev + 1] + c[lev], c[lev], 3), (c[lev], c[lev], 3)]
    spec.append((16, 16, 1))
    par, at = [], 0
    for ci, co, k in spec:
        w = theta[at:at + k ** 3 * co * ci].bfloat16().double().requires_grad_()
        at += k ** 3 * co * ci
        par += [w, theta[at:at + co].clone().requires_grad_()]
        at += co

    def conv(h, q):
        ci, co, k = spec[q]
        w = par[2 * q].view(k, k, k, co, ci).permute(3, 4, 0, 1, 2)
        return torch.nn.functional.conv3d(h, w, par[2 * q + 1], padding=k // 2)

    def block(h, q):
        f = torch.nn.functional
        return f.gelu(conv(f.gelu(conv(h, q), approximate="tanh"), q + 1), approximate="tanh")

    skips, h = [], x
    for lev in range(4):
        if lev:
            h = torch.nn.functional.avg_pool3d(h, 2)
        h = block(h, 2 * lev)
        skips.append(h)
    for q, lev in enumerate((2, 1, 0)):
        up = h.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
        h = block(torch.cat([up, skips[lev]], dim=1), 8 + 2 * q)
    out = conv(h, 14)
    loss = ((out[0, 0] - t) ** 2).mean()
    loss.backward()
    rows = torch.zeros((n[2] + 2, n[1] + 2, n[0] + 2, 16), **F64)
    rows[1:-1, 1:-1, 1:-1] = out.detach()[0].permute(1, 2, 3, 0)
    return dict(loss=float(loss.detach()), grads=torch.cat([p.grad.reshape(-1) for p in par]), out=rows.reshape(-1, 16))


def exact(case, seed):
    """None for the two levels: without a multigrid of its own a solve of that size takes minutes."""
    if case["kind"] == "amr":
        return None
    return {"nodal": _exact_nodal, "mac": _exact_mac, "eb_nodal": _exact_eb_nodal, "eb_mac": _exact_eb_mac,
            "tensor": _exact_tensor, "unet": _exact_unet}[case["kind"]](case, seed)
