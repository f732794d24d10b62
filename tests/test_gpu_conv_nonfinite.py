"""BF16 convolutions of inputs that are not finite everywhere: a NaN or infinite voxel reaches the voxels of its 3x3x3
neighbourhood and no others, whatever the number of voxels per GEMM row (grids that split into groups of 4, 2 or not)."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from tests.test_gpu_nn import GELU, _run, bf, close, conv, halo, pad_cl, taps_fwd, unpad

pytestmark = pytest.mark.gpu

CASES = [((16, 8, 24), [16], 16, 27), ((16, 8, 8), [16], 16, 1), ((8, 16, 8), [32, 16], 16, 27), ((8, 8, 16), [32], 32, 27),
         ((136, 8, 8), [32], 64, 27), ((264, 8, 8), [16], 16, 27), ((9, 7, 5), [16], 16, 27), ((8, 8, 8), [64], 64, 27)]
SPOTS = [(0, 0, 0), (3, 4, 5), (7, 6, 4), (6, 0, 2)]  # x, y, z: a corner, the middle, the end of a row (8), a side


def _compare(out, ref, spots, dims, ntaps):
    """non-finite where a spot is within reach, as close as ever elsewhere"""
    r = 1 if ntaps == 27 else 0
    reach = torch.zeros(dims[2], dims[1], dims[0], dtype=torch.bool, device="cuda")
    for x, y, z in spots:
        reach[max(z - r, 0):z + r + 1, max(y - r, 0):y + r + 1, max(x - r, 0):x + r + 1] = True
    assert not torch.isfinite(out[:, reach]).any()
    assert torch.isfinite(out[:, ~reach]).all()
    close(torch.where(reach, torch.zeros_like(out), out), torch.where(reach, torch.zeros_like(ref), ref))


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")], ids=["nan", "inf", "-inf"])
@pytest.mark.parametrize("dims,cins,cout,ntaps", CASES, ids=[f"{c[0]}-{c[1]}-{c[2]}-{c[3]}" for c in CASES])
def test_forward(gpu_lib, dims, cins, cout, ntaps, value):
    torch.manual_seed(0)
    xs = [bf(torch.randn(c, dims[2], dims[1], dims[0], device="cuda")) for c in cins]
    k = 3 if ntaps == 27 else 1
    w = bf(torch.randn(cout, sum(cins), k, k, k, device="cuda") / np.sqrt(ntaps * sum(cins)))
    w = torch.where(w == 0, torch.full_like(w, 0.01), w)  # 0 x inf is NaN: every tap counts
    w = bf(w)
    spots = [tuple(min(s[d], dims[d] - 1) for d in range(3)) for s in SPOTS]
    ref = F.conv3d(torch.cat(xs)[None], w, padding=k // 2)[0]
    for x, y, z in spots:
        xs[0][5, z, y, x] = value
    (out,), _ = conv(gpu_lib, dims, [pad_cl(x) for x in xs], cins, taps_fwd(w), ntaps, cout)
    torch.cuda.synchronize()
    _compare(unpad(out, cout, dims), ref, spots, dims, ntaps)
    assert halo(out, cout, dims).abs().max().item() == 0.0


@pytest.mark.parametrize("dims,segs,cout", [((16, 8, 8), [16], 16), ((8, 24, 8), [32, 16], 16)])
def test_data_gradient(gpu_lib, dims, segs, cout):
    torch.manual_seed(2)
    cin = sum(segs)
    w = bf(torch.randn(cout, cin, 3, 3, 3, device="cuda") / np.sqrt(27 * cin))
    g = bf(torch.randn(cout, dims[2], dims[1], dims[0], device="cuda"))
    ref = torch.nn.grad.conv3d_input((1, cin) + tuple(g.shape[1:]), w, g[None], padding=1)[0]
    for x, y, z in SPOTS:
        g[3, z, y, x] = float("nan")
    wt = w.permute(2, 3, 4, 1, 0).reshape(27, cin, cout).to(torch.bfloat16).contiguous()
    outs = [pad_cl(torch.zeros(c, dims[2], dims[1], dims[0], device="cuda")) for c in segs]
    _run(gpu_lib, dims, [pad_cl(g)], [cout], wt, 27, cin, None, segs, outs, None, 0, 1)
    torch.cuda.synchronize()
    _compare(torch.cat([unpad(o, c, dims) for o, c in zip(outs, segs)]), ref, SPOTS, dims, 27)


def test_all_nan_and_bias(gpu_lib):
    """Every voxel NaN: NaN everywhere inside, zeros in the halo."""
    dims = (16, 8, 8)
    torch.manual_seed(1)
    w = bf(torch.randn(16, 16, 3, 3, 3, device="cuda") / np.sqrt(27 * 16))
    x = torch.full((16, dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    (out,), _ = conv(gpu_lib, dims, [pad_cl(x)], [16], taps_fwd(w), 27, 16, torch.randn(16, device="cuda"), flags=GELU)
    torch.cuda.synchronize()
    assert torch.isnan(unpad(out, 16, dims)).all() and halo(out, 16, dims).abs().max().item() == 0.0
