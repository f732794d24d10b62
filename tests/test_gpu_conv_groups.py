"""BF16 convolutions with several voxels per GEMM row (grids whose planes split into groups of 2 or 4 voxels) against
PyTorch FP32, with the tolerances of test_gpu_nn.py: weights resident or with each step, one box for three rows of taps or
a box each (wide grids), several activation boxes per row (two inputs), flipped taps, weight gradients."""
import ctypes

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from tests.test_gpu_nn import _run, bf, close, conv, halo, ints, pad_cl, taps_fwd, unpad

pytestmark = pytest.mark.gpu

FORWARD = [
    ((16, 8, 24), [16], 16, 27), ((16, 8, 8), [16], 16, 1), ((8, 16, 8), [32, 16], 16, 27), ((8, 8, 16), [32], 32, 27),
    ((16, 8, 8), [64, 32], 32, 27), ((264, 8, 8), [16], 16, 27), ((136, 8, 8), [32], 64, 27), ((24, 8, 8), [16, 64], 16, 27),
]


@pytest.mark.parametrize("dims,cins,cout,ntaps", FORWARD, ids=[f"{c[0]}-{c[1]}-{c[2]}-{c[3]}" for c in FORWARD])
def test_forward(gpu_lib, dims, cins, cout, ntaps):
    torch.manual_seed(0)
    xs = [bf(torch.randn(c, dims[2], dims[1], dims[0], device="cuda")) for c in cins]
    k = 3 if ntaps == 27 else 1
    w = bf(torch.randn(cout, sum(cins), k, k, k, device="cuda") / np.sqrt(ntaps * sum(cins)))
    bias = torch.randn(cout, device="cuda") * 0.1
    ref = F.conv3d(torch.cat(xs)[None], w, bias, padding=k // 2)[0]
    (out,), _ = conv(gpu_lib, dims, [pad_cl(x) for x in xs], cins, taps_fwd(w), ntaps, cout, bias)
    torch.cuda.synchronize()
    close(unpad(out, cout, dims), ref)
    assert halo(out, cout, dims).abs().max().item() == 0.0


@pytest.mark.parametrize("dims,segs,cout", [((16, 8, 8), [16], 16), ((8, 24, 8), [32, 16], 16), ((264, 8, 8), [16], 16),
                                            ((8, 8, 16), [64, 32], 32)])
def test_data_gradient(gpu_lib, dims, segs, cout):
    torch.manual_seed(2)
    cin = sum(segs)
    w = bf(torch.randn(cout, cin, 3, 3, 3, device="cuda") / np.sqrt(27 * cin))
    g = bf(torch.randn(cout, dims[2], dims[1], dims[0], device="cuda"))
    ref = torch.nn.grad.conv3d_input((1, cin) + tuple(g.shape[1:]), w, g[None], padding=1)[0]
    wt = w.permute(2, 3, 4, 1, 0).reshape(27, cin, cout).to(torch.bfloat16).contiguous()
    outs = [pad_cl(torch.zeros(c, dims[2], dims[1], dims[0], device="cuda")) for c in segs]
    _run(gpu_lib, dims, [pad_cl(g)], [cout], wt, 27, cin, None, segs, outs, None, 0, 1)
    torch.cuda.synchronize()
    close(torch.cat([unpad(o, c, dims) for o, c in zip(outs, segs)]), ref)


@pytest.mark.parametrize("dims,cin,cout,ntaps", [((16, 8, 24), 16, 16, 27), ((8, 8, 8), 16, 32, 27), ((8, 16, 8), 32, 16, 27),
                                                 ((16, 8, 8), 32, 64, 27), ((16, 8, 8), 16, 16, 1), ((264, 8, 8), 16, 16, 27)])
def test_weight_gradient(gpu_lib, dims, cin, cout, ntaps):
    torch.manual_seed(3)
    x = bf(torch.randn(cin, dims[2], dims[1], dims[0], device="cuda"))
    g = bf(torch.randn(cout, dims[2], dims[1], dims[0], device="cuda"))
    k = 3 if ntaps == 27 else 1
    ref = torch.nn.grad.conv3d_weight(x[None], (cout, cin, k, k, k), g[None], padding=k // 2)
    ref = ref.permute(2, 3, 4, 0, 1).reshape(ntaps, cout, cin)
    dw = torch.zeros(ntaps, cout, cin, device="cuda")
    xp, gp = pad_cl(x), pad_cl(g)  # keep both alive across the call
    rc = gpu_lib.gbp_nn_conv3d_wgrad(ints(dims), ctypes.c_void_p(xp.data_ptr()), cin, 0, cin, ctypes.c_void_p(gp.data_ptr()),
                                     cout, ntaps, ctypes.c_void_p(dw.data_ptr()),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, gpu_lib.gbp_last_error().decode()
    torch.cuda.synchronize()
    assert (dw - ref).abs().max().item() <= 1e-4 * ref.abs().max().item() + 1e-4
