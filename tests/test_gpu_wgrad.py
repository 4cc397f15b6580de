"""Gradients of the warm-start network at image sizes where the tensor-core
weight gradients have ragged strips (widths off 64), shares of few rows and
borders on every side, against autograd of the FP32 mirror on the CPU, with the
bounds of the network's other gradient tests.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,thickness,S", [(200, 24, 2), (72, 136, 2), (130, 70, 3), (520, 33, 1)])
def test_gradients_match_fp32_mirror(nx, thickness, S):
    from test_gpu_warmstart import TOL_GRAD_ELEM, TOL_GRAD_REL, _mirror, _net_case, _split_params
    plan, net, Ahwb = _net_case(seed=23, nx=nx, thick=thickness, S=S)
    p, gain = net.get_params()
    target = torch.randn(Ahwb.shape, generator=torch.Generator(device="cuda").manual_seed(29), device="cuda").contiguous()
    net.backprop(Ahwb, target)
    grads = net.grads()
    net.backprop(Ahwb, target)
    assert np.array_equal(grads, net.grads())
    grads = _split_params(torch.from_numpy(grads))
    pt = torch.from_numpy(p).requires_grad_(True)
    _, y, sc, _ = _mirror(pt, Ahwb.cpu(), gain)
    t = target.cpu().transpose(1, 2) / (sc[:, None, None] * gain)
    ((y[:, :thickness, :nx] - t) ** 2).mean().backward()
    ref = _split_params(pt.grad.detach())
    for k in ref:
        a, b = grads[k].double(), ref[k].double()
        assert ((a - b).norm() / b.norm().clamp_min(1e-30)).item() < TOL_GRAD_REL, k
        assert (a - b).abs().max().item() <= TOL_GRAD_ELEM * b.abs().max().item() + 1e-12, k


@pytest.mark.parametrize("n,H,W,c0,c1,N,split", [
    (3, 9, 257, 16, 0, 16, 16),      # four-row tiles, a last row and a last column of one
    (1, 4, 128, 32, 16, 16, 16),     # concatenated input
    (2, 3, 130, 16, 0, 48, 32),      # two-row tiles, outputs split over two tensors
    (1, 1, 1, 64, 0, 32, 32),        # one pixel
    (2, 5, 127, 32, 0, 64, 64),
])
def test_small_layer_convolution_matches_fp32(n, H, W, c0, c1, N, split):
    # Bound: BF16 rounding of the outputs, 2^-9 relative each (2e-3 in norm),
    # doubled for the sums' own rounding: as the other convolution tests.
    from feilab_b200 import warmstart
    from test_gpu_warmstart import _close, _ref_conv
    g = torch.Generator(device="cuda").manual_seed(H * W + N)
    x0 = torch.randn((n, H, W, c0), generator=g, device="cuda").bfloat16()
    x1 = torch.randn((n, H, W, c1), generator=g, device="cuda").bfloat16() if c1 else None
    w = (torch.randn((9, N, c0 + c1), generator=g, device="cuda") / (3 * (c0 + c1) ** 0.5)).bfloat16()
    b = torch.randn((N,), generator=g, device="cuda")
    ref = _ref_conv(x0, x1, w, b, True)
    if split < N:
        o0, o1 = warmstart.conv3x3(x0, w, b, True, in1=x1, nsplit=split)
        _close(o0, ref[..., :split])
        _close(o1, ref[..., split:])
    else:
        _close(warmstart.conv3x3(x0, w, b, True, in1=x1), ref)
    assert warmstart.device_error() == 0
