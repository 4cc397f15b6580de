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
