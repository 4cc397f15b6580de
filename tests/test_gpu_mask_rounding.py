"""Rounding of the mask's 2-D filtering against 64 bits, over the sizes of its
kernels.  The relative L2 error of an FP32 FFT with accurate twiddles grows as
0.6 2^-24 sqrt(levels) (Gentleman and Sande 1966; levels: radix-2 levels, each with
a rounding of random sign), here 4 log2 n levels; bound 2^-24 sqrt(4 log2 n), which
leaves the filter's product and the separation of row pairs their share, and which
twiddles formed by products exceed (5.3e-7 at n = 512 against 3.6e-7).
"""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_mask_rounding(n):
    from feilab_b200 import tools
    m = tools.Mask(n, np.linspace(-60, 60, 41).astype(np.float32), 0.125, 0.0, True, capacity=2)
    x = torch.randn(2, n, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    got = m.apply(x, 0, n).cpu().numpy()
    f = torch.from_numpy(m.filter().astype(np.float64)).cuda()
    ref = torch.fft.irfft2(torch.fft.rfft2(x.double()) * f, s=(n, n)).cpu().numpy()
    assert rel_l2(got, ref) < 2.0**-24 * np.sqrt(4 * np.log2(n))
