"""The adjoint y-pass (row gather, then the FFT along y) against the FP64
oracle at the edges of its variants: every FFT length class (n1 = 16 and 64:
shared-memory FFT with idle threads; 128, 256, 512, 1024: register FFT; 2048:
shared-memory FFT, blocks of 1024 threads), every slice-group size, both
windows, rows without entries, and tilts up to 90 degrees, whose windows reach
the wrapped halo rows.

Bound 1e-5: the window is evaluated in float as the reference does, u = n x
with a rounding of 2^-24 n |x| <= 3e-5 for n = 1024 and a slope of phi of at
most 0.3 per grid unit; the FP32 sums and FFTs add about 1e-6.
"""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5
STEEP = np.array([-90.0, -71.3, -45.0, -10.0, 0.5, 33.0, 60.0, 88.9, 90.0], np.float32)
FEW = np.array([-1.0, 0.0, 1.5], np.float32)          # nearly all buffer rows without entries


@pytest.mark.parametrize("nx,th", [(24, 8), (40, 20), (33, 64), (96, 100), (50, 200), (64, 300), (130, 513)])
@pytest.mark.parametrize("S,window,tilts", [(1, "gauss6", STEEP), (2, "kb4", STEEP), (4, "gauss6", STEEP),
                                            (11, "gauss6", STEEP), (8, "kb4", FEW)])
def test_adjoint_matches_fp64_oracle(nx, th, S, window, tilts):
    from feilab_b200.icon import IconPlan
    from oracle.oracle import OraclePlan
    p = IconPlan(nx, th, tilts, capacity=S, window=window)
    o = OraclePlan(nx, th, tilts, "f64", window=window)
    rng = np.random.default_rng(7)
    f = (rng.standard_normal((S, p.M)) + 1j * rng.standard_normal((S, p.M))).astype(np.complex64)
    a = p.nufft_adjoint(torch.from_numpy(f).cuda())
    again = p.nufft_adjoint(torch.from_numpy(f).cuda())
    assert torch.equal(a, again)
    a = a.cpu().numpy()
    for s in {0, S // 2, S - 1}:
        assert rel_l2(a[s], o.adjoint(f[s].astype(np.complex128))) < TOL, s
