"""The transforms at the edges of their variants, against the FP64 oracle.

Forward (x-pass, y-pass with the window, interpolation) of real and complex
images: grids n0 = 32 (shared-memory x-pass) to 8192 and n1 = 16 to 2048, so that
every half-length and full-length x-kernel, both y-kernels and every number of
slices a group can have run, with image sides and slice counts that fill no
tile of the layout kernels.  Bound 1e-5: the window is evaluated in float as
the reference does, u = n x with a rounding of 2^-24 n |x|, 3e-5 for n = 1024 and
a slope of phi of at most 0.3 per grid unit; sides of 4096 points and more have
4 and 8 times that, 4e-5 and 8e-5.

Toeplitz iteration from a random start: y lengths of every register FFT (32 times
4, 6, 8, 10, 12, 16, 20, 24 and 32) and the shared-memory FFT above, the half
spectrum of a real image and x-kernels of every number of slices a CTA takes,
against one iteration with the exact transform.  Bound 1e-5 as for the tests of
the operator: float rounding of transforms of at most 2^13 x 2^11 points.
"""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_toeplitz import _exact_iteration

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TILTS = np.array([-63.0, -40.5, -7.0, 0.25, 31.0, 66.0], np.float32)


@pytest.mark.parametrize("nx,th,S", [
    (12, 8, 1), (12, 8, 9), (30, 20, 3), (33, 40, 8), (64, 130, 11), (100, 61, 2), (150, 33, 4), (260, 129, 5),
    (257, 100, 1), (520, 48, 9), (640, 9, 2), (1030, 24, 3), (2050, 9, 2), (70, 513, 4), (60, 600, 9)])
@pytest.mark.parametrize("cplx,window", [(False, "gauss6"), (True, "kb4")])
def test_forward_matches_fp64_oracle(nx, th, S, cplx, window):
    from feilab_b200.icon import IconPlan
    from oracle.oracle import OraclePlan
    p = IconPlan(nx, th, TILTS, capacity=S, window=window)
    o = OraclePlan(nx, th, TILTS, "f64", window=window)
    rng = np.random.default_rng(nx * th + S)
    img = rng.standard_normal((S, nx, th)).astype(np.float32)
    if cplx:
        img = (img + 1j * rng.standard_normal((S, nx, th))).astype(np.complex64)
    d = torch.from_numpy(img).cuda()
    f = p.nufft_forward(d)
    assert torch.equal(f, p.nufft_forward(d))
    f = f.cpu().numpy()
    tol = 1e-5 * max(1, 2 * nx // 1024)
    for s in {0, S // 2, S - 1}:
        assert rel_l2(f[s], o.forward(img[s].astype(np.complex128 if cplx else np.float64))) < tol, s


@pytest.mark.parametrize("nx,th,S", [
    (24, 50, 1), (24, 60, 4), (40, 90, 9), (24, 125, 2), (24, 150, 8), (24, 190, 3), (24, 250, 1), (24, 300, 9),
    (24, 380, 2), (24, 500, 4), (24, 530, 8), (24, 530, 1), (130, 20, 9), (260, 20, 9), (520, 20, 9), (520, 20, 2),
    (1030, 12, 4)])
def test_toeplitz_iteration_matches_exact_transform(nx, th, S):
    from feilab_b200.icon import IconPlan
    from oracle.oracle import OraclePlan
    o = OraclePlan(nx, th, TILTS, "f64")
    w = o.geometry()[1].astype(np.float64)
    rng = np.random.default_rng(nx + th + S)
    m0 = rng.standard_normal((S, nx, th)).astype(np.float32)
    Ahwb = (rng.standard_normal((S, nx, th)) + 1j * rng.standard_normal((S, nx, th))).astype(np.complex64)
    p = IconPlan(nx, th, TILTS, capacity=S)
    p.set_operator("toeplitz")
    m1, al, rt = p.solve(torch.from_numpy(Ahwb).cuda(), (1, 0, 0), 2, 0.0, m0=torch.from_numpy(m0).cuda(), history=True)
    m1 = m1.cpu().numpy()
    for s in {0, S - 1}:
        me, ale, rte = _exact_iteration(o, w, m0[s], Ahwb[s].astype(np.complex128))
        assert rel_l2(m1[s], me) < 1e-5, s
        assert abs(al[0, s] - ale) <= 1e-5 * abs(ale)
        assert abs(rt[0, s] - rte) <= 1e-5 * abs(rte)
