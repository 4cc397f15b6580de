"""The Toeplitz kernel at numbers of nodes that do not fill its chunks of 16, for
series whose last tilt is 0 (a half series, or an order that ends there: its
nodes lie on the axis x1 = 0).

One iteration from a random start against the FP64 NDFT, bound 1e-5 (float
rounding of the convolution and of the step length, as for other series), and at
a size whose kernel is summed in one range against the NUFFT operator (the
Gaussian window's error, 1e-6 per application, under the same bound).
"""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5


def _iteration(p, op, Ahwb, m0):
    p.set_operator(op)
    m, al, rt = p.solve(torch.from_numpy(Ahwb).cuda(), (1, 0, 0), 2, 0.0, m0=torch.from_numpy(m0).cuda(), history=True)
    return m.cpu().numpy(), al, rt


def _inputs(S, nx, th):
    rng = np.random.default_rng(nx + th)
    m0 = rng.standard_normal((S, nx, th)).astype(np.float32)
    return m0, (rng.standard_normal((S, nx, th)) + 1j * rng.standard_normal((S, nx, th))).astype(np.complex64)


@pytest.mark.parametrize("S", [1, 3, 9])
@pytest.mark.parametrize("nx,th,tilts", [
    (100, 9, np.linspace(-60, 0, 31)),       # 3100 nodes: 12 in the last chunk
    (40, 150, np.linspace(-60, 0, 13)),      # 520: 8
    (33, 20, np.linspace(50, 0, 9)),         # 297: 9
    (64, 48, np.linspace(-60, 0, 31)),       # 1984: whole chunks, ragged ranges
    (25, 8, np.array([30.0, -30.0, 0.0])),   # 75: 11
])
def test_last_tilt_at_zero_matches_exact_transform(nx, th, tilts, S):
    from feilab_b200.icon import IconPlan
    from oracle.oracle import OraclePlan
    tilts = np.asarray(tilts, np.float32)
    assert tilts[-1] == 0.0
    o = OraclePlan(nx, th, tilts, "f64")
    w = o.geometry()[1].astype(np.float64)
    m0, Ahwb = _inputs(S, nx, th)
    p = IconPlan(nx, th, tilts, capacity=S)
    m, al, rt = _iteration(p, "toeplitz", Ahwb, m0)
    for s in {0, S - 1}:
        rh = o.ndft_adjoint(w * o.ndft_forward(m0[s].astype(np.float64))) - Ahwb[s].astype(np.complex128)
        rtr = float((np.abs(rh) ** 2).sum())
        ale = rtr / float((w * np.abs(o.ndft_forward(rh)) ** 2).sum())
        assert rel_l2(m[s], m0[s] - ale * rh.real) < TOL, s
        assert abs(al[0, s] - ale) <= TOL * ale
        assert abs(rt[0, s] - rtr) <= TOL * rtr
    p.close()


def test_last_tilt_at_zero_in_one_range_matches_nufft_iteration():
    from feilab_b200.icon import IconPlan
    nx, th = 4095, 500                       # 512 tiles of K; 45045 nodes: 5 in the last chunk
    p = IconPlan(nx, th, np.linspace(-60, 0, 11).astype(np.float32), capacity=1)
    m0, Ahwb = _inputs(1, nx, th)
    mn, aln, rtn = _iteration(p, "nufft", Ahwb, m0)
    mt, alt, rtt = _iteration(p, "toeplitz", Ahwb, m0)
    assert rel_l2(mt, mn) < TOL
    assert abs(alt[0, 0] - aln[0, 0]) <= TOL * abs(aln[0, 0])
    assert abs(rtt[0, 0] - rtn[0, 0]) <= TOL * abs(rtn[0, 0])
    p.close()
