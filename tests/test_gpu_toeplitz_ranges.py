"""The Toeplitz kernel's order of summation: its node ranges go by the grid and the
width alone, so equal solves give equal bits whatever the plan's capacity (of one
group size) and number of weight sets, and a tilt at weight 0 gives the kernel of
the series without it.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(64, 40, 31), (8, 8, 3), (512, 256, 61), (1024, 300, 61)]


def _rows(S, nt, nx):
    return np.random.default_rng(nx).standard_normal((S, nt, nx)).astype(np.float32)


def _solve(p, rows):
    p.set_operator("toeplitz")
    return p.solve(p.prepare_rhs(torch.from_numpy(rows).cuda()), (2, 16, 2), 2, 0.0).cpu().numpy()


@pytest.mark.parametrize("nx,th,nt", SHAPES)
def test_same_bits_at_every_capacity(nx, th, nt):
    from feilab_b200.icon import IconPlan
    tilts = np.linspace(-60, 55, nt).astype(np.float32)
    rows = _rows(8, nt, nx)
    out = []
    for capacity in (8, 24, 64):
        p = IconPlan(nx, th, tilts, capacity=capacity)
        out.append((p.B, _solve(p, rows)))
        p.close()
    assert {b for b, _ in out} == {8} and np.all(np.isfinite(out[0][1]))
    for _, m in out[1:]:
        assert np.array_equal(m, out[0][1])


@pytest.mark.parametrize("nx,th,nt", SHAPES)
def test_same_bits_with_other_weight_sets_and_without_the_tilt(nx, th, nt):
    from feilab_b200.icon import IconPlan
    tilts = np.linspace(-60, 55, nt).astype(np.float32)
    omit = nt // 2
    keep = [k for k in range(nt) if k != omit]
    red = IconPlan(nx, th, tilts[keep], capacity=8)
    rows = _rows(8, nt, nx)
    want = _solve(red, np.ascontiguousarray(rows[:, keep]))
    wr = red.geometry()[1].reshape(nt - 1, nx)
    p = IconPlan(nx, th, tilts, capacity=24)
    plain = _solve(p, rows)
    w = np.zeros((nt, nx), np.float32)
    w[keep] = wr
    p.set_group_weights(np.stack([p.geometry()[1].ravel(), w.ravel(), 0.5 * w.ravel()]))   # three sets
    m = _solve(p, np.concatenate([rows] * 3))
    assert np.array_equal(m[:8], plain)
    assert np.array_equal(m[8:16], want)
    red.close()
    p.close()
