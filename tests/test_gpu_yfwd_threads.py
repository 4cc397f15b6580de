"""The forward y-pass's threads go by the number of CTAs, the entries and real or
complex input; a slice's values do not depend on them: slices transformed in calls
of one group and of several (other thread counts), equal bit for bit, and equal the
FP64 oracle to the window's float rounding (1e-5, as the other transform tests).
"""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity,group", [(24, 8), (12, 4), (4, 2), (2, 1)])
@pytest.mark.parametrize("nx,th", [(256, 40), (300, 100), (40, 300)])
def test_same_bits_at_every_thread_count(nx, th, capacity, group, monkeypatch):
    from feilab_b200.icon import IconPlan
    from oracle.oracle import OraclePlan
    monkeypatch.setenv("ICON_BATCH", str(group))
    tilts = np.linspace(-60, 57, 41).astype(np.float32)
    p = IconPlan(nx, th, tilts, capacity=capacity)
    assert p.B == group
    o = OraclePlan(nx, th, tilts, "f64")
    rng = np.random.default_rng(nx)
    x = rng.standard_normal((capacity, nx, th)).astype(np.float32)
    z = (x + 1j * rng.standard_normal(x.shape)).astype(np.complex64)
    for img in (x, z):
        d = torch.from_numpy(img).cuda()
        many = p.nufft_forward(d)
        one = torch.cat([p.nufft_forward(d[s:s + group].contiguous()) for s in range(0, capacity, group)])
        assert torch.equal(many, one)
        assert rel_l2(many[0].cpu().numpy(), o.forward(img[0])) < 1e-5
    d = torch.from_numpy(x).cuda()
    many = p.reproject(d, 3.0)
    one = torch.cat([p.reproject(d[s:s + group].contiguous(), 3.0) for s in range(0, capacity, group)])
    assert torch.equal(many, one)
    p.close()
