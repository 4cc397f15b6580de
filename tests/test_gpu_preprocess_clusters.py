"""Stack pre-processing at every cluster size that the number and size of the
projections choose (1, 2, 4 and 8 CTAs a projection), out of place and in place,
against the restatement: the mode subtraction bit for bit, the normalised stack to
2e-6 of its largest value (two roundings of 2^-24 to float behind a variance in
double, and the reference's float mean).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,ny,nx", [
    (140, 12, 100),     # 1, in one round
    (149, 20, 60),      # 1, in two rounds
    (41, 64, 130),      # 2
    (70, 33, 200),      # 2
    (21, 50, 64),       # 4
    (37, 31, 77),       # 4
    (3, 96, 128),       # 8
    (18, 90, 101),      # 8: every place of a cluster taken
])
def test_every_cluster_size_matches_oracle(nz, ny, nx):
    from feilab_b200 import tools
    from oracle.preprocess import preprocess
    rng = np.random.default_rng(nz)
    st = (1000 + 40 * rng.standard_normal((nz, ny, nx))).astype(np.float32)
    tilts = np.linspace(-50, 50, nz).astype(np.float32)
    d = torch.from_numpy(st).cuda()
    np.testing.assert_array_equal(tools.preprocess(d).cpu().numpy(), preprocess(st))
    ref = preprocess(st, tilts, 120)
    got = tools.preprocess(d, tilts, 120)
    assert np.max(np.abs(got.cpu().numpy() - ref)) <= 2e-6 * np.max(np.abs(ref))
    assert torch.equal(tools.preprocess(d, tilts, 120, out=d), got)
