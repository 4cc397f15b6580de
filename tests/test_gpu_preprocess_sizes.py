"""Stack pre-processing at the edges of its kernel against the oracle's
restatement of the reference tool: fewer rows than the CTAs of a cluster, odd
widths (scalar loads) and multiples of four (float4), rows longer than the
shared-memory cache holds, an unaligned stack, a constant projection.

Mode subtraction bit for bit; the normalisation within 2e-6 of the largest
value (float results of double sums taken in another order).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,ny,nx,shift", [(1, 1, 1, 0), (3, 5, 7, 0), (2, 9, 64, 0), (5, 33, 130, 0), (2, 40, 1028, 0),
                                            (1, 17, 50001, 0), (1, 16, 47108, 0), (3, 64, 96, 1)])
def test_preprocess_matches_oracle(nz, ny, nx, shift):
    from feilab_b200 import tools
    from oracle.preprocess import preprocess
    rng = np.random.default_rng(3)
    st = (1000 + 40 * rng.standard_normal((nz, ny, nx))).astype(np.float32)
    if nz > 2:
        st[1] = 7.25          # no spread
    tilts = np.linspace(-50, 50, nz).astype(np.float32)
    buf = torch.empty(st.size + 8, dtype=torch.float32, device="cuda")
    d = buf[shift:shift + st.size].view(st.shape)
    d.copy_(torch.from_numpy(st))
    np.testing.assert_array_equal(tools.preprocess(d).cpu().numpy(), preprocess(st))
    got, ref = tools.preprocess(d, tilts, 120).cpu().numpy(), preprocess(st, tilts, 120)
    fine = np.isfinite(ref)
    assert np.array_equal(fine, np.isfinite(got))
    if fine.any():
        assert np.max(np.abs(got[fine] - ref[fine])) <= 2e-6 * np.max(np.abs(ref[fine]))
