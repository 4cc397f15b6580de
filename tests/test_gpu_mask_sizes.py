"""The mask's 2-D filtering at the sizes where its kernels change (rows and
columns per CTA, FFT radix), crops of odd height at both ends, against the
FP64 restatement.  Bound 2e-6 relative L2: two FP32 FFTs of at most 2 x 13
radix-2 levels, each level rounding to 2^-24 with random signs
(sqrt(52) 2^-24 = 4e-7), doubled for the filter's and pairing's products and
with a factor 2 for the crop's share of the energy.
"""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S,ystart,thickness", [(16, 3, 0, 16), (16, 1, 15, 1), (64, 5, 7, 33), (512, 2, 300, 212),
                                                  (1024, 2, 0, 5), (2048, 1, 900, 301), (4096, 1, 3, 1001),
                                                  (8192, 1, 4000, 257)])
def test_mask_apply_matches_fp64(n, S, ystart, thickness):
    from feilab_b200 import tools
    from oracle import mask as om
    tilts = np.linspace(-50, 60, 23).astype(np.float32)
    m = tools.Mask(n, tilts, 0.25, 0.0, True, capacity=S)
    sl = np.random.default_rng(n).standard_normal((S, n, n)).astype(np.float32)
    got = m.apply(torch.from_numpy(sl).cuda(), ystart, thickness).cpu().numpy()
    ref = om.apply(sl, m.filter(), ystart, thickness)
    for s in range(S):
        assert rel_l2(got[s], ref[s]) < 2e-6, s
