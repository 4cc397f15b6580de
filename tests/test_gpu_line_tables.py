"""Reprojection lines keep no tables of the adjoint gather: what a new angle adds to
the plan's device memory (icon_plan_query) stays within its windows and entries.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _mib(p):
    from feilab_b200 import icon
    d = (ctypes.c_int * 10)()
    assert icon.lib().icon_plan_query(p._h, d) == 0
    return d[8]


@pytest.mark.parametrize("capacity", [1, 2, 8])
def test_line_memory(capacity):
    from feilab_b200.icon import IconPlan
    nx, th, lines = 1024, 64, 12
    p = IconPlan(nx, th, np.linspace(-60, 60, 5).astype(np.float32), capacity=capacity)
    m = torch.randn(capacity, nx, th, device="cuda")
    p.reproject(m, 0.25)
    mib = _mib(p)
    for k in range(lines):
        p.reproject(m, 1.0 + k)
    # per node: position, two windows (14 and 16 values), taps, weight; per entry
    # (14 a node): tap, first row, 16 window values; one offset per grid row
    line = nx * (8 + 4 * (14 + 16 + 2 + 1) + 14 * (4 + 4 + 64)) + 4 * (2 * nx + 1)
    assert _mib(p) - mib <= lines * line / 2**20 + 1
    p.close()
