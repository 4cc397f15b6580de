"""The table reads of the adjoint gather (CPU): every index that a warp of
yadj_gather forms with the rules of csrc/adj_gather.h stays within its grid row's
entries, for the series that leave the fewest of them in a row (2 to 9 tilts, widths
around powers of two, both windows), every slice-group size and FFT length.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle.oracle import OraclePlan

# Walks the chunks of every row and warp as the kernel does: chunks from the
# warp's first entry on, `stages` in flight and one more node load ahead.
# Returns the reads outside the row, or of another entry than the one staged.
DRIVER = r"""
#include <algorithm>
#include <vector>
#include "adj_gather.h"
using namespace icon;
extern "C" long check(const int *ix0, const int *iy0, int M, int tlo, int thi, int n0, int n1, int B, int warps,
                      int stages, long *reads)
{
    std::vector<std::vector<int>> rows(n0);
    for (int j = 0; j < M; ++j)
        for (int t = tlo; t <= thi; ++t) rows[((ix0[j] + t) % n0 + n0) % n0].push_back(iy0[j]);
    const int ph = ywin_ph(B), nr = ywin_nr(B), nblk = ywin_blocks(n1, B), C = B >= 2 ? B / 2 : 1, CH = kAdjChunk;
    std::vector<unsigned short> off(nblk + 1), cut(warps + 1);
    long bad = 0;
    *reads = 0;
    for (auto &r : rows) {
        std::sort(r.begin(), r.end());
        const int cnt = (int)r.size();
        adj_row_tables(r.data(), cnt, n1 / 2 + kHalo + tlo, ph, nblk, warps, off.data(), cut.data());
        if (off[nblk] != cnt || cut[0] != 0 || cut[warps] != nblk) ++bad;
        for (int w = 0; w < warps; ++w) {
            const int b0 = cut[w], b1 = cut[w + 1];
            if (b1 < b0) ++bad;
            const int bs = adj_first_block(b0, b1, nr), es = off[bs], ee = off[b1];
            if (bs > b1 || (b0 == b1 && bs != b1)) ++bad;    // a warp without blocks walks none
            if (b0 < b1 && bs != std::max(b0 - (nr - 1), 0)) ++bad;
            if (ee <= es) continue;               // a warp without entries reads no nodes
            for (int c0 = es; c0 < ee + (stages + 1) * CH; c0 += CH)
                for (int lane = 0; lane < 32; ++lane) {
                    const int at = lane / C, e = adj_entry(c0, at, ee);
                    ++*reads;
                    if (e < es || e >= ee || e >= cnt) ++bad;
                    if (at < CH && c0 + at < ee && e != c0 + at) ++bad;
                }
        }
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("gather")
    (d / "d.cpp").write_text(DRIVER)
    so = str(d / "d.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "feilab_b200", "csrc"),
                    "-o", so, str(d / "d.cpp")], check=True)
    f = ctypes.CDLL(so).check
    f.restype = ctypes.c_long
    return f


@pytest.mark.parametrize("window", ["gauss6", "kb4"])
@pytest.mark.parametrize("nx,th", [(33, 8), (40, 20), (31, 64), (65, 100), (130, 200), (127, 400), (257, 513)])
def test_gather_reads_stay_in_the_row(driver, nx, th, window):
    tlo, thi = (0, 13) if window == "gauss6" else (3, 10)
    for nt in range(2, 10):
        for tilts in (np.linspace(-1.0, 1.5, nt), np.linspace(-60, 60, nt), np.linspace(0, 90, nt)):
            o = OraclePlan(nx, th, tilts.astype(np.float32), "f64", window=window)
            xy = o.geometry()[0]                  # first taps floor(n x) - 6, in float
            ix0, iy0 = (np.ascontiguousarray(np.floor(np.float32(n) * xy[:, k]), np.int32) - 6
                        for k, n in enumerate((o.n0, o.n1)))
            for B in (1, 2, 4, 8):
                # threads of the y-pass: the register FFT's, or n1 B values by 16 or 32
                fft = {o.n1 // 32 * B} if o.n1 in (128, 256, 512, 1024) else {o.n1 * B // 16, o.n1 * B // 32}
                for warps in {max(t, 64) // 32 for t in fft}:
                    reads = ctypes.c_long()
                    bad = driver(ix0.ctypes.data_as(ctypes.c_void_p), iy0.ctypes.data_as(ctypes.c_void_p), o.M, tlo, thi,
                                 o.n0, o.n1, B, warps, 3 if warps <= 8 else 2, ctypes.byref(reads))
                    assert reads.value > 0 and bad == 0, (nt, B, warps, bad)
