// adj_gather.h -- layout and index rules of the adjoint gather (yadj_gather in
// icon_kernels.cuh) that its tables are built by: plain C++, so that they can be
// checked without a device.
#pragma once

#ifdef __CUDACC__
#define ICON_HD __host__ __device__
#else
#define ICON_HD
#endif

namespace icon {

constexpr int kHalo = 8;      // halo rows on each side of a rotated row buffer

// Layout of the gather for groups of B slices: a warp's lanes are ywin_ph(B)
// neighbouring buffer rows times B slices (two slices a lane for B = 8), and an
// entry's window, starting anywhere within a block of ph rows, covers at most nr
// blocks.
ICON_HD constexpr int ywin_ph(int B) { return B >= 4 ? 8 : B == 2 ? 16 : 32; }
ICON_HD constexpr int ywin_nr(int B) { return B >= 4 ? 3 : 2; }
ICON_HD constexpr int ywin_lp(int B) { return ywin_ph(B) * ywin_nr(B); }
ICON_HD constexpr int ywin_pos(int ph, int p, int k) { return k < 2 ? 2 * p + k : 2 * ph + p; }
ICON_HD constexpr int ywin_blocks(int n1, int B) { return (n1 + 2 * kHalo + ywin_ph(B) - 1) / ywin_ph(B); }

// Entries per staged chunk.
constexpr int kAdjChunk = 8;

// Tables of one grid row whose cnt entries have the first non-zero taps at buffer
// rows iy[e] + ofs, sorted: off[v], v = 0..nblk, the entries that start below
// block v (ph rows each), and cut[w], w = 0..warps, the block ranges of the warps,
// cut at equal shares of entries + blocks (a block's store and bounds cost about
// as much as an entry).
inline void adj_row_tables(const int *iy, int cnt, int ofs, int ph, int nblk, int warps, unsigned short *off,
                           unsigned short *cut)
{
    int e = 0;
    for (int v = 0; v <= nblk; ++v) {
        while (e < cnt && iy[e] + ofs < v * ph) ++e;
        off[v] = (unsigned short)e;
    }
    const long long total = (long long)cnt + nblk;
    for (int w = 0, v = 0; w <= warps; ++w) {
        while (v < nblk && (long long)(off[v] + v) * warps < total * w) ++v;
        cut[w] = (unsigned short)(w == warps ? nblk : v);
    }
}

// First block that a warp with blocks b0..b1-1 walks: windows of the nr - 1 blocks
// before reach into its own.  A warp without blocks walks none.
ICON_HD inline int adj_first_block(int b0, int b1, int nr)
{
    return b0 == b1 ? b1 : b0 < nr - 1 ? 0 : b0 - (nr - 1);
}

// Entry of the row whose node the lane of place `at` copies for the chunk from
// entry c0 on, in a warp whose entries end before ee: past the end the last one
// again.  Only for warps that have entries; c0 and at are not negative.
ICON_HD inline int adj_entry(int c0, int at, int ee) { return c0 + at < ee ? c0 + at : ee - 1; }

}  // namespace icon
