// dg_noalloc_limit.h -- which grids dg_compute_step_noalloc takes (no CUDA
// needed to compile it; the host checks the rule).
//
// The step's scratch once held 56 bytes of partial results per block, beside
// the control block in 1 MiB, and that bounded a grid's size.  A step needs no
// memory per block any more.  The bound stays, as an interface: a caller that
// sizes its grids by it keeps every answer.  So this is the block count of the
// kernels and splits the bound came from, on its own here: it does not follow
// the present kernels' tiles or chunks.
#pragma once

namespace dg {
namespace noalloc {

constexpr int kMostBlocks = 18134;
constexpr int kSmsThen = 148;

inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// Blocks of an nx x ny x nz grid (interior cells).  fused: the arithmetic of
// DG_ROUNDING_FAST, in 64-column tiles; else 32-column ones.
inline long long limit_blocks(int nx, int ny, int nz, bool f64, bool fused) {
    if (!fused) {
        // enough blocks for 14 waves of two per SM, at least 20 planes each
        const long long tiles = ceil_div(ny, f64 ? 4 : 8) * ceil_div(nz, 32);
        const long long want = ceil_div(2LL * kSmsThen * 14, tiles), most = nx / 20 > 0 ? nx / 20 : 1;
        const long long planes = ceil_div(nx, want < most ? want : most);
        return tiles * ceil_div(nx, planes);
    }
    const int rows = f64 ? 4 : 14;
    const long long tiles = ceil_div(ny, rows) * ceil_div(nz, 64);
    // tiles two cells clear of every y and z face
    const int iy = (ny - 2) / rows - 1, iz = (nz - 2) / 64 - 1;
    const long long interior = iy > 0 && iz > 0 ? (long long)iy * iz : 0;
    if (interior >= kSmsThen) return interior + (tiles - interior) * ceil_div(nx, nx < 64 ? nx : 64);
    // the split of at least 24 planes with the fewest waves x (planes + 3)
    long long best = -1, split = 1;
    for (int c = 1; c == 1 || (c <= nx / 24 && c <= 64); ++c) {
        const long long cost = ceil_div(tiles * c, kSmsThen) * (ceil_div(nx, c) + 3);
        if (best < 0 || cost < best) {
            best = cost;
            split = c;
        }
    }
    return tiles * ceil_div(nx, ceil_div(nx, split));
}

inline bool accepted(int nx, int ny, int nz, bool f64, bool fused) {
    return limit_blocks(nx, ny, nz, f64, fused) <= kMostBlocks;
}

}  // namespace noalloc
}  // namespace dg
