// dg_kernels.cuh -- device-side data structures shared by the kernels and
// the C-ABI layer.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "dg_physics.cuh"

namespace dg {

constexpr int kHist = 4096;      // dt history ring on the device
constexpr unsigned kStatusNonFinite = 0x1u;
constexpr unsigned kStatusTimeout = 0x2u;

// Step control block, one per grid, in device memory.  The step kernel of
// step s reads dt[s & 1] (computed from the state at the start of step s)
// and its last block writes dt[(s + 1) & 1] from the updated state, so dt
// never travels through the host.
struct DevCtl {
    unsigned long long step;   // steps completed since the state was set
    unsigned int counter;      // blocks of the running launch that finished
    unsigned int flags;        // sticky status bits (kStatus*)
    unsigned long long wmax;   // largest wave speed of the running launch so far (bits; 0 between launches)
    double dt[2];
    double sums[5];            // FP64 interior sums of the current state
    double hist[kHist];        // dt used by step s at hist[s % kHist]
};

// Per-block partial sums, added in a fixed order by the launch's last block.
struct Partial {
    double sums[5];
};

// Where the five fields of a state live outside the pitched buffers: base
// pointers in the grid's field order and element strides along the grid's
// axes.
template <class T> struct FieldView {
    T *f[5];
    long long sx, sy, sz;
};

// Geometry and physics of one grid as the kernels see it.
template <class T> struct GridArgs {
    const T *src;              // state read by the step (5 fields)
    T *dst;                    // state written by the step
    int nx, ny, nz;            // ghosted extents (interior + 4)
    int pitch;                 // elements between consecutive z-rows
    long long fstride;         // elements between fields
    int bc[6];                 // Bc per face (x-, x+, y-, y+, z-, z+)
    int heat;                  // bit a: the lower face of axis a is a conducting wall
    int gravity;
    int limiter;               // 0 central slopes, 1 minmod
    int nparts;                // work items of this grid in a batched launch
    long long wait_budget;     // SM clocks a wait for a staged plane may take (kWaitBudget)
    Consts<T> k;
    DevCtl *ctl;
    Partial *part;             // conservation sums only (kReduceBlocks entries)
    int chain;                 // kChain*: this step among the steps of one call (here, not ahead of k: the
                               // constants keep their alignment, 3.09 instead of 3.18 ms per 512^3 step)
};

// GridArgs::chain.  Wait: the launch before is the step before, which lets this
// one start early; Let: the launch after is a step that waits.
enum : int { kChainWait = 1, kChainLet = 2 };

// Boundary types of dg_sim_info (DG_BC_*) into the kernels' form.  A
// conducting wall (DG_BC_CONDUCTING_WALL = 3, the reference CUDA variant's
// BC::CONDUCTING_WALL) follows the wall rule for every ghost (kernels.h:327)
// and adds a heat source to the energy flux of its face.  The reference adds
// it at the flux of lower-cell index 1 for a lower face and n - 2 for an
// upper face (kernels.h:561-661): only the lower face's reaches an interior
// cell, so only lower faces set a heat bit.
constexpr int kBcConductingWall = 3;
inline bool valid_bc_pair(int lo, int hi) {
    return lo >= 0 && lo <= kBcConductingWall && hi >= 0 && hi <= kBcConductingWall &&
           (lo == kPeriodic) == (hi == kPeriodic);
}
template <class T> inline void set_boundaries(GridArgs<T> &a, const int32_t bcs[6]) {
    a.heat = 0;
    for (int f = 0; f < 6; ++f) {
        const bool cond = bcs[f] == kBcConductingWall;
        a.bc[f] = cond ? (int)kWall : (int)bcs[f];
        if (cond && (f & 1) == 0) a.heat |= 1 << (f / 2);
    }
}

// SMs of a B200 (2 dies x 74); grid sizes below are multiples of it
constexpr int kSms = 148;
constexpr int kReduceBlocks = kSms * 8;   // grid of the state-reduction kernel

// The step kernels: one cell per lane (dg_march_impl.cuh) with the
// reference's rounding in double and in float and with fused arithmetic in
// double, and the packed fused-arithmetic sweep in float (dg_sweep_impl.cuh).
enum KernelKind : int { kRefF64 = 0, kRefF32 = 1, kFastF32 = 2, kFastF64 = 3 };

inline bool is_sweep(int kind) { return kind == kFastF32; }

// Owned tile rows (y) of each kernel; a block also runs two halo warps.
#ifndef DG_SWEEP_ROWS_F32
#define DG_SWEEP_ROWS_F32 14
#endif
constexpr int kSweepRowsF32 = DG_SWEEP_ROWS_F32;
constexpr int kMarchRows = 14;   // 16 warps of 128 registers
constexpr int kMarchRing = 2;    // staged planes
inline int step_tile_rows(int kind) { return is_sweep(kind) ? kSweepRowsF32 : kMarchRows; }
// Tile columns (z) and the staged box width (2-cell halo each side).
inline int step_tile_cols(int kind) { return is_sweep(kind) ? 64 : 32; }
inline int step_box_cols(int kind) { return step_tile_cols(kind) + 4; }
inline int step_threads(int kind) { return 32 * (step_tile_rows(kind) + 2); }

// Tiles of a sweep step.  Interior tiles are full tiles (rows x cols) at
// least two cells clear of every y and z face, so that no row or column of
// them is on a face or writes a ghost image: they form the rectangle of tile
// rows [1, 1 + ny) x tile columns [1, 1 + nz) (tile row t starts at cell
// 2 + t * rows and needs 2 + (t + 1) * rows <= interior cells); ny = nz = 0
// when either side has none.  The other tiles are the frame.  A step with
// interior tiles is two launches: the interior tiles, one block per tile
// marching all of x, built without the owned warps' boundary switches, and
// the frame in x-chunks (launch_sweep).
struct InteriorTiles {
    int tiles_y, tiles_z, ny, nz;
    __host__ __device__ InteriorTiles(int ghosted_ny, int ghosted_nz, int rows, int cols) {
        const int iy = ghosted_ny - 4, iz = ghosted_nz - 4;
        tiles_y = (iy + rows - 1) / rows;
        tiles_z = (iz + cols - 1) / cols;
        ny = iy >= 2 ? (iy - 2) / rows - 1 : 0;
        nz = iz >= 2 ? (iz - 2) / cols - 1 : 0;
        if (ny <= 0 || nz <= 0) ny = nz = 0;
    }
    __host__ __device__ int interior() const { return ny * nz; }
    __host__ __device__ int frame() const { return tiles_y * tiles_z - ny * nz; }
    // tile of frame index f: the rows outside the rectangle whole, then the
    // rectangle's rows left and right of it
    __host__ __device__ void frame_tile(int f, int &ty, int &tz) const {
        const int full = (tiles_y - ny) * tiles_z;
        if (f < full) {
            const int r = f / tiles_z;
            tz = f % tiles_z;
            ty = r < 1 ? r : r + ny;
        } else {
            const int g = f - full, w = tiles_z - nz;
            ty = 1 + g / w;
            const int c = g % w;
            tz = c < 1 ? c : c + nz;
        }
    }
};

// x-planes per block of a sweep step's interior launch: whole columns when
// the interior tiles alone fill the SMs at least once (the frame's shorter
// blocks then fill the interior launch's last wave), else the frame's chunk
// (a few long blocks would leave most SMs idle).
inline int interior_chunk(int nx, const InteriorTiles &it, int chunk) {
    return it.interior() >= kSms ? nx - 4 : chunk;
}

// Blocks of one step: (y tiles) x (z tiles) x (x chunks of `chunk` planes);
// for a sweep step with interior tiles, the interior tiles x their chunks
// (interior_chunk) plus the frame tiles x chunks (both launches together).
inline int step_grid_blocks(int nx, int ny, int nz, int kind, int chunk) {
    const int ty = step_tile_rows(kind), tzc = step_tile_cols(kind);
    const int chunks = (nx - 4 + chunk - 1) / chunk;
    if (is_sweep(kind)) {
        const InteriorTiles it(ny, nz, ty, tzc);
        const int ci = interior_chunk(nx, it, chunk);
        return it.interior() * ((nx - 4 + ci - 1) / ci) + it.frame() * chunks;
    }
    const int tiles_z = (nz - 4 + tzc - 1) / tzc;
    const int tiles_y = (ny - 4 + ty - 1) / ty;
    return tiles_z * tiles_y * chunks;
}
// Blocks' finishing time on the SMs, in planes, of a sweep launch over
// `tiles` tiles and nxi planes in `chunk`-plane blocks, one block per SM, the
// shorter last chunk's blocks dispatched last: every SM takes full chunks in
// turn, then the remainders go to whichever SMs are free first.  A block
// costs its planes plus kBlockPlanes: the two planes it computes beyond its
// chunk and about two planes' time of launch, first copies and reduction
// (measured on the FP32 kernel: 8 us + 4.1 us per plane marched; the split it
// chooses is within 5 % of the best one for all four kernels on seven grids of
// 24^3 to 190x170x180).
constexpr int kBlockPlanes = 4;
inline long long sweep_makespan(long long tiles, int nxi, int chunk) {
    const long long full = tiles * (nxi / chunk), rest = nxi % chunk ? tiles : 0;
    const long long cf = chunk + kBlockPlanes, cr = nxi % chunk + kBlockPlanes;
    // SMs that got one full block more than the others
    long long n_late = full % kSms, t_late = (full / kSms + (n_late ? 1 : 0)) * cf;
    long long n_free = kSms - n_late, t_free = full / kSms * cf, left = rest, end = n_late ? t_late : t_free;
    while (left > 0) {
        long long &t = (n_late == 0 || t_free <= t_late) ? t_free : t_late;
        left -= &t == &t_free ? n_free : n_late;
        t += cr;
        if (t > end) end = t;
    }
    return end;
}

// The split of x into chunks that minimises waves x (planes per block + 3
// re-staged), at least 24 planes per block unless no more than `small` blocks
// come of it.
inline int waves_chunk(long long tiles, int nxi, long long small) {
    const int maxc = nxi / 24 > 0 ? nxi / 24 : 1;
    long long best = -1;
    int bestc = 1;
    for (int c = 1; c <= nxi && c <= 64; ++c) {
        if (c > maxc && tiles * c > small) break;
        const long long per = (nxi + c - 1) / c;
        const long long waves = (tiles * c + kSms - 1) / kSms;
        const long long cost = waves * (per + 3);
        if (best < 0 || cost < best) { best = cost; bestc = c; }
    }
    return (nxi + bestc - 1) / bestc;
}

// Default x-planes per block (one block per SM).  The packed sweep with
// interior tiles that fill the SMs: the frame launch's chunk (the interior
// launch marches whole columns); with fewer interior tiles: the split of x that
// minimises waves x (planes + 3 re-staged), at least 24 planes per block
// unless that leaves SMs idle (40x300x130: 181 -> 102 us); with none, the
// split that ends first (sweep_makespan), down to single planes: a small grid
// is latency-bound, a block's time being its planes one after another, so
// short chunks on all SMs win although each block recomputes two planes (FP32,
// periodic, us per step when the rule was chosen, at least 24 planes per block
// -> this rule: 48^3 116 -> 25, 64^3 146 -> 29, 128^3 124 -> 93, 300x40x70 116
// -> 75).
inline int choose_chunk(int nx, int ny, int nz, int kind) {
    const int ty = step_tile_rows(kind), tzc = step_tile_cols(kind);
    // sweep steps whose interior tiles fill the SMs (interior_chunk): the
    // frame's blocks fill the interior launch's last wave, in short chunks
    // (32-64 planes measured 38.2-38.6 GCUPS on 512^3 Sod, whole columns
    // 34.1-34.4)
    if (is_sweep(kind) && InteriorTiles(ny, nz, ty, tzc).interior() >= kSms) return nx - 4 < 64 ? nx - 4 : 64;
    const long long tiles = (long long)((ny - 4 + ty - 1) / ty) * ((nz - 4 + tzc - 1) / tzc);
    const int nxi = nx - 4;
    if (is_sweep(kind) && InteriorTiles(ny, nz, ty, tzc).interior() > 0) {
        return waves_chunk(tiles, nxi, 4 * kSms);
    }
    int bestp = nxi;
    long long best = sweep_makespan(tiles, nxi, nxi);
    for (int p = nxi - 1; p >= 1; --p) {
        // short chunks only where they fill idle SMs: a large grid's count
        // of blocks stays that of 24 planes or more
        const long long c = (nxi + p - 1) / p;
        if ((p < 24 || c > 64) && tiles * c > 4 * kSms) continue;
        const long long t = sweep_makespan(tiles, nxi, p);
        if (t < best) { best = t; bestp = p; }
    }
    return bestp;
}

// Launch helpers.  EXACT selects the reference-rounding policy
// (dg_step_ref.cu, built with --fmad=false) or the fast one
// (dg_step_fast.cu); float/fast, float/exact and double/exact exist.
template <class T> cudaError_t launch_sums(const GridArgs<T> &a, cudaStream_t st);
template <class T, bool EXACT>
cudaError_t launch_cons_to_prim_policy(const GridArgs<T> &a, const T *cons, T *prim, long long prim_fstride,
                                       int prim_pitch, cudaStream_t st);
// Message returned by dg_last_error(NULL) (errors not tied to a context).
void set_global_error(const std::string &msg);

// The step; the tensor map's box is step_box_cols x (step_tile_rows + 4) x 1
// x 5.  launch_sweep: kFastF32; launch_march: the other kinds.
cudaError_t launch_sweep(const GridArgs<float> &a, const CUtensorMap *tmap_src, int chunk, cudaStream_t st);
cudaError_t launch_march(const GridArgs<float> &a, const CUtensorMap *tmap_src, int kind, int chunk, cudaStream_t st);
cudaError_t launch_march(const GridArgs<double> &a, const CUtensorMap *tmap_src, int kind, int chunk, cudaStream_t st);
// A state from src into a.dst with its ghosts, the dt of the coming step
// (number `step`) and a fresh control block.  prims: src holds primitives;
// exact: the wave speeds round like the reference (FP64 always does).  src
// may be a.dst itself: then the ghosts are written, and interior cells that
// share a 16-byte access with one, with their own values.
template <class T>
cudaError_t launch_set_state(const GridArgs<T> &a, const FieldView<const T> &src, bool prims, bool exact,
                             unsigned long long step, cudaStream_t st);
// The state at src (a's fields through the view's strides) as five dense
// arrays of n0 x n1 x n2 cells.
template <class T>
cudaError_t launch_get_state(const FieldView<const T> &src, T *const dst[5], int n0, int n1, int n2, cudaStream_t st);

}  // namespace dg
