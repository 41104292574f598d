// dg_conv_index.h -- index arithmetic and division of work of the convolution
// kernels that the host can check too (no CUDA needed to compile it).
#pragma once

#ifdef __CUDACC__
#define DG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define DG_HOST_DEVICE inline
#endif

namespace dg {
namespace net {

// A position (y, z) along x in a tensor [b][x][y][z][channels]: the element of
// channel c0 in plane x is at + (x - x0) * step.  All of it in 64 bits: one
// plane may hold 2^30 positions of 32 channels.
struct PlaneIndex {
    long long at, step;
    DG_HOST_DEVICE PlaneIndex(int b, int x0, int y, int z, int nx, int ny, int nz, int channels, int c0)
        : at(((((long long)b * nx + x0) * ny + y) * nz + z) * channels + c0),
          step((long long)ny * nz * channels) {}
    DG_HOST_DEVICE long long plane(int k) const { return at + k * step; }
};

// A block's share of the work: columns of `len` steps, `work` steps in all.  A
// piece of a column takes kStartSteps beside its own.  As many rounds of whole
// columns as every block gets one of, neighbouring columns in step with each
// other, so that the rows they share come from L2; then an equal range of the
// remaining columns' steps, or, on columns so short that a range costs no less
// than a column (it may reach into a second one), those columns whole.  next()
// gives a column, its first step and the count of steps in it.  A column's
// outputs do not depend on the split.
//
// Measured on whole forward passes, us: fixed chunks of 8-64 planes, as many as
// gave each block four | whole columns, each block starting a column a little
// further in and wrapping around, then ranges | this rule.  (1, 9, 400, 400)
// 180 | 201 | 167, (1, 20, 400, 400) 466 | 452 | 410, (4, 12, 300, 300) 518 |
// 572 | 473, (8, 73, 73, 73) 789 | 432 | 418, (1, 100, 200, 200) 866 | 582 |
// 566, (1, 264, 264, 264) 2995 | 2681 | 2628: the wrap costs a piece per
// column, and blocks in step ask no slower than blocks spread out.
constexpr int kStartSteps = 2;

struct Share {
    long long column, pos = 0, end = 0;
    int len, blocks, rounds;
    DG_HOST_DEVICE Share(long long work, int len_, int block, int blocks_)
        : column(block), len(len_), blocks(blocks_) {
        const long long columns = work / len, rest = columns % blocks;
        rounds = (int)(columns / blocks);
        if (rest * len / blocks + 1 + 2 * kStartSteps <= len + kStartSteps) {
            pos = (columns - rest) * len + rest * len * block / blocks;
            end = (columns - rest) * len + rest * len * (block + 1) / blocks;
        } else if (block < rest) {
            ++rounds;
        }
    }
    DG_HOST_DEVICE bool next(long long &col, int &first, int &count) {
        if (rounds > 0) {
            col = column;
            first = 0;
            count = len;
            --rounds;
            column += blocks;
            return true;
        }
        if (pos >= end) return false;
        col = pos / len;
        first = (int)(pos - col * len);
        count = (int)(len - first < end - pos ? len - first : end - pos);
        pos += count;
        return true;
    }
};

}  // namespace net
}  // namespace dg
