// dg_conv_index.h -- index arithmetic of the convolution kernels that the
// host can check too (no CUDA needed to compile it).
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

}  // namespace net
}  // namespace dg
