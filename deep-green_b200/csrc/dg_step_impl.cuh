// dg_step_impl.cuh -- the set-up and read-back kernels beside the step: state
// reduction (first dt, conservation sums), ghost fill, conversions between
// primitives and conserved totals.  Templated on precision and arithmetic
// policy (dg_physics.cuh); instantiated by dg_step_fast.cu (fused
// multiply-add allowed) and dg_step_ref.cu (compiled with --fmad=false:
// reference rounding).
#pragma once
#include <cstdio>

#include "dg_common.cuh"
#include "dg_host.h"

namespace dg {

// ---------------------------------------------------------------------------
// Helper kernels (set-up and read-back; not on the per-step path)
// ---------------------------------------------------------------------------

// Reduction of the current state (dt of the first step, conservation sums).
template <class T, bool EXACT>
__global__ void __launch_bounds__(256) reduce_kernel(const GridArgs<T> a, int set_dt) {
    __shared__ double red[8 * 7];
    __shared__ int is_last;
    const int tid = threadIdx.x;
    const long long nyi = a.ny - 4, nzi = a.nz - 4;
    const long long total = (long long)(a.nx - 4) * nyi * nzi;
    double sum[5] = {0, 0, 0, 0, 0};
    double wm = INFINITY;
    unsigned nanf = 0;
    float smax = 0.0f;   // fast policy: max wave speed (NaN-propagating)
    // the cells c = blockIdx.x * 256 + tid + k * stride, with (x, y, z)
    // advanced by the stride's own decomposition (no division per cell)
    const long long stride = (long long)gridDim.x * 256;
    long long c = blockIdx.x * 256LL + tid;
    int x = (int)(c / (nyi * nzi)), y = (int)((c / nzi) % nyi), z = (int)(c % nzi);
    const int sx = (int)(stride / (nyi * nzi)), sy = (int)((stride / nzi) % nyi), sz = (int)(stride % nzi);
    for (; c < total; c += stride) {
        const long long o = ((long long)(x + 2) * a.ny + (y + 2)) * a.pitch + (z + 2);
        z += sz;
        if (z >= nzi) { z -= (int)nzi; ++y; }
        y += sy;
        if (y >= nyi) { y -= (int)nyi; ++x; }
        x += sx;
        T u[5], w[5];
        for (int f = 0; f < 5; ++f) u[f] = a.src[f * a.fstride + o];
        Phys<T, EXACT>::prim(u, w, a.k);
        if constexpr (EXACT) {
            const T wd = Phys<T, EXACT>::wave_dt(w, a.k);
            if (wd != wd) nanf = 1;
            else wm = fmin(wm, (double)wd);
        } else {
            smax = max_nan(smax, fast_speed(w[0], w[1], w[2], w[3], w[4], a.k.gamma));
        }
        for (int f = 0; f < 5; ++f) sum[f] += (double)u[f];
    }
    if constexpr (!EXACT) {
        if (smax != smax) nanf = 1;
        else wm = (double)__fdiv_rn(a.k.ds, smax);
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int f = 0; f < 5; ++f) sum[f] += __shfl_xor_sync(0xffffffffu, sum[f], o);
        wm = fmin(wm, __shfl_xor_sync(0xffffffffu, wm, o));
        nanf |= __shfl_xor_sync(0xffffffffu, nanf, o);
    }
    if ((tid & 31) == 0) {
        for (int f = 0; f < 5; ++f) red[(tid >> 5) * 7 + f] = sum[f];
        red[(tid >> 5) * 7 + 5] = wm;
        red[(tid >> 5) * 7 + 6] = (double)nanf;
    }
    __syncthreads();
    if (tid == 0) {
        Partial p;
        for (int f = 0; f < 5; ++f) p.sums[f] = 0;
        p.wmin = INFINITY;
        p.nan = 0;
        for (int w = 0; w < 8; ++w) {
            for (int f = 0; f < 5; ++f) p.sums[f] += red[w * 7 + f];
            p.wmin = fmin(p.wmin, red[w * 7 + 5]);
            p.nan |= red[w * 7 + 6] != 0.0;
        }
        p.pad = 0;
        a.part[blockIdx.x] = p;
        __threadfence();
        is_last = atomicAdd(&a.ctl->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    final_reduce<T>(a, tid, 256, red, set_dt ? kSetDt : kSumsOnly, gridDim.x);
}

// Copy every ghost cell of buf from its interior source (boundary rules).
// Ghost cell e (0 .. ghost_cells - 1) as ghosted coordinates: the two
// layers of each x face (4 ny nz cells), then those of each y face over the
// interior x (4 (nx-4) nz), then those of each z face over the interior x, y
// (4 (nx-4)(ny-4)).
__device__ __forceinline__ void ghost_cell(long long e, int nx, int ny, int nz, int &x, int &y, int &z) {
    const long long fx = 4LL * ny * nz, fy = 4LL * (nx - 4) * nz;
    if (e < fx) {
        const int s = (int)(e / ((long long)ny * nz));
        const long long r = e - (long long)s * ny * nz;
        x = s < 2 ? s : nx - 4 + s;
        y = (int)(r / nz);
        z = (int)(r - (long long)y * nz);
    } else if (e < fx + fy) {
        e -= fx;
        const int xi = (int)(e / (4LL * nz));
        const int r = (int)(e - (long long)xi * 4 * nz);
        const int s = r / nz;
        x = xi + 2;
        y = s < 2 ? s : ny - 4 + s;
        z = r - s * nz;
    } else {
        e -= fx + fy;
        const long long row = e >> 2;
        const int s = (int)(e & 3);
        x = (int)(row / (ny - 4)) + 2;
        y = (int)(row - (long long)(x - 2) * (ny - 4)) + 2;
        z = s < 2 ? s : nz - 4 + s;
    }
}

template <class T> __global__ void fill_ghosts_kernel(const GridArgs<T> a, T *buf) {
    const long long total = (long long)a.nx * a.ny * a.nz - (long long)(a.nx - 4) * (a.ny - 4) * (a.nz - 4);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total;
         c += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        ghost_cell(c, a.nx, a.ny, a.nz, x, y, z);
        int fx, fy, fz;
        const int sx = axis_source(x, a.nx, a.bc[0], a.bc[1], &fx);
        const int sy = axis_source(y, a.ny, a.bc[2], a.bc[3], &fy);
        const int sz = axis_source(z, a.nz, a.bc[4], a.bc[5], &fz);
        const long long o = ((long long)x * a.ny + y) * a.pitch + z;
        const long long so = ((long long)sx * a.ny + sy) * a.pitch + sz;
        buf[o] = buf[so];
        buf[a.fstride + o] = fx ? -buf[a.fstride + so] : buf[a.fstride + so];
        buf[2 * a.fstride + o] = fy ? -buf[2 * a.fstride + so] : buf[2 * a.fstride + so];
        buf[3 * a.fstride + o] = fz ? -buf[3 * a.fstride + so] : buf[3 * a.fstride + so];
        buf[4 * a.fstride + o] = buf[4 * a.fstride + so];
    }
}

// calc_conserved over the interior (physics.rs:143-175); prim is dense
// with its own pitch/field stride.
template <class T>
__global__ void prim_to_cons_kernel(const GridArgs<T> a, const T *prim, long long pfs, int ppitch, T *cons) {
    const long long total = (long long)a.nx * a.ny * a.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total;
         c += (long long)gridDim.x * blockDim.x) {
        const long long xy = c / a.nz;
        const int z = (int)(c % a.nz);
        const long long po = xy * ppitch + z, co = xy * a.pitch + z;
        T w[5], u[5];
        for (int f = 0; f < 5; ++f) w[f] = prim[f * pfs + po];
        prim_to_cons(w, u, a.k.vol, a.k.gm1);
        for (int f = 0; f < 5; ++f) cons[f * a.fstride + co] = u[f];
    }
}

// calc_primitives over every cell (ghosts included).
template <class T, bool EXACT>
__global__ void cons_to_prim_kernel(const GridArgs<T> a, const T *cons, T *prim, long long pfs, int ppitch) {
    const long long total = (long long)a.nx * a.ny * a.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total;
         c += (long long)gridDim.x * blockDim.x) {
        const long long xy = c / a.nz;
        const int z = (int)(c % a.nz);
        const long long po = xy * ppitch + z, co = xy * a.pitch + z;
        T u[5], w[5];
        for (int f = 0; f < 5; ++f) u[f] = cons[f * a.fstride + co];
        Phys<T, EXACT>::prim(u, w, a.k);
        for (int f = 0; f < 5; ++f) prim[f * pfs + po] = w[f];
    }
}

// ---------------------------------------------------------------------------
// Launch wrappers (instantiated per policy by the two translation units)
// ---------------------------------------------------------------------------
template <class T, bool EXACT> cudaError_t launch_reduce_policy(const GridArgs<T> &a, int set_dt, cudaStream_t st) {
    const long long total = (long long)(a.nx - 4) * (a.ny - 4) * (a.nz - 4);
    long long blocks = (total + 255) / 256;
    if (blocks > kReduceBlocks) blocks = kReduceBlocks;
    reduce_kernel<T, EXACT><<<(int)blocks, 256, 0, st>>>(a, set_dt);
    return cudaGetLastError();
}

inline int flat_blocks(long long total) {
    long long b = (total + 255) / 256;
    if (b > kSms * 16) b = kSms * 16;
    if (b < 1) b = 1;
    return (int)b;
}

template <class T, bool EXACT>
cudaError_t launch_cons_to_prim_policy(const GridArgs<T> &a, const T *cons, T *prim, long long pfs, int ppitch,
                                       cudaStream_t st) {
    cons_to_prim_kernel<T, EXACT><<<flat_blocks((long long)a.nx * a.ny * a.nz), 256, 0, st>>>(a, cons, prim, pfs,
                                                                                             ppitch);
    return cudaGetLastError();
}

}  // namespace dg
