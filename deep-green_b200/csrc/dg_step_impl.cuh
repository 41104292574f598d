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

// FP64 sums of the conserved fields over the interior, in a fixed order.
template <class T> __global__ void __launch_bounds__(256) sums_kernel(const GridArgs<T> a) {
    __shared__ double red[8][5];
    __shared__ int is_last;
    const int tid = threadIdx.x;
    const long long nyi = a.ny - 4, nzi = a.nz - 4;
    const long long total = (long long)(a.nx - 4) * nyi * nzi;
    double sum[5] = {0, 0, 0, 0, 0};
    // the cells c = blockIdx.x * 256 + tid + k * stride, with (x, y, z)
    // advanced by the stride's own decomposition (no division per cell)
    const long long stride = (long long)gridDim.x * 256;
    long long c = blockIdx.x * 256LL + tid;
    int x = (int)(c / (nyi * nzi)), y = (int)((c / nzi) % nyi), z = (int)(c % nzi);
    const int sx = (int)(stride / (nyi * nzi)), sy = (int)((stride / nzi) % nyi), sz = (int)(stride % nzi);
    // kAhead cells' loads in flight before their additions, which keep their
    // order (508^3 FP32 985 us with one load after the other, 687 / 620 / 500 /
    // 672 with 1 / 2 / 4 / 8 cells; 300^3 FP64 243, 203 / 254 / 192 / 292)
    constexpr int kAhead = 4;
    while (c < total) {
        T u[kAhead][5];
        const long long left = (total - 1 - c) / stride;   // cells behind this one
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const long long o = ((long long)(x + 2) * a.ny + (y + 2)) * a.pitch + (z + 2);
#pragma unroll
            for (int f = 0; f < 5; ++f) u[k][f] = k <= left ? a.src[f * a.fstride + o] : T(0);
            z += sz;
            if (z >= nzi) { z -= (int)nzi; ++y; }
            y += sy;
            if (y >= nyi) { y -= (int)nyi; ++x; }
            x += sx;
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (k <= left) {
#pragma unroll
                for (int f = 0; f < 5; ++f) sum[f] += (double)u[k][f];
            }
        c += kAhead * stride;
    }
    auto block_sum = [&](int f) {
        double t = 0;
        for (int w = 0; w < 8; ++w) t += red[w][f];
        return t;
    };
    auto warps_to_red = [&] {
        for (int o = 16; o > 0; o >>= 1)
            for (int f = 0; f < 5; ++f) sum[f] += __shfl_xor_sync(0xffffffffu, sum[f], o);
        if ((tid & 31) == 0)
            for (int f = 0; f < 5; ++f) red[tid >> 5][f] = sum[f];
        __syncthreads();
    };
    warps_to_red();
    if (tid == 0) {
        for (int f = 0; f < 5; ++f) a.part[blockIdx.x].sums[f] = block_sum(f);
        __threadfence();
        is_last = atomicAdd(&a.ctl->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int f = 0; f < 5; ++f) sum[f] = 0;
    for (unsigned b = tid; b < gridDim.x; b += 256) {
        const volatile Partial *p = a.part + b;
        for (int f = 0; f < 5; ++f) sum[f] += p->sums[f];
    }
    warps_to_red();
    if (tid == 0) {
        for (int f = 0; f < 5; ++f) a.ctl->sums[f] = block_sum(f);
        a.ctl->counter = 0;
        __threadfence();
    }
}

// V consecutive values; V > 1 is one 16-byte access.
template <class T, int V> struct alignas(V * sizeof(T)) Quad {
    T v[V];
};
template <class T> constexpr int kVec = 16 / (int)sizeof(T);

// A state into the pitched layout: every ghosted cell from its interior
// source (the boundary rules' composed per-axis sources), converted from
// primitives if asked (calc_conserved, physics.rs:143-175), and the interior's
// largest wave speed, i.e. the dt of the coming step.  Bound by memory: one
// pass in place of a copy per field, a ghost fill and a reduction.  One warp
// per row, V values per lane (V > 1: 16-byte accesses, for views whose rows
// allow them).
template <class T, bool EXACT, bool PRIM, int V>
__global__ void __launch_bounds__(256) set_state_kernel(const GridArgs<T> a, const FieldView<const T> src,
                                                        unsigned long long step) {
    __shared__ unsigned long long s_max;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = gridDim.x * 8;
    const int rows = a.nx * a.ny;
    const bool in_place = !PRIM && src.f[0] == a.dst;
    T smax = T(0);
    for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += nw) {
        const int x = row / a.ny, y = row - x * a.ny;
        int fx, fy;
        const int sx = axis_source(x, a.nx, a.bc[0], a.bc[1], &fx);
        const int sy = axis_source(y, a.ny, a.bc[2], a.bc[3], &fy);
        const bool inner_row = sx == x && sy == y;
        const long long so = sx * src.sx + sy * src.sy, o = (long long)row * a.pitch;
        for (int z = lane * V; z < a.nz; z += 32 * V) {
            Quad<T, V> u[5];
            const bool inner_z = z >= 2 && z + V <= a.nz - 2;
            bool fz[V];
            if (V > 1 && inner_z) {
#pragma unroll
                for (int f = 0; f < 5; ++f) u[f] = *reinterpret_cast<const Quad<T, V> *>(src.f[f] + so + z);
#pragma unroll
                for (int i = 0; i < V; ++i) fz[i] = false;
            } else {
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    int flip;
                    const int sz = axis_source(min(z + i, a.nz - 1), a.nz, a.bc[4], a.bc[5], &flip);
                    fz[i] = flip != 0;
#pragma unroll
                    for (int f = 0; f < 5; ++f) u[f].v[i] = src.f[f][so + sz * src.sz];
                }
            }
#pragma unroll
            for (int i = 0; i < V; ++i) {
                T w[5], c[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) c[f] = u[f].v[i];
                if constexpr (PRIM) {
                    T q[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) q[f] = c[f];
                    prim_to_cons(q, c, a.k.vol, a.k.gm1);
                }
                if (inner_row && z + i >= 2 && z + i < a.nz - 2) {
                    T sp;
                    Phys<T, EXACT>::prim(c, w, a.k);
                    if constexpr (EXACT)
                        sp = sqrt(a.k.gamma * w[4] / w[0]) + sqrt(w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
                    else sp = fast_speed(w[0], w[1], w[2], w[3], w[4], a.k.gamma);
                    smax = (smax != smax || sp != sp) ? smax + sp : (sp > smax ? sp : smax);
                }
                u[0].v[i] = c[0];
                u[1].v[i] = fx ? -c[1] : c[1];
                u[2].v[i] = fy ? -c[2] : c[2];
                u[3].v[i] = fz[i] ? -c[3] : c[3];
                u[4].v[i] = c[4];
            }
            if (in_place && inner_row && inner_z) continue;
            if (z + V <= a.nz) {
#pragma unroll
                for (int f = 0; f < 5; ++f) *reinterpret_cast<Quad<T, V> *>(a.dst + f * a.fstride + o + z) = u[f];
            } else {
#pragma unroll
                for (int f = 0; f < 5; ++f)
#pragma unroll
                    for (int i = 0; i < V; ++i)
                        if (z + i < a.nz) a.dst[f * a.fstride + o + z + i] = u[f].v[i];
            }
        }
    }
    finish_speed<false>(a, smax, &s_max, gridDim.x, step);
}

// Five dense arrays of n0 x n1 x n2 cells from a state seen through strides;
// one warp per row, field after field, so that the rows in flight lie
// together (all five fields per row: 2.6 ms at 512^3 FP32).
template <class T, int V>
__global__ void __launch_bounds__(256) get_state_kernel(const FieldView<const T> src, const FieldView<T> dst, int n0,
                                                        int n1, int n2) {
    const int lane = threadIdx.x & 31, nw = gridDim.x * 8, rows = n0 * n1;
    for (long long r = blockIdx.x * 8 + (threadIdx.x >> 5); r < 5LL * rows; r += nw) {
        const int f = (int)(r / rows), row = (int)(r - (long long)f * rows);
        const int i = row / n1, j = row - i * n1;
        const T *s = src.f[0];
        T *d = dst.f[0];
#pragma unroll
        for (int g = 1; g < 5; ++g)
            if (f == g) {
                s = src.f[g];
                d = dst.f[g];
            }
        s += i * src.sx + j * src.sy;
        d += (long long)row * n2;
        if constexpr (V > 1) {
#pragma unroll 4
            for (int k = lane; k < n2 / V; k += 32)
                reinterpret_cast<Quad<T, V> *>(d)[k] = reinterpret_cast<const Quad<T, V> *>(s)[k];
        } else {
#pragma unroll 4
            for (int k = lane; k < n2; k += 32) d[k] = s[k * src.sz];
        }
    }
}

// Whether every row of the view, and of rows `n` values apart behind the other
// pointers, starts on a 16-byte boundary and its values are adjacent.
template <class T, class U> inline bool vector_rows(const FieldView<T> &v, U *const other[5], long long n) {
    if (v.sz != 1 || v.sx % kVec<U> || v.sy % kVec<U> || n % kVec<U>) return false;
    uintptr_t bits = 0;
    for (int f = 0; f < 5; ++f) bits |= reinterpret_cast<uintptr_t>(v.f[f]) | reinterpret_cast<uintptr_t>(other[f]);
    return (bits & 15) == 0;
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
template <class T> cudaError_t launch_sums_kernel(const GridArgs<T> &a, cudaStream_t st) {
    const long long total = (long long)(a.nx - 4) * (a.ny - 4) * (a.nz - 4);
    long long blocks = (total + 255) / 256;
    if (blocks > kReduceBlocks) blocks = kReduceBlocks;
    sums_kernel<T><<<(int)blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

// Blocks of the row kernels: one row per warp, 8 blocks of 8 warps per SM.
inline int row_blocks(long long rows) {
    const long long b = (rows + 7) / 8;
    return (int)(b > kSms * 8 ? kSms * 8 : b);
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
