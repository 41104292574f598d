// dg_common.cuh -- pieces shared by the step kernels: PTX wrappers for
// mbarrier and TMA, the ghost-image rules of the reference's boundary
// conditions, and the fixed-order reduction of per-block partials.
#pragma once
#include <cstdio>

#include "dg_kernels.cuh"

namespace dg {

// ---------------------------------------------------------------------------
// PTX helpers (mbarrier, TMA)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_inval(uint64_t *bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bounded wait on an mbarrier phase: false after ~`budget` SM clocks; a
// negative budget gives up without waiting (the timeout test hook).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long budget) {
    if (budget < 0) return false;
    const uint32_t addr = smem_u32(bar);
    auto try_wait = [&]() {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        return ok != 0;
    };
    if (try_wait()) return true;   // the usual case: no clock reads
    const long long t0 = clock64();
    while (true) {
        if (try_wait()) return true;
        if (clock64() - t0 > budget) return false;
    }
}

// 4-D tiled TMA load (z, y, x, field) into shared memory, completing on bar.
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int c0, int c1, int c2,
                                            int c3, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

constexpr long long kWaitBudget = 4000000000LL;  // ~2 s of SM clock

// The budget a step kernel gives its waits for staged planes: the grid's own
// (a context created with DG_DEBUG_WAIT_BUDGET set; negative: give up at
// once) or the default (0).  Waits that let copies in flight land before a
// block exits keep kWaitBudget.
template <class A> __device__ __forceinline__ long long wait_budget_of(const A &a) {
    return a.wait_budget != 0 ? a.wait_budget : kWaitBudget;
}

// 8 floats of read-only memory with one 32-byte load (p 32-byte aligned).
__device__ __forceinline__ void load8_f32(const float *p, float *v) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}

// ---------------------------------------------------------------------------
// Ghost images along one axis of extent n: bit g (0-3) is set when ghost index
// 0, 1, n-2, n-1 holds an image of interior coordinate c (boundaries.rs /
// handle_walls source rules, inverted), bit 4 + g when that image is a wall's
// mirror (normal momentum negated).
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ unsigned image_bits(int c, int n, int lo, int hi) {
    unsigned b = 0;
    if (lo == kPeriodic) {
        if (c == n - 4) b |= 1u;
        if (c == n - 3) b |= 2u;
    } else if (lo == kOutflow) {
        if (c == 2) b |= 3u;
    } else {
        if (c == 2) b |= 0x22u;
        if (c == 3) b |= 0x11u;
    }
    if (hi == kPeriodic) {
        if (c == 2) b |= 4u;
        if (c == 3) b |= 8u;
    } else if (hi == kOutflow) {
        if (c == n - 3) b |= 12u;
    } else {
        if (c == n - 3) b |= 0x44u;
        if (c == n - 4) b |= 0x88u;
    }
    return b;
}
__host__ __device__ __forceinline__ int ghost_at(int g, int n) { return g < 2 ? g : n - 4 + g; }

// Source interior coordinate of ghosted coordinate g along one axis, and
// whether the copy is a wall mirror.
__host__ __device__ __forceinline__ int axis_source(int g, int n, int lo, int hi, int *flip) {
    *flip = 0;
    if (g >= 2 && g <= n - 3) return g;
    if (g < 2) {
        if (lo == kPeriodic) return g == 0 ? n - 4 : n - 3;
        if (lo == kOutflow) return 2;
        *flip = 1;
        return g == 1 ? 2 : 3;
    }
    if (hi == kPeriodic) return g == n - 2 ? 2 : 3;
    if (hi == kOutflow) return n - 3;
    *flip = 1;
    return g == n - 2 ? n - 3 : n - 4;
}

// Wave speeds (>= 0, or NaN) as unsigned keys of the same order, NaN on top.
__device__ __forceinline__ unsigned long long speed_key(float v) {
    return v != v ? 0x7fffffffull : (unsigned long long)(__float_as_uint(v) & 0x7fffffffu);
}
__device__ __forceinline__ unsigned long long speed_key(double v) {
    return v != v ? 0x7fffffffffffffffull : (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ void key_speed(unsigned long long k, float &v) { v = __uint_as_float((unsigned)k); }
__device__ __forceinline__ void key_speed(unsigned long long k, double &v) { v = __longlong_as_double((long long)k); }
__device__ __forceinline__ unsigned long long warp_max(float v) {
    return __reduce_max_sync(0xffffffffu, (unsigned)speed_key(v));
}
__device__ __forceinline__ unsigned long long warp_max(double v) {
    unsigned long long k = speed_key(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long n = __shfl_xor_sync(0xffffffffu, k, o);
        k = n > k ? n : k;
    }
    return k;
}

// The launch's largest wave speed, and by its last block (of the nb of this
// grid) the next dt: calc_timestep's CFL * min(ds / speed) is CFL * (ds / max
// speed), division being monotone, or CFL * 1.0 when a NaN was seen
// (physics.rs:191-195).  A maximum does not depend on its order, so one
// atomic per warp in shared memory and one per block in the control block
// replace partial results; s_max is zeroed before a barrier that precedes
// the call.  ADVANCE: a step finished (record its dt, advance the counter);
// else a state was set before step `step`.
template <bool ADVANCE, class T>
__device__ __forceinline__ void finish_speed(const GridArgs<T> &a, T smax, unsigned long long *s_max, int nb,
                                             unsigned long long step = 0) {
    const unsigned long long k = warp_max(smax);
    if ((threadIdx.x & 31) == 0) atomicMax(s_max, k);
    __syncthreads();
    if (threadIdx.x != 0) return;
    DevCtl *c = a.ctl;
    atomicMax(&c->wmax, *s_max);
    __threadfence();
    if (atomicAdd(&c->counter, 1u) != (unsigned)nb - 1) return;
    __threadfence();
    T m;
    key_speed(atomicExch(&c->wmax, 0ull), m);
    const bool nan = m != m;
    const T dtn = nan ? a.k.cfl * T(1.0) : a.k.cfl * (a.k.ds / m);
    if constexpr (ADVANCE) {
        const unsigned long long st = c->step;
        c->hist[st % kHist] = c->dt[st & 1];
        c->dt[(st + 1) & 1] = (double)dtn;
        c->step = st + 1;
        if (nan) c->flags |= kStatusNonFinite;
    } else {
        c->dt[step & 1] = (double)dtn;
        c->step = step;
        c->flags = nan ? kStatusNonFinite : 0u;
    }
    c->counter = 0;
    __threadfence();
}

}  // namespace dg
