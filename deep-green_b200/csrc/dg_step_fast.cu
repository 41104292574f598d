// dg_step_fast.cu -- the FP32 fused-arithmetic step (fast policy;
// multiply-add contraction allowed).  Kernels: dg_sweep_impl.cuh,
// dg_step_impl.cuh.
#include "dg_host.h"
#include "dg_step_impl.cuh"
#include "dg_sweep_impl.cuh"

namespace dg {

namespace {
// five staged planes when they fit in shared memory, else four
constexpr int kSweepRing = sizeof(sweep::Smem<float, kSweepRowsF32, 5>) + 1024 <= 232448 ? 5 : 4;

// One step: with interior tiles (InteriorTiles) two launches sharing one
// reduction -- the interior tiles, with the owned warps' boundary switches
// compiled out (419 instead of 594 instructions per cell), in whole columns
// when they fill the SMs and else in `chunk`-plane blocks
// (interior_chunk), then the frame in `chunk`-plane blocks, launched as a
// programmatic dependent so that it fills the SMs the interior launch's last
// wave leaves free.  Without interior tiles, one launch of the general
// kernel over all tiles.  (One kernel body holding both variants of the
// loop ran slower than either alone.)
template <int LIM, bool GRAV>
cudaError_t launch_sweep_t(const GridArgs<float> &a, const CUtensorMap *tmap, int chunk, cudaStream_t st) {
    constexpr int TY = kSweepRowsF32, R = kSweepRing;
    auto k_in = sweep::sweep_step_kernel<float, TY, R, LIM, GRAV, true>;
    auto k_frame = sweep::sweep_step_kernel<float, TY, R, LIM, GRAV, false>;
    constexpr int smem = sweep::smem_bytes<float, TY, R>();
    static std::atomic<unsigned long long> attr_in{0}, attr_frame{0};
    cudaError_t e = ensure_dynamic_smem(k_in, smem, attr_in);
    if (e == cudaSuccess) e = ensure_dynamic_smem(k_frame, smem, attr_frame);
    if (e != cudaSuccess) return e;
    const InteriorTiles it(a.ny, a.nz, TY, sweep::kTileZ);
    const int chunk_in = interior_chunk(a.nx, it, chunk);
    const int n_in = it.interior() * ((a.nx - 4 + chunk_in - 1) / chunk_in);
    const int n_fr = it.frame() * ((a.nx - 4 + chunk - 1) / chunk);
    const int nparts = n_in + n_fr;
    if (n_in > 0) {
        k_in<<<n_in, 32 * (TY + 2), smem, st>>>(a, *tmap, chunk_in, nparts);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return launch_after(k_frame, n_fr, 32 * (TY + 2), smem, st, n_in > 0 || (a.chain & kChainWait), a, *tmap, chunk,
                        nparts);
}

}  // namespace

// One kernel per (limiter, gravity): the slope and flux code of the march
// is fixed at compile time.
cudaError_t launch_sweep(const GridArgs<float> &a, const CUtensorMap *tmap, int chunk, cudaStream_t st) {
    if (a.gravity)
        return a.limiter == 0 ? launch_sweep_t<0, true>(a, tmap, chunk, st) : launch_sweep_t<1, true>(a, tmap, chunk, st);
    return a.limiter == 0 ? launch_sweep_t<0, false>(a, tmap, chunk, st) : launch_sweep_t<1, false>(a, tmap, chunk, st);
}

template cudaError_t launch_cons_to_prim_policy<float, false>(const GridArgs<float> &, const float *, float *,
                                                              long long, int, cudaStream_t);
}  // namespace dg
