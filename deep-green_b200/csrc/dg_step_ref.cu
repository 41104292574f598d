// dg_step_ref.cu -- the reference-rounding policy (FP64, and FP32 on
// request).  This file is compiled with --fmad=false so that no multiply-add
// is fused and every operation rounds as in the reference's scalar code.
// Also holds the set-up kernels, part of which must round like the reference
// (calc_conserved), and the FP64 step with fused arithmetic (every fused
// operation is written as one).  Kernels:
// dg_march_impl.cuh, dg_step_impl.cuh.
#include "dg_march_impl.cuh"
#include "dg_step_impl.cuh"

namespace dg {

cudaError_t launch_march(const GridArgs<double> &a, const CUtensorMap *tmap, int kind, int chunk, cudaStream_t st) {
    const int blocks = step_grid_blocks(a.nx, a.ny, a.nz, kind, chunk);
    return kind == kFastF64
               ? march::launch<double, march::FusedArith, kMarchRows, kMarchRing>(a, tmap, blocks, chunk, st)
               : march::launch<double, march::RefArith<double>, kMarchRows, kMarchRing>(a, tmap, blocks, chunk, st);
}

cudaError_t launch_march(const GridArgs<float> &a, const CUtensorMap *tmap, int kind, int chunk, cudaStream_t st) {
    const int blocks = step_grid_blocks(a.nx, a.ny, a.nz, kind, chunk);
    return march::launch<float, march::RefArith<float>, kMarchRows, kMarchRing>(a, tmap, blocks, chunk, st);
}

template <class T, bool EXACT, bool PRIM>
static void set_state(const GridArgs<T> &a, const FieldView<const T> &src, bool vec, unsigned long long step,
                      cudaStream_t st) {
    const int blocks = row_blocks((long long)a.nx * a.ny);
    if (vec) set_state_kernel<T, EXACT, PRIM, kVec<T>><<<blocks, 256, 0, st>>>(a, src, step);
    else set_state_kernel<T, EXACT, PRIM, 1><<<blocks, 256, 0, st>>>(a, src, step);
}

template <class T>
cudaError_t launch_set_state(const GridArgs<T> &a, const FieldView<const T> &src, bool prims, bool exact,
                             unsigned long long step, cudaStream_t st) {
    T *const dst[5] = {a.dst, a.dst + a.fstride, a.dst + 2 * a.fstride, a.dst + 3 * a.fstride, a.dst + 4 * a.fstride};
    const bool vec = vector_rows(src, dst, a.pitch);
    if (exact || sizeof(T) == 8) {
        if (prims) set_state<T, true, true>(a, src, vec, step, st);
        else set_state<T, true, false>(a, src, vec, step, st);
    } else if constexpr (sizeof(T) == 4) {
        if (prims) set_state<T, false, true>(a, src, vec, step, st);
        else set_state<T, false, false>(a, src, vec, step, st);
    }
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_get_state(const FieldView<const T> &src, T *const dst[5], int n0, int n1, int n2, cudaStream_t st) {
    const FieldView<T> d{{dst[0], dst[1], dst[2], dst[3], dst[4]}, 0, 0, 1};
    const int blocks = row_blocks(5LL * n0 * n1);
    if (vector_rows(src, dst, n2)) get_state_kernel<T, kVec<T>><<<blocks, 256, 0, st>>>(src, d, n0, n1, n2);
    else get_state_kernel<T, 1><<<blocks, 256, 0, st>>>(src, d, n0, n1, n2);
    return cudaGetLastError();
}

template <class T> cudaError_t launch_sums(const GridArgs<T> &a, cudaStream_t st) { return launch_sums_kernel(a, st); }

#define DG_REF_INSTANTIATE(T)                                                                                      \
    template cudaError_t launch_sums<T>(const GridArgs<T> &, cudaStream_t);                                         \
    template cudaError_t launch_cons_to_prim_policy<T, true>(const GridArgs<T> &, const T *, T *, long long, int,   \
                                                             cudaStream_t);                                        \
    template cudaError_t launch_set_state<T>(const GridArgs<T> &, const FieldView<const T> &, bool, bool,           \
                                             unsigned long long, cudaStream_t);                                    \
    template cudaError_t launch_get_state<T>(const FieldView<const T> &, T *const[5], int, int, int, cudaStream_t);

DG_REF_INSTANTIATE(float)
DG_REF_INSTANTIATE(double)

}  // namespace dg
