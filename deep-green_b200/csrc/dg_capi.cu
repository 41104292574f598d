// dg_capi.cu -- the C ABI declared in include/deepgreen.h.
//
// A context owns two device copies of the ghosted state (the step reads one
// and writes the other), the step control block (dt, sums, history) and
// the partials of the sum reduction, plus one TMA descriptor per state buffer.
#include <cudaTypedefs.h>

#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>

#include "../../include/deepgreen.h"
#include "dg_ctx.h"
#include "dg_pointer.h"

using namespace dg;


namespace {

// message of the calling thread's last failure outside a context
thread_local std::string g_create_err = "no error";

// A driver function by name, or NULL.
template <class Fn> Fn driver_fn(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
        return reinterpret_cast<Fn>(p);
    return nullptr;
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
    static const auto fn = driver_fn<PFN_cuTensorMapEncodeTiled_v12000>("cuTensorMapEncodeTiled");
    return fn;
}

// What the driver says of p (nothing known: not device memory).
PointerInfo pointer_info(const void *p) {
    static const auto get = driver_fn<PFN_cuPointerGetAttributes_v7000>("cuPointerGetAttributes");
    static const auto current = driver_fn<PFN_cuCtxGetCurrent_v4000>("cuCtxGetCurrent");
    PointerInfo m = {false, -1, false, 0, 0};
    unsigned type = 0, managed = 0;
    int device = -1;
    CUcontext owner = nullptr, own = nullptr;
    unsigned long long start = 0;
    size_t size = 0;
    CUpointer_attribute attr[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE,      CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL,   CU_POINTER_ATTRIBUTE_CONTEXT,
                                  CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void *out[] = {&type, &managed, &device, &owner, &start, &size};
    if (!get || !current || current(&own) != CUDA_SUCCESS ||
        get(6, attr, out, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS)
        return m;
    m.device_memory = type == CU_MEMORYTYPE_DEVICE && !managed;
    m.device = device;
    m.foreign_context = owner && owner != own;      // memory of pools has no context
    m.start = (uintptr_t)start;
    m.size = size;
    return m;
}

int auto_chunk(const dg_ctx *c) {
    return c->chunk > 0 ? c->chunk : c->chunk_auto;
}

int encode_map(dg_ctx *c, int i) {
    auto fn = get_encode_fn();
    if (!fn) return fail(c, DG_ERR_CUDA, "cuTensorMapEncodeTiled not available from the driver");
    const int ty = step_tile_rows(c->kind);
    cuuint64_t dims[4] = {(cuuint64_t)c->nz, (cuuint64_t)c->ny, (cuuint64_t)c->nx, 5};
    cuuint64_t strides[3] = {(cuuint64_t)c->pitch * c->elem, (cuuint64_t)c->pitch * c->ny * c->elem,
                             (cuuint64_t)c->fstride * c->elem};
    cuuint32_t box[4] = {(cuuint32_t)step_box_cols(c->kind), (cuuint32_t)(ty + 4), 1, 5};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(&c->tmap[i], c->elem == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                    4, c->buf[i], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(c, DG_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return DG_OK;
}

int use_device(dg_ctx *c) {
    DG_CUDA(c, cudaSetDevice(c->info.device));
    return DG_OK;
}

// The control fields before the dt history; a launch that timed out may
// have left its counters half way.
int reset_ctl(dg_ctx *c) {
    DG_CUDA(c, cudaMemsetAsync(c->ctl, 0, offsetof(DevCtl, hist), c->stream));
    return DG_OK;
}

// Five arrays of the ghosted extents, C order.
template <class T> FieldView<T> dense_view(const dg_ctx *c, void *const f[5]) {
    FieldView<T> v;
    for (int i = 0; i < 5; ++i) v.f[i] = static_cast<T *>(f[i]);
    v.sx = (long long)c->ny * c->nz;
    v.sy = c->nz;
    v.sz = 1;
    return v;
}

// Five consecutive dense fields at base.
struct Fields5 {
    void *f[5];
};
Fields5 consecutive(const dg_ctx *c, const void *base) {
    const size_t fb = (size_t)c->nx * c->ny * c->nz * c->elem;
    Fields5 r;
    for (int i = 0; i < 5; ++i) r.f[i] = const_cast<char *>(static_cast<const char *>(base)) + i * fb;
    return r;
}

// A pitched state buffer seen through strides.
template <class T> FieldView<T> pitched_view(const dg_ctx *c, const void *buf) {
    FieldView<T> v;
    for (int i = 0; i < 5; ++i) v.f[i] = const_cast<T *>(static_cast<const T *>(buf)) + i * c->fstride;
    v.sx = (long long)c->ny * c->pitch;
    v.sy = c->pitch;
    v.sz = 1;
    return v;
}

// The current state from the dense device fields `src` (NULL: from its own
// interior), ghosts and the first dt included.
template <class T> cudaError_t set_state(dg_ctx *c, void *const src[5], bool prims) {
    const auto a = grid_args<T>(c, c->buf[c->cur], c->buf[c->cur]);
    const FieldView<const T> v = src ? dense_view<const T>(c, src) : pitched_view<const T>(c, c->buf[c->cur]);
    return launch_set_state<T>(a, v, prims, c->exact, 0, c->stream);
}

int finish_state(dg_ctx *c, void *const src[5] = nullptr, bool prims = false) {
    const cudaError_t e = c->elem == 8 ? set_state<double>(c, src, prims) : set_state<float>(c, src, prims);
    if (e != cudaSuccess) return cuda_fail(c, e, "state set-up kernel");
    c->has_state = true;
    c->steps = 0;
    return DG_OK;
}

bool null_field(const void *const f[5]) {
    for (int i = 0; i < 5; ++i)
        if (!f[i]) return true;
    return false;
}

// Host transfers move each field as one contiguous copy (the copy engines'
// fast case; row-by-row copies of the pitched layout from host memory run
// at about half the rate) through a dense device copy of the fields.
size_t dense_field_bytes(const dg_ctx *c) { return (size_t)c->nx * c->ny * c->nz * c->elem; }

int upload_dense(dg_ctx *c, void *dense, const void *const src[5]) {
    const size_t fb = dense_field_bytes(c);
    for (int f = 0; f < 5; ++f)
        DG_CUDA(c, cudaMemcpyAsync(static_cast<char *>(dense) + f * fb, src[f], fb, cudaMemcpyHostToDevice,
                                   c->stream));
    return DG_OK;
}

int download_dense(dg_ctx *c, void *const dst[5], const void *dense) {
    const size_t fb = dense_field_bytes(c);
    for (int f = 0; f < 5; ++f)
        DG_CUDA(c, cudaMemcpyAsync(dst[f], static_cast<const char *>(dense) + f * fb, fb, cudaMemcpyDeviceToHost,
                                   c->stream));
    return DG_OK;
}

// Whether the kernels may access the caller's five dense device fields.
bool kernel_fields(const dg_ctx *c, const void *const f[5]) {
    for (int i = 0; i < 5; ++i)
        if (!kernel_may_access(pointer_info(f[i]), reinterpret_cast<uintptr_t>(f[i]), dense_field_bytes(c),
                               (size_t)c->elem, c->info.device))
            return false;
    return true;
}

// The current state into or from dense device fields that they may not, by
// copies between the layouts.
int copy_fields(dg_ctx *c, void *const dense[5], bool in) {
    const size_t row = (size_t)c->nz * c->elem, pitched = (size_t)c->pitch * c->elem;
    for (int f = 0; f < 5; ++f) {
        char *own = static_cast<char *>(c->buf[c->cur]) + (size_t)f * c->fstride * c->elem;
        DG_CUDA(c, cudaMemcpy2DAsync(in ? own : dense[f], in ? pitched : row, in ? dense[f] : own, in ? row : pitched,
                                     row, (size_t)c->nx * c->ny, cudaMemcpyDeviceToDevice, c->stream));
    }
    return DG_OK;
}

// The current state into dense device fields.
int get_state(dg_ctx *c, void *const dst[5]) {
    cudaError_t e;
    if (c->elem == 8) {
        double *d[5];
        for (int f = 0; f < 5; ++f) d[f] = static_cast<double *>(dst[f]);
        e = launch_get_state<double>(pitched_view<const double>(c, c->buf[c->cur]), d, c->nx, c->ny, c->nz, c->stream);
    } else {
        float *d[5];
        for (int f = 0; f < 5; ++f) d[f] = static_cast<float *>(dst[f]);
        e = launch_get_state<float>(pitched_view<const float>(c, c->buf[c->cur]), d, c->nx, c->ny, c->nz, c->stream);
    }
    return e == cudaSuccess ? DG_OK : cuda_fail(c, e, "state copy kernel");
}

int check_flags(dg_ctx *c) {
    unsigned flags = 0;
    DG_CUDA(c, cudaMemcpyAsync(&flags, &c->ctl->flags, sizeof(flags), cudaMemcpyDeviceToHost, c->stream));
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    if (flags & kStatusTimeout) {
        c->has_state = false;
        return fail(c, DG_ERR_TIMEOUT, "a device-side wait timed out; state invalid, set a new state");
    }
    return DG_OK;
}

int enqueue(dg_ctx *c, int nsteps) {
    const int chunk = auto_chunk(c);
    for (int s = 0; s < nsteps; ++s) {
        const int src = c->cur, dst = 1 - c->cur;
        const int chain = (s > 0 ? kChainWait : 0) | (s + 1 < nsteps ? kChainLet : 0);
        cudaError_t e;
        if (c->elem == 8) {
            auto a = grid_args<double>(c, c->buf[src], c->buf[dst]);
            a.chain = chain;
            e = launch_march(a, &c->tmap[src], c->kind, chunk, c->stream);
        } else {
            auto a = grid_args<float>(c, c->buf[src], c->buf[dst]);
            a.chain = chain;
            e = c->exact ? launch_march(a, &c->tmap[src], c->kind, chunk, c->stream)
                         : launch_sweep(a, &c->tmap[src], chunk, c->stream);
        }
        if (e != cudaSuccess) return cuda_fail(c, e, "step kernel launch");
        c->cur = dst;
        ++c->steps;
    }
    return DG_OK;
}

int read_dts(dg_ctx *c, int nsteps, double *dts) {
    // dt of steps [steps - nsteps, steps) sit in the history ring
    if (nsteps > kHist) return fail(c, DG_ERR_INVALID, "at most 4096 dt values per read");
    if ((unsigned long long)nsteps > c->steps) return fail(c, DG_ERR_INVALID, "fewer steps taken than requested");
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    const unsigned long long first = c->steps - nsteps;
    int done = 0;
    while (done < nsteps) {
        const int pos = (int)((first + done) % kHist);
        const int n = std::min(nsteps - done, kHist - pos);
        DG_CUDA(c, cudaMemcpy(dts + done, &c->ctl->hist[pos], n * sizeof(double), cudaMemcpyDeviceToHost));
        done += n;
    }
    return DG_OK;
}

}  // namespace

// Entry points for the other C-ABI sources of the library (dg_ctx.h).
int dg::ctx_enqueue(dg_ctx *c, int nsteps) { return enqueue(c, nsteps); }

int dg::ctx_begin_state(dg_ctx *c) {
    int r = use_device(c);
    return r != DG_OK ? r : reset_ctl(c);
}

int dg::ctx_finish_state(dg_ctx *c) { return finish_state(c); }

int dg::ctx_check_flags(dg_ctx *c) { return check_flags(c); }

namespace {
// dt of the coming step := dt (the step counter lives on the device)
__global__ void set_next_dt_kernel(DevCtl *ctl, double dt) { ctl->dt[ctl->step & 1] = dt; }
}  // namespace

void dg::set_global_error(const std::string &msg) { g_create_err = msg; }

extern "C" {

int32_t dg_abi_version(void) { return DG_ABI_VERSION; }

int32_t dg_create(const dg_sim_info *info, dg_ctx **out) {
    auto set_err = [](const std::string &m) { g_create_err = m; };
    if (!out) return DG_ERR_INVALID;
    *out = nullptr;
    if (!info) { set_err("null info"); return DG_ERR_INVALID; }
    if (info->nghosts != 2) { set_err("nghosts must be 2"); return DG_ERR_INVALID; }
    if (info->nx < 2 || info->ny < 2 || info->nz < 2) { set_err("each axis needs >= 2 interior cells"); return DG_ERR_INVALID; }
    if (!(info->ds > 0) || !(info->gamma > 1) || !(info->cfl > 0)) { set_err("ds > 0, gamma > 1, cfl > 0 required"); return DG_ERR_INVALID; }
    if (info->precision != DG_F32 && info->precision != DG_F64) { set_err("precision must be DG_F32 or DG_F64"); return DG_ERR_INVALID; }
    if (info->limiter != DG_LIMITER_NONE && info->limiter != DG_LIMITER_MINMOD) { set_err("unknown limiter"); return DG_ERR_INVALID; }
    if (info->rounding != DG_ROUNDING_DEFAULT && info->rounding != DG_ROUNDING_REFERENCE &&
        info->rounding != DG_ROUNDING_FAST) { set_err("unknown rounding policy"); return DG_ERR_INVALID; }
    for (int a = 0; a < 3; ++a) {
        const int lo = info->bcs[2 * a], hi = info->bcs[2 * a + 1];
        if (lo < 0 || lo > DG_BC_CONDUCTING_WALL || hi < 0 || hi > DG_BC_CONDUCTING_WALL) { set_err("unknown boundary type"); return DG_ERR_INVALID; }
        // Simulation::new (grid.rs:55-63) pairs periodic faces
        if (!valid_bc_pair(lo, hi)) { set_err("periodic faces must come in pairs"); return DG_ERR_INVALID; }
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || info->device < 0 || info->device >= ndev) {
        set_err("no CUDA device with that ordinal");
        return DG_ERR_NO_DEVICE;
    }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, info->device) != cudaSuccess || prop.major != 10) {
        set_err("the kernels are built for sm_100a (B200)");
        return DG_ERR_NO_DEVICE;
    }
    dg_ctx *c = new (std::nothrow) dg_ctx();
    if (!c) { set_err("out of host memory"); return DG_ERR_INVALID; }
    c->info = *info;
    c->elem = info->precision == DG_F64 ? 8 : 4;
    c->exact = info->rounding == DG_ROUNDING_REFERENCE || (c->elem == 8 && info->rounding == DG_ROUNDING_DEFAULT);
    c->kind = c->elem == 8 ? (c->exact ? kRefF64 : kFastF64) : (c->exact ? kRefF32 : kFastF32);
    c->nx = info->nx + 4;
    c->ny = info->ny + 4;
    c->nz = info->nz + 4;
    c->pitch = (c->nz + 31) / 32 * 32;
    c->chunk_auto = choose_chunk(c->nx, c->ny, c->nz, c->kind);
    // Test hook: a context created while DG_DEBUG_WAIT_BUDGET is set gives
    // its step kernels' waits for staged planes that many SM clocks (0 or
    // less: every such wait gives up at once, without waiting) instead of
    // ~2 s, so that a test can make the waits run out and check that the
    // step reports DG_ERR_TIMEOUT and the device stays usable.
    if (const char *wb = std::getenv("DG_DEBUG_WAIT_BUDGET")) {
        const long long v = std::atoll(wb);
        c->wait_budget = v > 0 ? v : -1;
    }
    c->fstride = (long long)c->nx * c->ny * c->pitch;
    c->state_bytes = (size_t)5 * c->fstride * c->elem;
    auto bail = [&](int code) {
        set_err(c->err);
        dg_destroy(c);
        return code;
    };
    if (cudaSetDevice(info->device) != cudaSuccess) { c->err = "cudaSetDevice failed"; return bail(DG_ERR_CUDA); }
    cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = cudaMalloc(&c->buf[i], c->state_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&c->ctl, sizeof(DevCtl));
    if (e == cudaSuccess) e = cudaMalloc(&c->part, kReduceBlocks * sizeof(Partial));
    if (e != cudaSuccess) { c->err = std::string("device allocation: ") + cudaGetErrorString(e); return bail(DG_ERR_CUDA); }
    for (int i = 0; i < 2; ++i)
        if (encode_map(c, i) != DG_OK) return bail(DG_ERR_CUDA);
    if (cudaMemsetAsync(c->ctl, 0, sizeof(DevCtl), c->stream) != cudaSuccess ||
        cudaMemsetAsync(c->buf[0], 0, c->state_bytes, c->stream) != cudaSuccess ||
        cudaMemsetAsync(c->buf[1], 0, c->state_bytes, c->stream) != cudaSuccess ||
        cudaStreamSynchronize(c->stream) != cudaSuccess) {
        c->err = "initial memset failed";
        return bail(DG_ERR_CUDA);
    }
    *out = c;
    return DG_OK;
}

int32_t dg_destroy(dg_ctx *c) {
    if (!c) return DG_OK;
    cudaSetDevice(c->info.device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    for (int i = 0; i < 2; ++i)
        if (c->buf[i]) cudaFree(c->buf[i]);
    if (c->ctl) cudaFree(c->ctl);
    if (c->part) cudaFree(c->part);
    if (c->prim_scratch) cudaFree(c->prim_scratch);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return DG_OK;
}

// A state from host fields: the dense upload into the other state buffer,
// then the set-up kernel from there.
static int set_from_host(dg_ctx *c, const void *const src[5], bool prims) {
    if (null_field(src)) return fail(c, DG_ERR_INVALID, "null field pointer");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if ((r = reset_ctl(c)) != DG_OK) return r;
    void *stage = c->buf[1 - c->cur];
    if ((r = upload_dense(c, stage, src)) != DG_OK) return r;
    if ((r = finish_state(c, consecutive(c, stage).f, prims)) != DG_OK) return r;
    return check_flags(c);
}

int32_t dg_set_conserved(dg_ctx *c, const void *const cons[5]) {
    if (!c || !cons) return fail(c, DG_ERR_INVALID, "null argument");
    return set_from_host(c, cons, false);
}

int32_t dg_set_conserved_device(dg_ctx *c, const void *const cons[5]) {
    if (!c || !cons) return fail(c, DG_ERR_INVALID, "null argument");
    if (null_field(cons)) return fail(c, DG_ERR_INVALID, "null field pointer");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if ((r = reset_ctl(c)) != DG_OK) return r;
    void *src[5];
    for (int f = 0; f < 5; ++f) src[f] = const_cast<void *>(cons[f]);
    if (kernel_fields(c, cons)) {
        if ((r = finish_state(c, src)) != DG_OK) return r;
    } else {
        if ((r = copy_fields(c, src, true)) != DG_OK) return r;
        if ((r = finish_state(c)) != DG_OK) return r;
    }
    return check_flags(c);
}

int32_t dg_set_primitives(dg_ctx *c, const void *const prim[5]) {
    if (!c || !prim) return fail(c, DG_ERR_INVALID, "null argument");
    return set_from_host(c, prim, true);
}

int32_t dg_enqueue_steps(dg_ctx *c, int32_t nsteps) {
    if (!c || nsteps < 0) return fail(c, DG_ERR_INVALID, "bad argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    return enqueue(c, nsteps);
}

int32_t dg_get_dts(dg_ctx *c, int32_t nsteps, double *dts) {
    if (!c || !dts || nsteps < 0) return fail(c, DG_ERR_INVALID, "bad argument");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if ((r = read_dts(c, nsteps, dts)) != DG_OK) return r;
    return check_flags(c);
}

int32_t dg_synchronize(dg_ctx *c) {
    if (!c) return DG_ERR_INVALID;
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_flags(c);
}

int32_t dg_compute_step(dg_ctx *c, int32_t nsteps, double *dts) {
    if (!c || nsteps < 0) return fail(c, DG_ERR_INVALID, "bad argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    int done = 0;
    while (done < nsteps) {
        const int n = std::min(nsteps - done, kHist);
        if ((r = enqueue(c, n)) != DG_OK) return r;
        if (dts) {
            if ((r = read_dts(c, n, dts + done)) != DG_OK) return r;
        }
        done += n;
    }
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_flags(c);
}

int32_t dg_next_dt(dg_ctx *c, double *dt) {
    if (!c || !dt) return fail(c, DG_ERR_INVALID, "null argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    DG_CUDA(c, cudaMemcpyAsync(dt, &c->ctl->dt[c->steps & 1], sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_flags(c);
}

int32_t dg_compute_step_dt(dg_ctx *c, double dt) {
    if (!c) return fail(c, DG_ERR_INVALID, "null argument");
    if (!(dt > 0.0) || !std::isfinite(dt)) return fail(c, DG_ERR_INVALID, "dt must be positive and finite");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    set_next_dt_kernel<<<1, 1, 0, c->stream>>>(c->ctl, dt);
    DG_CUDA(c, cudaGetLastError());
    if ((r = enqueue(c, 1)) != DG_OK) return r;
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_flags(c);
}

int32_t dg_get_conserved(dg_ctx *c, void *const cons[5]) {
    if (!c || !cons) return fail(c, DG_ERR_INVALID, "null argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    if (null_field(cons)) return fail(c, DG_ERR_INVALID, "null field pointer");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if (!c->prim_scratch) DG_CUDA(c, cudaMalloc(&c->prim_scratch, c->state_bytes));
    if ((r = get_state(c, consecutive(c, c->prim_scratch).f)) != DG_OK) return r;
    if ((r = download_dense(c, cons, c->prim_scratch)) != DG_OK) return r;
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return DG_OK;
}

int32_t dg_get_conserved_device(dg_ctx *c, void *const cons[5]) {
    if (!c || !cons) return fail(c, DG_ERR_INVALID, "null argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    if (null_field(cons)) return fail(c, DG_ERR_INVALID, "null field pointer");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if ((r = kernel_fields(c, cons) ? get_state(c, cons) : copy_fields(c, cons, false)) != DG_OK) return r;
    // the destination belongs to the caller's streams: return after the copies
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return DG_OK;
}

int32_t dg_get_primitives(dg_ctx *c, void *const prim[5]) {
    if (!c || !prim) return fail(c, DG_ERR_INVALID, "null argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    if (null_field(prim)) return fail(c, DG_ERR_INVALID, "null field pointer");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    if (!c->prim_scratch) DG_CUDA(c, cudaMalloc(&c->prim_scratch, c->state_bytes));
    // the state at the start of the last step is the other buffer; the
    // primitives are written densely for contiguous host copies
    const void *src = c->steps > 0 ? c->buf[1 - c->cur] : c->buf[c->cur];
    const long long dfs = (long long)c->nx * c->ny * c->nz;
    cudaError_t e;
    if (c->elem == 8) {
        auto a = grid_args<double>(c, src, nullptr);
        e = launch_cons_to_prim_policy<double, true>(a, static_cast<const double *>(src),
                                                     static_cast<double *>(c->prim_scratch), dfs, c->nz, c->stream);
    } else {
        auto a = grid_args<float>(c, src, nullptr);
        auto *dstp = static_cast<float *>(c->prim_scratch);
        e = c->exact ? launch_cons_to_prim_policy<float, true>(a, static_cast<const float *>(src), dstp, dfs, c->nz,
                                                               c->stream)
                     : launch_cons_to_prim_policy<float, false>(a, static_cast<const float *>(src), dstp, dfs, c->nz,
                                                                c->stream);
    }
    if (e != cudaSuccess) return cuda_fail(c, e, "cons_to_prim");
    if ((r = download_dense(c, prim, c->prim_scratch)) != DG_OK) return r;
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return DG_OK;
}

int32_t dg_conservation_sums(dg_ctx *c, double out[5]) {
    if (!c || !out) return fail(c, DG_ERR_INVALID, "null argument");
    if (!c->has_state) return fail(c, DG_ERR_NO_STATE, "no state set");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    // FP64 sums of the current state, reduced on the device in a fixed order
    const cudaError_t e = c->elem == 8 ? launch_sums(grid_args<double>(c, c->buf[c->cur], nullptr), c->stream)
                                       : launch_sums(grid_args<float>(c, c->buf[c->cur], nullptr), c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "sum reduction");
    DG_CUDA(c, cudaMemcpyAsync(out, c->ctl->sums, 5 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    return DG_OK;
}

int32_t dg_get_stream(dg_ctx *c, void **stream) {
    if (!c || !stream) return fail(c, DG_ERR_INVALID, "null argument");
    *stream = (void *)c->stream;
    return DG_OK;
}

int32_t dg_step_launch_shape(dg_ctx *c, int32_t *blocks, int32_t *threads, int32_t *chunk) {
    if (!c) return DG_ERR_INVALID;
    const int ch = auto_chunk(c);
    const int b = step_grid_blocks(c->nx, c->ny, c->nz, c->kind, ch);
    if (blocks) *blocks = b;
    if (threads) *threads = step_threads(c->kind);
    if (chunk) *chunk = ch;
    return DG_OK;
}

int32_t dg_set_chunk(dg_ctx *c, int32_t chunk) {
    if (!c || chunk < 0) return fail(c, DG_ERR_INVALID, "bad argument");
    c->chunk = chunk;
    return DG_OK;
}

int32_t dg_status(dg_ctx *c, uint32_t *flags) {
    if (!c || !flags) return fail(c, DG_ERR_INVALID, "null argument");
    int r;
    if ((r = use_device(c)) != DG_OK) return r;
    unsigned f = 0;
    DG_CUDA(c, cudaMemcpyAsync(&f, &c->ctl->flags, sizeof(f), cudaMemcpyDeviceToHost, c->stream));
    DG_CUDA(c, cudaStreamSynchronize(c->stream));
    *flags = f;
    return DG_OK;
}

const char *dg_last_error(const dg_ctx *c) {
    return c ? c->err.c_str() : g_create_err.c_str();
}

}  // extern "C"
