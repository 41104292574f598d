// dg_pointer.h -- which of a caller's pointers the kernels may follow (no CUDA
// needed to compile it; the host checks the rule).
#pragma once
#include <cstddef>
#include <cstdint>

namespace dg {

// What the driver says of a pointer.
struct PointerInfo {
    bool device_memory;        // device memory, not managed, not host memory
    int device;                // the GPU that holds it
    bool foreign_context;      // belongs to another context of that GPU
    uintptr_t start;           // the allocation it lies in
    size_t size;
};

// Whether a kernel on `device` may access `bytes` at p as elements of `elem`
// bytes.  A copy serves more than a kernel's loads and stores: fields on
// another GPU, host memory, addresses off their elements' alignment; and it
// reports a range that ends outside its allocation as an error where a kernel
// would fault.  What fails here is copied.
inline bool kernel_may_access(const PointerInfo &m, uintptr_t p, size_t bytes, size_t elem, int device) {
    return m.device_memory && m.device == device && !m.foreign_context && p % elem == 0 && p >= m.start &&
           bytes <= m.size && p - m.start <= m.size - bytes;
}

}  // namespace dg
