// Prints kernel_may_access (dg_pointer.h) for lines of
// device_memory device foreign start size p bytes elem ctx_device.
#include <cstdio>

#include "dg_pointer.h"

int main() {
    unsigned long long start, size, p, bytes, elem;
    int mem, device, foreign, ctx;
    while (std::scanf("%d %d %d %llu %llu %llu %llu %llu %d", &mem, &device, &foreign, &start, &size, &p, &bytes, &elem,
                      &ctx) == 9) {
        const dg::PointerInfo m = {mem != 0, device, foreign != 0, (uintptr_t)start, (size_t)size};
        std::printf("%d\n", (int)dg::kernel_may_access(m, (uintptr_t)p, (size_t)bytes, (size_t)elem, ctx));
    }
}
