// Prints the block count and the answer of dg_noalloc_limit.h for lines of
// nx ny nz f64 fused.
#include <cstdio>

#include "dg_noalloc_limit.h"

int main() {
    int nx, ny, nz, f64, fused;
    while (std::scanf("%d %d %d %d %d", &nx, &ny, &nz, &f64, &fused) == 5)
        std::printf("%lld %d\n", dg::noalloc::limit_blocks(nx, ny, nz, f64 != 0, fused != 0),
                    (int)dg::noalloc::accepted(nx, ny, nz, f64 != 0, fused != 0));
}
