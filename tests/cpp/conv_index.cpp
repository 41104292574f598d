// Prints PlaneIndex's element of plane k (dg_conv_index.h) for lines of
// b x0 y z nx ny nz channels c0 k.
#include <cstdio>

#include "dg_conv_index.h"

int main() {
    int v[10];
    for (;;) {
        for (int &x : v)
            if (std::scanf("%d", &x) != 1) return 0;
        const dg::net::PlaneIndex p(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]);
        std::printf("%lld\n", p.plane(v[9]));
    }
}
