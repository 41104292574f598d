// For lines of `work len blocks`: checks that the blocks' shares (dg_conv_index.h)
// take every step of every column once, and prints the most steps that a block
// takes, the starts of its pieces included.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "dg_conv_index.h"

int main() {
    long long work;
    int len, blocks;
    while (std::scanf("%lld %d %d", &work, &len, &blocks) == 3) {
        std::vector<unsigned char> seen((size_t)work, 0);
        long long most = 0;
        bool once = true;
        for (int b = 0; b < blocks; ++b) {
            dg::net::Share s(work, len, b, blocks);
            long long col, mine = 0;
            int first, count;
            while (s.next(col, first, count)) {
                if (count < 1 || first < 0 || first + count > len || col < 0 || (col + 1) * len > work) return 1;
                for (int i = 0; i < count; ++i) once &= seen[(size_t)(col * len + first + i)]++ == 0;
                mine += count + dg::net::kStartSteps;
            }
            most = std::max(most, mine);
        }
        for (unsigned char c : seen) once &= c == 1;
        std::printf("%d %lld\n", (int)once, most);
    }
}
