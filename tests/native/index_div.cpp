// div_by(n, d, div_magic(d)) against n / d: around every multiple of d below `top` at most `most` of them, and at the range's end.
#include "../../aspen_b200/csrc/index_div.h"

#include <cstdio>
#include <initializer_list>

static bool same(unsigned n, unsigned d) {
    if (div_by(n, d, div_magic(d)) == n / d) return true;
    printf("%u / %u: %u, not %u\n", n, d, div_by(n, d, div_magic(d)), n / d);
    return false;
}

int main() {
    const unsigned divisors[] = {1, 2, 3, 5, 7, 24, 64, 147, 512, 65535, 65536, 65537, 150528, 200704, 300000, 602112, 1u << 24, 2147483647u};
    for (unsigned d : divisors) {
        const unsigned last = 0xffffffffu - d, steps = last / d < 200000u ? last / d : 200000u;
        for (unsigned i = 0; i <= steps; i++) {
            const unsigned n = d * i, end = last - (last % d) - d * (i < last / d ? i : 0u);
            for (unsigned at : {n, n + 1u, n + d - 1u, end, end ? end - 1u : 0u})
                if (at <= last && !same(at, d)) return 1;
        }
    }
    return 0;
}
