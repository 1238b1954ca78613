// div_by(n, make_divisor(d)) against n / d: around multiples of d from both ends of the range n < 2^31.
#include "../../aspen_b200/csrc/index_div.h"

#include <algorithm>
#include <cstdio>
#include <initializer_list>

int main() {
    const unsigned top = 1u << 31, divisors[] = {1, 2, 3, 5, 7, 24, 64, 147, 512, 65535, 65536, 65537, 150528, 200704, 300000, 602112, 1u << 24, 2147483647u};
    for (unsigned d : divisors) {
        const Divisor v = make_divisor(d);
        const unsigned multiples = (top - 1u) / d;
        for (unsigned i = 0; i < std::min(multiples + 1u, 200000u); i++)
            for (unsigned at : {i * d, (multiples - i) * d})
                for (unsigned n : {at - 1u, at, at + 1u}) {
                    if (n >= top) continue;
                    if (div_by(n, v) != n / d || (d > 1u && div_by_2_up(n, v) != n / d)) { printf("%u / %u: %u, not %u\n", n, d, div_by(n, v), n / d); return 1; }
                }
    }
    return 0;
}
