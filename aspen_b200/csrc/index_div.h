// Division of an index by a number that is fixed for a layer, as a multiplication and a shift.
#pragma once

#ifdef __CUDACC__
#define INDEX_DIV_FN __host__ __device__ __forceinline__
#else
#define INDEX_DIV_FN inline
#endif

struct Divisor {
    unsigned magic, shift;      // magic 0: the divisor is 1
};

// With 2^shift < d <= 2^(shift + 1) and magic = ceil(2^(32 + shift) / d), which fits 32 bits, n * magic / 2^(32 + shift) exceeds
// n / d by less than n / 2^(32 + shift): the quotient is exact while n * d < 2^(32 + shift), that is for every n < 2^31.
inline Divisor make_divisor(unsigned d) {
    Divisor v = {0u, 0u};
    if (d <= 1u) return v;
    while ((d - 1u) >> (v.shift + 1u)) v.shift++;
    v.magic = (unsigned)(((1ull << (32u + v.shift)) + d - 1u) / d);
    return v;
}

// n / d for d >= 2 (and n < 2^31)
INDEX_DIV_FN unsigned div_by_2_up(unsigned n, Divisor v) {
#ifdef __CUDA_ARCH__
    return __umulhi(n, v.magic) >> v.shift;
#else
    return (unsigned)(((unsigned long long)n * v.magic) >> 32) >> v.shift;
#endif
}
INDEX_DIV_FN unsigned div_by(unsigned n, Divisor v) { return v.magic ? div_by_2_up(n, v) : n; }
