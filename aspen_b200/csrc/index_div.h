// Division by a number that is fixed for a whole tile, as one multiplication.
#pragma once

#ifdef __CUDACC__
#define INDEX_DIV_FN __host__ __device__ __forceinline__
#else
#define INDEX_DIV_FN inline
#endif

// ceil(2^32 / d); 0 stands for d = 1
INDEX_DIV_FN unsigned div_magic(unsigned d) { return d == 1u ? 0u : 0xffffffffu / d + 1u; }

// n / d, m = div_magic(d), for every n with n + d < 2^32.  The product's high word is the quotient or, where n times m's rounding
// passes 2^32 (n * d >= 2^32 at the earliest: a connected layer over more than 65536 channels reaches that), one more.
INDEX_DIV_FN unsigned div_by(unsigned n, unsigned d, unsigned m) {
#ifdef __CUDA_ARCH__
    const unsigned q = m ? __umulhi(n, m) : n;
#else
    const unsigned q = m ? (unsigned)(((unsigned long long)n * m) >> 32) : n;
#endif
    return q * d > n ? q - 1u : q;
}
