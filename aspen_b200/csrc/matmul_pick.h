// The choice of aspen_b200_matmul_noalloc's kernel, by the shape alone.
#pragma once

// What runs a layer of more than 8 columns, by the longest SM: blocks are dealt whole, so an SM runs ceil(blocks / SMs) of them.  us of a call, fitted
// to each kernel's times over 330 shapes (9 - 4096 columns, k and m 64 - 3072, k % 4 and k % 2 in turn): launch and wait, and for every
// block of an SM a part for its start and end and one for k.  The fit is off by 5 % (root mean square); where blocks of two sizes take as long, the smaller
// FMA ones are preferred (1.3 and 2.5 us), because they have more partial sums and so the smaller error.  Over the 330 shapes what is picked takes 0.13 %
// longer than the fastest on average, 12 % at worst (1558 columns, k = 150, m = 780: 37 us in 32 x 32 blocks, 33 in 64 x 64).
// On either side of the lines, columns x k x m: 64 x 3072 x 3072 60 us in FMA blocks of 32 x 32 and 81 split by 64; 333 x 770 x 1000 40 and 36;
// 963 x 392 x 836 39 and 25; 1024 x 768 x 2048 split by 64 54 and by 128 42; 4096 x 3072 x 3072 1696 in FMA blocks of 64 x 64 and 522 split by 128.
// `split` false: FMA blocks only (so many calls run at once that there is no number for this one: call_slots.h).
// Splitting is for k >= 256: its error against 64 bits is mostly what the accumulator of a 32-deep chunk cuts off, whatever k is, so that of
// short sums would be larger than before.  Both errors: gemm_split.cuh.
enum MatmulKernel { FMA_128x64, FMA_64x64, FMA_32x32, SPLIT_128, SPLIT_64 };
inline MatmulKernel pick_matmul(unsigned n_cols, unsigned k, unsigned m, unsigned sms, int vec, bool split = true) {
    auto rounds = [&](unsigned bm, unsigned bn) { return (double)(((unsigned long long)((m + bm - 1) / bm) * ((n_cols + bn - 1) / bn) + sms - 1) / sms); };
    const double copies = vec == 4 ? 1.0 : vec == 2 ? 1.2 : 1.5, loads = vec == 4 ? 1.0 : vec == 2 ? 1.03 : 1.06, chunks = (k + 31) / 32;
    const double cost[] = {19 + rounds(128, 64) * (1.4 + 0.0566 * k * copies), 15.5 + rounds(64, 64) * (1.4 + 0.0284 * k * copies),
                           13 + rounds(32, 32) * (0.75 + 0.0081 * k * copies), 13.5 + rounds(128, 128) * (7 + 0.87 * chunks * loads), 14 + rounds(64, 128) * (3.3 + 0.675 * chunks * loads)};
    unsigned best = 0;
    for (unsigned i = 1; i < (k < 256 || !split ? 3u : 5u); i++) if (cost[i] < cost[best]) best = i;
    return (MatmulKernel)best;
}
