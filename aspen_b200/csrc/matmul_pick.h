// The choice of aspen_b200_matmul_noalloc's kernel, by the shape alone.
#pragma once

// What runs a layer of more than 8 columns.  Blocks are dealt whole, so an SM runs at most ceil(blocks / SMs) of them.
//
// FMA blocks: the shape with the shortest longest SM, a block's multiply-adds at its share of the FMA rate.  Of 292 shapes with k < 256 (9 - 4096
// columns, m 64 - 3072, k % 4, k % 2 and odd in turn) that is 0.9 % behind the fastest on average, 28 % at worst; by the estimate below 0.4 and 10 %, but
// then blocks with fewer partial sums, and so larger errors, run shapes that had better ones.
// Split operands (gemm_split.cuh) where the estimate is below that of these FMA blocks, for k >= 256: the error of splitting is mostly what the
// accumulator of a 32-deep chunk cuts off, whatever k is, so that of short sums would be larger than before.  The estimate is fitted to each kernel's
// times over 420 shapes: launch and wait, for each block of the longest SM a part for its start and end and one for k, and a share of k that comes once;
// loads of 8 and of 4 bytes take `pairs` and `singles` times as long.  It is off by 2 to 5 % (root mean square).  Over the 128 shapes with k >= 256
// what is picked takes 0.04 % longer than the fastest on average, 3 % at worst.  On either side of the line, columns x k x m: 64 x 3072 x 3072 60 us
// in FMA blocks of 32 x 32 and 81 split by 64; 333 x 770 x 1000 44 and 38; 963 x 392 x 836 39 and 25; 1024 x 768 x 2048 split by 64 54 and by 128
// 42; 4096 x 3072 x 3072 1696 in FMA blocks of 64 x 64 and 531 split by 128.
// `split` false: FMA blocks only (so many calls run at once that there is no number for this one: call_slots.h).
enum MatmulKernel { FMA_128x64, FMA_64x64, FMA_32x32, SPLIT_128, SPLIT_64 };
inline MatmulKernel pick_matmul(unsigned n_cols, unsigned k, unsigned m, unsigned sms, int vec, bool split = true) {
    // rows and columns of a block; `rate`: of FMAs; us; `step`: the k that `per_step` and `once` count
    static const struct { unsigned bm, bn; float rate; double call, block, per_step, once, pairs, singles; unsigned step; } kernels[] = {
        {128, 64, 0.80f, 14.9, 2.01, 0.0527, 0.0054, 1.08, 1.36, 1}, {64, 64, 0.80f, 13.2, 1.88, 0.0264, 0.0032, 1.08, 1.30, 1},
        {32, 32, 0.65f, 12.3, 0.95, 0.0077, 0.0015, 1.16, 1.58, 1}, {128, 128, 0, 13.3, 5.06, 0.778, 0.0117, 1.05, 1.16, 32},
        {64, 128, 0, 13.7, 2.40, 0.628, 0.0087, 1.04, 1.12, 32}};
    auto rounds = [&](unsigned i) {
        return ((unsigned long long)((m + kernels[i].bm - 1) / kernels[i].bm) * ((n_cols + kernels[i].bn - 1) / kernels[i].bn) + sms - 1) / sms;
    };
    auto us = [&](unsigned i) {
        const auto &q = kernels[i];
        const double steps = (k + q.step - 1) / q.step;
        return q.call + (double)rounds(i) * (q.block + q.per_step * steps) * (vec == 4 ? 1.0 : vec == 2 ? q.pairs : q.singles) + q.once * steps;
    };
    unsigned best = 0;
    float shortest = 0;
    for (unsigned i = 0; i < 3; i++) {
        const float work = (float)rounds(i) * (float)(kernels[i].bm * kernels[i].bn) / kernels[i].rate;
        if (i == 0 || work < shortest) { best = i; shortest = work; }
    }
    for (unsigned i = 3; i < 5 && split && k >= 256; i++) if (us(i) < us(best)) best = i;
    return (MatmulKernel)best;
}
