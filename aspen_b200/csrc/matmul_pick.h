// The choice of aspen_b200_matmul_noalloc's kernel, by the shape alone.
#pragma once

// What runs a layer of more than 8 columns, by the longest SM: blocks are dealt whole, so an SM runs ceil(blocks / SMs) of them.
// Measured, us: FMA blocks 3 and their multiply-adds at 131000 a us (32 x 32: 105000; rows that admit only 8- or 4-byte copies take
// 1.2 or 1.5 times as long), the tensor cores with split operands 16 and per 32 of k 0.16 and 0.69 a block of 64 rows, 0.2 and 0.93
// of 128.  k = 3072, 4096 columns, m = 3072: 1698 us in FMA blocks, 733 and 510 split; 64 columns: 61 and 82.
// `split` false: FMA blocks only (so many calls run at once that there is no number for this one: call_slots.h).
// Splitting is for k >= 256: its error against 64 bits grows with what the accumulator of a 32-deep chunk cuts off, not with k, so that of
// short sums would be larger than before.  2-norm, N(0, 1) operands, k = 258 / 512 / 770 / 3072: FMA blocks 1.5e-7 / 2.1e-7 / 1.9e-7 /
// 5.0e-7, split 0.9e-7 / 1.0e-7 / 1.2e-7 / 1.9e-7.
enum MatmulKernel { FMA_128x64, FMA_64x64, FMA_32x32, SPLIT_128, SPLIT_64 };
inline MatmulKernel pick_matmul(unsigned n_cols, unsigned k, unsigned m, unsigned sms, int vec, bool split = true) {
    auto rounds = [&](unsigned bm, unsigned bn) { return (double)(((unsigned long long)((m + bm - 1) / bm) * ((n_cols + bn - 1) / bn) + sms - 1) / sms); };
    const double copies = vec == 4 ? 1.0 : vec == 2 ? 1.2 : 1.5, chunks = (k + 31) / 32;
    const double cost[] = {3 + rounds(128, 64) * 8192.0 * k / 131000 * copies, 3 + rounds(64, 64) * 4096.0 * k / 131000 * copies,
                           3 + rounds(32, 32) * 1024.0 * k / 105000 * copies, 16 + chunks * (0.2 + 0.93 * rounds(128, 128)), 16 + chunks * (0.16 + 0.69 * rounds(64, 128))};
    unsigned best = 0;
    for (unsigned i = 1; i < (k < 256 || !split ? 3u : 5u); i++) if (cost[i] < cost[best]) best = i;
    return (MatmulKernel)best;
}
