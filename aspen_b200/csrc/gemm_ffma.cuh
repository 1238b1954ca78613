// fp32 contraction blocks on the CUDA cores: D[m][n] = sum_k W[m][k] * X[n][k] with fp32 FMA, by 256 threads of a CTA.
// Used by the allocation-free matmul (noalloc.cu) and by the fp32 mode's contraction tiles (tiles_simt.cuh).
//
// A block is BM x BN outputs; the 256 threads form KS groups that each take one 32-deep slice of a step's KS * 32 values of
// k, and a group's threads each own TM x TN outputs in registers:
//     128 x 64, 8 x 4, KS = 1     the throughput shape
//      64 x 64, 8 x 4, KS = 2     half the work per block, for layers that would leave SMs idle
//      32 x 32, 4 x 4, KS = 4     smaller still; KS keeps eight warps busy on a block of 1024 outputs
// Operands are staged as they lie in memory (k contiguous) by cp.async, STAGES deep, so neither registers nor a transposing
// store stand between global memory and the FMAs; a row's 16-byte piece c sits at c ^ (row / 4 % 8): eight lanes that own
// four rows each read without bank conflicts.  Two FMAs are one packed fma.rn.f32x2 (sm_100) over a pair of k, each half
// rounded like fmaf; the two partial sums of an output are added at the end.  With scalar FMAs alone every issue slot
// would be taken and the shared-memory reads would come on top.  B200, 4096 x 3072 outputs, k = 3072: 44 TFLOP/s for the
// first two shapes, 40 for the third (FMA pipe active 65 %, shared-memory wavefronts 74 % of their peak).
#pragma once
#include "device_types.h"

namespace fmablk {

constexpr unsigned THREADS = 256;

__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    return x + y;
}
// BYTES-wide asynchronous copy; `ok` false writes zeros.
template <int BYTES>
__device__ __forceinline__ void copy_async(unsigned dst, const void *src, bool ok) {
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16u : 0u) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(ok ? (unsigned)BYTES : 0u) : "memory");
}

template <int BM_, int BN_, int TM_, int TN_, int KS_, int STAGES_ = 3>
struct Shape {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, KS = KS_, STAGES = STAGES_;
    static constexpr int KT = KS * 32;                                // k values per step
    static constexpr int STAGE_BYTES = (BM + BN) * 128 * KS;          // [slice][W rows, X rows][32 k]
    static constexpr int RED_BYTES = KS > 1 ? KS * BN * (BM + 4) * 4 : 0;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES > RED_BYTES ? STAGES * STAGE_BYTES : RED_BYTES;
    static constexpr int GROUP = (BM / TM) * (BN / TN);               // threads of a group
    static_assert(GROUP * KS == (int)THREADS, "256 threads");
    static constexpr int RW = BM / 32, RX = BN / 32;                  // rows a thread stages per slice: (tid / 8) + 32 i
};
typedef Shape<128, 64, 8, 4, 1> Large;
typedef Shape<64, 64, 8, 4, 2> Medium;
typedef Shape<32, 32, 4, 4, 4> Small;
typedef Shape<64, 32, 4, 2, 1, 2> Tight;      // 24 KB of staging, beside the tensor-core ring

// Loader (one per operand):  void row(int i, unsigned r): row r of the block is this thread's i-th row;
//     void at(unsigned k): the pieces that follow start at k;  void copy(unsigned dst, int i): stage 4 values of row i.
// The sums run over k0 (a multiple of 4) .. K - 1; the loaders give zeros from K on.
// Bar: barrier of the 256 threads.  Out: void operator()(unsigned m, unsigned n, const float *v): outputs m .. m+3 of column n.
template <typename S, typename LoadW, typename LoadX, typename Bar, typename Out>
__device__ __forceinline__ void block(unsigned char *smem, unsigned tid, unsigned K, LoadW &loadw, LoadX &loadx, Bar bar, Out &out, unsigned k0 = 0) {
    const unsigned group = tid / S::GROUP, gt = tid % S::GROUP;
    // lane bits 0, 3, 4 pick one of 8 groups of 4 output rows, bits 1, 2 one of 4 groups of columns: a quarter warp reads four
    // W rows and two or four X rows at a time (2 % faster than eight and one)
    const unsigned lane = gt & 31u, quad = gt >> 5;
    const unsigned ty = ((lane & 1u) | ((lane >> 2) & 6u)) + 8u * (quad % (S::BM / S::TM / 8)), tx = ((lane >> 1) & 3u) + 4u * (quad / (S::BM / S::TM / 8));
    const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
    const unsigned srow = tid >> 3, piece = tid & 7u, steps = (K - k0 + S::KT - 1) / S::KT;

    #pragma unroll
    for (int i = 0; i < S::RW; i++) loadw.row(i, srow + 32u * i);
    #pragma unroll
    for (int i = 0; i < S::RX; i++) loadx.row(i, srow + 32u * i);
    auto stage = [&](unsigned step) {
        if (step < steps) {
            #pragma unroll
            for (int s = 0; s < S::KS; s++) {
                const unsigned slice = base + (step % S::STAGES) * S::STAGE_BYTES + s * (S::BM + S::BN) * 128;
                const unsigned k = k0 + step * S::KT + s * 32u + piece * 4u;
                loadw.at(k);
                #pragma unroll
                for (int i = 0; i < S::RW; i++) {
                    const unsigned r = srow + 32u * i;
                    loadw.copy(slice + r * 128u + ((piece ^ ((r >> 2) & 7u)) << 4), i);
                }
                loadx.at(k);
                #pragma unroll
                for (int i = 0; i < S::RX; i++) {
                    const unsigned r = srow + 32u * i;
                    loadx.copy(slice + S::BM * 128u + r * 128u + ((piece ^ ((r >> 2) & 7u)) << 4), i);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    unsigned long long acc[S::TM][S::TN];
    #pragma unroll
    for (int i = 0; i < S::TM; i++)
        #pragma unroll
        for (int j = 0; j < S::TN; j++) acc[i][j] = 0ull;
    #pragma unroll
    for (int s = 0; s < S::STAGES - 1; s++) stage(s);
    for (unsigned step = 0; step < steps; step++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::STAGES - 2) : "memory");
        bar();                                        // everybody's copies of this step have landed, the oldest stage is free
        stage(step + S::STAGES - 1);
        const unsigned char *w = smem + (step % S::STAGES) * S::STAGE_BYTES + group * (S::BM + S::BN) * 128 + ty * 512;
        const unsigned char *x = smem + (step % S::STAGES) * S::STAGE_BYTES + group * (S::BM + S::BN) * 128 + S::BM * 128 + tx * (S::TN * 128);
        #pragma unroll
        for (unsigned c = 0; c < 8; c++) {            // 4 values of k at a time
            ulonglong2 b[S::TN];
            #pragma unroll
            for (int j = 0; j < S::TN; j++) b[j] = *reinterpret_cast<const ulonglong2 *>(x + j * 128 + ((c ^ ((tx * S::TN / 4u) & 7u)) << 4));
            #pragma unroll
            for (int i = 0; i < S::TM; i++) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(w + (i / 4) * (S::BM * 64) + (i % 4) * 128 + ((c ^ (ty & 7u)) << 4));
                #pragma unroll
                for (int j = 0; j < S::TN; j++) { fma2(acc[i][j], a.x, b[j].x); fma2(acc[i][j], a.y, b[j].y); }
            }
        }
    }
    if (S::KS == 1) {
        #pragma unroll
        for (int j = 0; j < S::TN; j++)
            #pragma unroll
            for (int i = 0; i < S::TM; i += 4) {
                const float v[4] = {pair_sum(acc[i][j]), pair_sum(acc[i + 1][j]), pair_sum(acc[i + 2][j]), pair_sum(acc[i + 3][j])};
                out(4u * ty + (i / 4) * (S::BM / 2), S::TN * tx + j, v);
            }
        bar();
    } else {
        // the groups' partial sums meet in shared memory; then every thread finishes whole 16-byte pieces, rows first
        float *red = reinterpret_cast<float *>(smem);
        constexpr int P = S::BM + 4;
        bar();
        #pragma unroll
        for (int j = 0; j < S::TN; j++)
            #pragma unroll
            for (int i = 0; i < S::TM; i += 4)
                *reinterpret_cast<float4 *>(red + (group * S::BN + S::TN * tx + j) * P + 4u * ty + (i / 4) * (S::BM / 2)) =
                    make_float4(pair_sum(acc[i][j]), pair_sum(acc[i + 1][j]), pair_sum(acc[i + 2][j]), pair_sum(acc[i + 3][j]));
        bar();
        #pragma unroll
        for (unsigned p = tid; p < S::BM * S::BN / 4; p += THREADS) {
            const unsigned m = 4u * (p % (S::BM / 4)), n = p / (S::BM / 4);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            #pragma unroll
            for (int g = 0; g < S::KS; g++) {
                const float4 t = *reinterpret_cast<const float4 *>(red + (g * S::BN + n) * P + m);
                v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
            }
            out(m, n, v);
        }
        bar();                                        // the staging may be written again
    }
}

}  // namespace fmablk
