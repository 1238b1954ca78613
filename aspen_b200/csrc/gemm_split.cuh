// fp32 contraction on the tensor cores: out[n][m] = act(bias[m] + sum_k W[m][k] X[n][k]) with every operand as a sum of three bf16 values.
//
// An fp32 value is x = b1 + b2 + b3 (8 bits each), exactly unless |x| < 2^-110, where b3 may need bits below the last of bf16, 2^-133.  W X is
// nine products of bf16 parts of which the six up to 2^-16 are kept -- the others are below half a unit of the fp32 product.  The tensor cores
// multiply bf16 exactly but truncate when they add to an accumulator: a chunk of k = 32 is summed there, smallest products first; two chunks are
// added to each other and then to the total in registers, with rounding to nearest.  Relative error, 2-norm, against 64 bits (k = 256 / 770 /
// 3072): N(0, 1) operands 0.8 / 1.0 / 1.4e-7, FMA blocks of 64 x 64 1.5 / 2.5 / 5.0, of 32 x 32 1.1 / 1.8 / 3.5; operands of one sign 0.7 / 0.8 /
// 1.1e-7, FMA blocks of 64 x 64 0.7 / 1.0 / 1.9, of 32 x 32 (eight partial sums) 0.5 / 0.6 / 1.0, the one place where they are closer: what
// the accumulators cut off is all of one sign there.  (Chunks added to the total one by one: 0.8 / 1.1 / 1.9 and 0.7 / 0.9 / 1.4.)
//
// A block is computed again by fp32 FMA blocks, so that its outputs are what fp32 sums give,
//     if one of its values has no such sum: infinities, NaN, values with bits below 2^-133, values that round past the range of bf16;
//     if a total is an infinity or a NaN: where a product overflows, those of the parts have either sign and leave inf - inf;
//     if a total is so small that what the accumulators truncate at the lower end of fp32, up to four units of 2^-149 a chunk, is more than 2^-24
//     of it (768 products around 2^-130: 2-norm error 1.3e-6, of fp32 sums 5.5e-7).
// That is done when the CTA is through with all of its blocks, so that nothing waits for it.  4096 x 768 x 3072: 180 us a call, 900 if every block
// is marked.
//
// What bounds it: shared memory.  A chunk of a 128 x 128 block is 12 MMAs that read 8 KB each, and 49 KB of parts written for them:
// 1150 cycles at 128 bytes a cycle, against 770 of the tensor pipe.  Hence
//     warps 4 - 11   read both operands from global memory into registers, split them and store the parts in the 64-byte swizzled K-major
//                    layout (a raw copy in shared memory would cost another 64 KB a chunk)
//     warp 0         12 MMAs a chunk, into four accumulators in turn
//     warps 12 - 19  add two finished accumulators to the totals (each holds 32 columns x N / 2 rows in registers), then bias, activation, stores
// N (128 or 64 rows of W a block) is the caller's choice; with 256 the totals leave too few registers for loads in flight (1.84 us a
// chunk against 2 x 0.93).  Persistent: a CTA takes every gridDim-th block, and the splitting of the next one goes on under the stores.
// 4096 x 3072 outputs, k = 3072: 146 TFLOP/s of fp32 products (FMA blocks: 46).
//
// Every wait is bounded (LIMIT_NS) and is for another role of the CTA; a thread that gives up sets the CTA's `gave_up`, all roles leave, TMEM is
// freed, and the call's word `failed` is set.
#pragma once
#include "tiles_tc.cuh"

namespace split {

constexpr unsigned THREADS = 640, SPLITTERS = 128, CHUNK = 32, ACCUMULATORS = 4, MAX_BLOCKS = 8192;
constexpr unsigned long long LIMIT_NS = 2000000000ull;

template <int N>
struct Shape {
    static constexpr int STAGES = N == 128 ? 3 : 4;      // what is left of the 228 KB holds the loads in flight: 4 stages of N = 128 cost 8 %
    static constexpr int PART_X = 128 * 64, PART_W = N * 64;                 // bytes of one part of a chunk: rows of 32 bf16
    static constexpr int STAGE_BYTES = 3 * (PART_X + PART_W);
    static constexpr int PIECES = (128 + N) / 16;                            // 16-byte loads of a splitting thread per chunk
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 8 * 4096;
};

struct Shared {
    unsigned long long full[4], empty[4];          // stage split / read by the MMAs
    unsigned long long acc_full[ACCUMULATORS], acc_empty[ACCUMULATORS];    // accumulator complete / added to the totals
    unsigned odd[MAX_BLOCKS / 32];                 // a bit for each of the CTA's blocks that is to be computed again
    unsigned gave_up;                              // a wait ran out
    unsigned tmem;
};

__device__ __forceinline__ bool wait(unsigned long long *bar, unsigned parity, unsigned *gave_up) {
    #pragma unroll 1
    for (unsigned spin = 0; spin < 4096u; spin++)
        if (tc::mbar_try_wait(bar, parity)) return true;
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    #pragma unroll 1
    for (unsigned spin = 1;; spin++) {
        if (tc::mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 0u) {
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (*(volatile unsigned *)gave_up != 0u) return false;
            if (now - t0 > LIMIT_NS) { atomicExch(gave_up, 1u); return false; }
        }
    }
}

__device__ __forceinline__ void mma_bf16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// K-major, 64-byte swizzle, 8-row groups 512 bytes apart (version 1 in bits 46-47)
__device__ __forceinline__ unsigned long long desc(unsigned addr) {
    return (unsigned long long)((512u >> 4) | 1u << 14 | 4u << 29) << 32 | (addr >> 4) | 1u << 16;
}

typedef unsigned long long Pair;         // two fp32 values
__device__ __forceinline__ Pair pack(float x, float y) { Pair p; asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(x), "f"(y)); return p; }
__device__ __forceinline__ Pair pack(unsigned x, unsigned y) { Pair p; asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(x), "r"(y)); return p; }
__device__ __forceinline__ void unpack(Pair p, unsigned &x, unsigned &y) { asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(p)); }
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) { Pair d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
// The next bf16 part of two values, x's in the low half; what is left of them stays.  The first part is rounded to nearest, so that the
// rest has either sign; the second is cut off; the third is what is left, eight bits: the lower half of its word is zero unless it would need bits
// below 2^-133, or the value is not finite (or rounds past the range of bf16), which leaves the NaN 0x7fffffff.
template <int PART>
__device__ __forceinline__ unsigned take_part(Pair &v) {
    unsigned x, y;
    unpack(v, x, y);
    if (PART == 0) { x += 0x8000u; y += 0x8000u; }
    if (PART < 2) v = fma2(pack(x & 0xffff0000u, y & 0xffff0000u), pack(-1.f, -1.f), v);
    return __byte_perm(x, y, 0x7632);
}

__device__ __forceinline__ unsigned either(Pair v) { unsigned x, y; unpack(v, x, y); return x | y; }       // bits of one or the other

__device__ __forceinline__ void add2(float &x, float &y, float a, float b) {
    unsigned long long s, t;
    asm("mov.b64 %0, {%1, %2};" : "=l"(s) : "f"(x), "f"(y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "f"(a), "f"(b));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s) : "l"(t));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(s));
}

// Eight columns of each of two accumulators.
__device__ __forceinline__ void tmem_ld8x2(unsigned first, unsigned second, float *v) {
    unsigned *r = reinterpret_cast<unsigned *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
                   "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15])
                 : "r"(first), "r"(second) : "memory");
}

// Every role is through: the operand stages are free, and what it has stored is seen by the others.
__device__ __forceinline__ void all_roles_done() {
    __syncwarp();
    tc::tc_fence_before();
    asm volatile("bar.sync 0;" ::: "memory");
}

// Load: float4 operator()(bool weight, unsigned row, unsigned k): four values of a row of W or X from k on, zeros outside;
//       const float *at(bool weight, unsigned row, unsigned k), unsigned ld(): their address (not read if outside), the distance of two rows;
//       float4 piece(const float *): the four values there.
// Out:  void operator()(unsigned n, unsigned m, const float4 &v): outputs m .. m + 3 of column n, both possibly outside;
//       void late(n, dn, cn, m, cm): the same thread's outputs of columns n, n + dn, ... (cn of them), rows m, m + 32, ... (cm) are stored.
// Again: void operator()(unsigned tid, unsigned n0, unsigned m0): the outputs of a block once more by 256 threads, as fp32 sums give them;
//       the operand stages are its shared memory.  At most MAX_BLOCKS blocks in all.
template <int N, typename Load, typename Out, typename Again>
__device__ __forceinline__ void blocks(unsigned char *smem, Shared *sh, unsigned *failed, unsigned cols, unsigned rows, unsigned K, const Load &load, const Out &out, const Again &again) {
    typedef Shape<N> S;
    const unsigned warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const unsigned row_blocks = (rows + N - 1) / N, total = row_blocks * ((cols + 127u) / 128u), chunks = (K + CHUNK - 1) / CHUNK;
    const unsigned base = tc::smem_u32(smem);
    unsigned *const gave_up = &sh->gave_up;
    if (threadIdx.x == 0) {
        sh->gave_up = 0u;
        for (int s = 0; s < S::STAGES; s++) { tc::mbar_init(&sh->full[s], SPLITTERS); tc::mbar_init(&sh->empty[s], 1u); }
        for (unsigned h = 0; h < ACCUMULATORS; h++) { tc::mbar_init(&sh->acc_full[h], 1u); tc::mbar_init(&sh->acc_empty[h], 8u); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_proxy_async_smem();
    }
    for (unsigned i = threadIdx.x; i < MAX_BLOCKS / 32; i += THREADS) sh->odd[i] = 0u;
    if (warp == 0) tc::tmem_alloc(&sh->tmem, 512u);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    // Registers: 128 x (40 + 2 x 112 + 2 x 104) = 128 x 472 of 640 x 96, what the launch holds.  Each share is set at the head of its roles' own branch:
    // behind a join of the branches the compiler keeps to the smallest one.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0) {
            // The whole warp walks, one lane issues: operands of the MMAs that the compiler knows to be the same in all lanes stay in
            // uniform registers (issued from one lane's own branch, an MMA took some 95 cycles whatever its size).
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((128u >> 4) << 24);      // D fp32, A and B bf16
            const unsigned tmem = __shfl_sync(0xffffffffu, sh->tmem, 0);
            unsigned s = 0, lap = 0, it = 0;
            bool ok = true;
            for (unsigned t = blockIdx.x; t < total && ok; t += gridDim.x)
                for (unsigned c = 0; c < chunks; c++, it++) {
                    const unsigned h = it % ACCUMULATORS, d = tmem + h * N;
                    ok = wait(&sh->acc_empty[h], ((it / ACCUMULATORS) & 1u) ^ 1u, gave_up) && wait(&sh->full[s], lap & 1u, gave_up);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const unsigned x = base + s * S::STAGE_BYTES, w = x + 3 * S::PART_X;
                    if (tc::elect_one()) {
                        // smallest products first: what the accumulator truncates then is small
                        constexpr unsigned char order[6][2] = {{2, 0}, {1, 1}, {0, 2}, {1, 0}, {0, 1}, {0, 0}};
                        #pragma unroll
                        for (int p = 0; p < 6; p++)
                            #pragma unroll
                            for (int j = 0; j < 2; j++)
                                mma_bf16(d, desc(x + order[p][0] * S::PART_X + j * 32u), desc(w + order[p][1] * S::PART_W + j * 32u), idesc, p + j);
                        tc::tc_commit(&sh->empty[s]);
                        tc::tc_commit(&sh->acc_full[h]);
                    }
                    __syncwarp();
                    if (++s == S::STAGES) { s = 0; lap++; }
                }
        }
        all_roles_done();
        if (warp == 0) {
            if (sh->gave_up) {
                // MMAs may still be in flight; they take microseconds
                unsigned long long t0, now;
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
                do { __nanosleep(1000); asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now)); } while (now - t0 < 2000000ull);
                if (lane == 0) *failed = 1u;
            }
            tc::tc_fence_after();
            tc::tmem_dealloc(sh->tmem, 512u);
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        // Two groups of four warps take the chunks in turn: while one splits, the other's loads are on their way.  (One group that asks for
        // a piece's next values as soon as it has split it waits for all its loads at every piece: 1.8 us a chunk of 256 rows.)
        // Thread: rows r0 + 16 i (X, then W), values 4 (lane % 8) .. + 3 of the chunk.
        const unsigned r0 = (warp & 3u) * 4u + (lane >> 3), k0 = (lane & 7u) * 4u, group = (warp >> 2) - 1u;
        constexpr int G = 4;
        float4 v[S::PIECES];
        unsigned left = 0;                            // what the third parts could not take, in the lower halves of the words
        unsigned t = blockIdx.x, c = group, s = group, lap = 0, block = 0;
        const size_t step = 16 * (size_t)load.ld();
        auto fetch = [&]() {
            const unsigned n0 = t / row_blocks * 128u, m0 = t % row_blocks * N, k = c * CHUNK;
            if (k + CHUNK <= K) {
                // at the edge, pieces past the last row read another row's values: their outputs go nowhere
                const unsigned xr = min(n0 + r0, cols - 1u), wr = min(m0 + r0, rows - 1u);
                const float *px = load.at(false, xr, k + k0), *pw = load.at(true, wr, k + k0);
                if (n0 + 128u <= cols && m0 + N <= rows) {
                    #pragma unroll
                    for (int i = 0; i < S::PIECES; i++) v[i] = load.piece(i < 8 ? px + i * step : pw + (i - 8) * step);
                } else {
                    const unsigned last_x = (cols - 1u - xr) / 16u, last_w = (rows - 1u - wr) / 16u;
                    #pragma unroll
                    for (int i = 0; i < S::PIECES; i++) v[i] = load.piece(i < 8 ? px + min((unsigned)i, last_x) * step : pw + min((unsigned)(i - 8), last_w) * step);
                }
            } else {
                #pragma unroll
                for (int i = 0; i < S::PIECES; i++) v[i] = i < 8 ? load(false, n0 + i * 16 + r0, k + k0) : load(true, m0 + (i - 8) * 16 + r0, k + k0);
            }
        };
        // 16-byte quarter of a row's 64 bytes: exclusive or with bits 1-2 of the row (64-byte swizzle); the same for every 16th row
        unsigned char *const first = smem + r0 * 64u + ((((lane & 7u) >> 1) ^ ((r0 >> 1) & 3u)) << 4) + ((lane & 1u) << 3);
        while (t < total) {
            fetch();
            if (!wait(&sh->empty[s], (lap & 1u) ^ 1u, gave_up)) break;
            #pragma unroll
            for (int i0 = 0; i0 < S::PIECES; i0 += G) {
                // G pieces side by side, so that no instruction waits for the one before it
                Pair lo[G], hi[G];
                uint2 part[3][G];
                #pragma unroll
                for (int i = 0; i < G; i++) { lo[i] = pack(v[i0 + i].x, v[i0 + i].y); hi[i] = pack(v[i0 + i].z, v[i0 + i].w); }
                #pragma unroll
                for (int i = 0; i < G; i++) part[0][i] = make_uint2(take_part<0>(lo[i]), take_part<0>(hi[i]));
                #pragma unroll
                for (int i = 0; i < G; i++) part[1][i] = make_uint2(take_part<1>(lo[i]), take_part<1>(hi[i]));
                #pragma unroll
                for (int i = 0; i < G; i++) {
                    part[2][i] = make_uint2(take_part<2>(lo[i]), take_part<2>(hi[i]));
                    left |= either(lo[i]) | either(hi[i]);
                }
                #pragma unroll
                for (int i = 0; i < G; i++) {
                    const int r = (i0 + i) * 16;
                    unsigned char *at = first + s * S::STAGE_BYTES + (r < 128 ? r * 64 : 3 * S::PART_X + (r - 128) * 64);
                    #pragma unroll
                    for (int p = 0; p < 3; p++) *reinterpret_cast<uint2 *>(at + p * (r < 128 ? S::PART_X : S::PART_W)) = part[p][i];
                }
            }
            tc::fence_proxy_async_smem();
            tc::mbar_arrive(&sh->full[s]);
            if ((s += 2u) >= (unsigned)S::STAGES) { s -= S::STAGES; lap++; }
            if ((c += 2u) >= chunks) {
                if (left & 0xffffu) atomicOr(&sh->odd[block / 32u], 1u << (block % 32u));
                left = 0;
                block++;
                c -= chunks;
                t += gridDim.x;
            }
        }
        all_roles_done();
        block = 0;
        for (unsigned t = blockIdx.x; t < total && !sh->gave_up; t += gridDim.x, block++)
            if (sh->odd[block / 32u] >> (block % 32u) & 1u) again(threadIdx.x - 128u, t / row_blocks * 128u, t % row_blocks * N);
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        const unsigned q = warp & 3u, first = (warp - 12u) / 4u * (N / 2);        // TMEM lanes 32 q .. + 31: columns; rows first .. + N / 2 - 1
        float *stage = reinterpret_cast<float *>(smem + S::STAGES * S::STAGE_BYTES + (warp - 12u) * 4096u);
        unsigned it = 0, block = 0;
        bool ok = true;
        for (unsigned t = blockIdx.x; t < total && ok; t += gridDim.x, block++) {
            const unsigned n0 = t / row_blocks * 128u + q * 32u, m0 = t % row_blocks * N + first;
            float sum[N / 2];
            #pragma unroll
            for (int i = 0; i < N / 2; i++) sum[i] = 0.f;
            for (unsigned c = 0; c < chunks; c += 2u) {
                // Two chunks are added to each other first: half as many roundings in the size of the totals.
                const bool two = c + 1u < chunks;
                const unsigned h0 = it % ACCUMULATORS, h1 = two ? (it + 1u) % ACCUMULATORS : h0, from = sh->tmem + first + (q << 21);
                ok = wait(&sh->acc_full[h0], (it / ACCUMULATORS) & 1u, gave_up) && (!two || wait(&sh->acc_full[h1], ((it + 1u) / ACCUMULATORS) & 1u, gave_up));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc::tc_fence_after();
                #pragma unroll
                for (int j = 0; j < N / 2; j += 8) {
                    float v[16];
                    tmem_ld8x2(from + h0 * N + j, from + h1 * N + j, v);
                    if (j + 8 == N / 2) {
                        tc::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) { tc::mbar_arrive(&sh->acc_empty[h0]); if (two) tc::mbar_arrive(&sh->acc_empty[h1]); }
                    }
                    #pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        add2(v[i], v[i + 1], two ? v[8 + i] : 0.f, two ? v[9 + i] : 0.f);
                        add2(sum[j + i], sum[j + i + 1], v[i], v[i + 1]);
                    }
                }
                it += two ? 2u : 1u;
            }
            if (!ok) break;
            // Too small, or not finite (of two magnitudes the larger bits are the larger value).  Outputs past the last row or column hold
            // another one's values or zeros.
            const unsigned least = __float_as_uint((float)chunks * 0x1p-123f);
            unsigned far = 0;
            #pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const unsigned u = __float_as_uint(sum[i]) & 0x7fffffffu;
                far = max(far, u == 0u ? 0u : u - least);
            }
            if (far >= 0x7f800000u - least) atomicOr(&sh->odd[block / 32u], 1u << (block % 32u));
            #pragma unroll
            for (int j = 0; j < N / 2; j += 32) {
                // 32 x 32 outputs through the warp's buffer: then consecutive lanes have consecutive rows
                float4 *st = reinterpret_cast<float4 *>(stage);
                #pragma unroll
                for (unsigned i = 0; i < 8; i++)
                    st[lane * 8u + (i ^ (lane & 7u))] = make_float4(sum[j + 4 * i], sum[j + 4 * i + 1], sum[j + 4 * i + 2], sum[j + 4 * i + 3]);
                __syncwarp();
                // not unrolled: the code of an activation once per piece
                #pragma unroll 1
                for (unsigned n = lane >> 3; n < 32u; n += 4u) out(n0 + n, m0 + j + (lane & 7u) * 4u, st[n * 8u + ((lane & 7u) ^ (n & 7u))]);
                __syncwarp();
            }
            out.late(n0 + (lane >> 3), 4u, 8u, m0 + (lane & 7u) * 4u, N / 64);
        }
        all_roles_done();
    }
}

}  // namespace split
