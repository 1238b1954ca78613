// aspen_b200_matmul_noalloc: one matmul layer for callers that must not allocate.
//
// Who cannot allocate: plug-ins that are handed a fixed memory budget by their host framework (a
// serving runtime that pre-sizes every pool at start-up and treats a later cudaMalloc as a bug), and
// latency-critical loops where the implicit device synchronisation of cudaMalloc / cudaFree is not
// acceptable.  The regular API builds a device image per nasm (arena, descriptors, counters, queue)
// with cudaMalloc; a single layer has no dependencies between its tiles, so this entry point is one kernel
// launch over the output blocks that needs no memory besides the caller's own buffers, and one wait.
//
//   * n_cols <= 8 (a few tokens): the layer reads its weights once and does next to nothing else, so a warp takes one
//     weight row, its lanes stride over k with wide loads, and the dot products with all columns end in a
//     warp reduction -- every SM pulls weights at once, which no 32-row block shape achieves here.
//     The line lies at 8: with 16 columns the 32 x 32 blocks below are faster (19.9 against 23.6 us at k = 768, m = 3072).
//   * larger: the fp32 FMA blocks of gemm_ffma.cuh, or the tensor cores over operands split into bf16 parts (gemm_split.cuh), by
//     `pick_matmul` (matmul_pick.h).
// B200, wall time of a call, launch and wait included (columns x k x rows):  1 x 768 x 768 17 us;  333 x 770 x 1000 39 us split (44 in
// FMA blocks);  4096 x 768 x 3072 180 split (466 in FMA blocks).
#include "internal.h"
#include "tiles_simt.cuh"
#include "gemm_ffma.cuh"
#include "gemm_split.cuh"
#include "call_slots.h"
#include "matmul_pick.h"

#include <cuda_runtime.h>
#include <algorithm>
#include <chrono>

namespace {

constexpr unsigned NOALLOC_MAX_TILES = ASPEN_B200_NOALLOC_MAX_TILES;
constexpr unsigned NOALLOC_TILE = 128;

struct Args {
    const float *x, *w, *bias;
    float *out;
    unsigned n_cols, k, m;
    int act;
    bool vec_out;             // rows of out start on 16-byte boundaries
};

// VEC consecutive values of a row in one load (16, 8 or 4 bytes, whatever every row's alignment allows); zeros outside.
template <int VEC>
struct Rows {
    const float *base;
    unsigned rows, k;
    __device__ __forceinline__ float4 operator()(unsigned row, unsigned k0) const {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= rows) return v;
        const float *p = base + (size_t)row * k + k0;
        if (VEC == 4) {
            if (k0 < k) v = __ldg(reinterpret_cast<const float4 *>(p));
        } else if (VEC == 2) {
            if (k0 < k) { const float2 a = __ldg(reinterpret_cast<const float2 *>(p)); v.x = a.x; v.y = a.y; }
            if (k0 + 2u < k) { const float2 a = __ldg(reinterpret_cast<const float2 *>(p + 2)); v.z = a.x; v.w = a.y; }
        } else {
            if (k0 < k) v.x = __ldg(p);
            if (k0 + 1u < k) v.y = __ldg(p + 1);
            if (k0 + 2u < k) v.z = __ldg(p + 2);
            if (k0 + 3u < k) v.w = __ldg(p + 3);
        }
        return v;
    }
};

// The rare activations stay out of line: inlined 32 times their double-precision forms are many times the instruction cache.
static __device__ __noinline__ float activate_rare(float x, int act) { return activate(x, act); }
__device__ __forceinline__ float act_value(float x, int act) {
    if (act == NO_ACTIVATION || act == LINEAR) return x;
    if (act == RELU) return x > 0.f ? x : 0.f;
    if (act == GELU) return 0.5f * x * (1.f + erff(x * 0.7071067811865475f));
    return activate_rare(x, act);
}

struct Finish {
    const Args &a;
    unsigned m0, n0;
    __device__ __forceinline__ void operator()(unsigned mi, unsigned ni, const float *v) const {
        const unsigned m = m0 + mi, n = n0 + ni;
        if (n >= a.n_cols || m >= a.m) return;
        float r[4];
        #pragma unroll
        for (unsigned j = 0; j < 4; j++) r[j] = act_value(v[j] + (a.bias && m + j < a.m ? __ldg(a.bias + m + j) : 0.f), a.act);
        float *o = a.out + (size_t)n * a.m + m;
        if (a.vec_out && m + 4u <= a.m) *reinterpret_cast<float4 *>(o) = make_float4(r[0], r[1], r[2], r[3]);
        else
            #pragma unroll
            for (unsigned j = 0; j < 4; j++) if (m + j < a.m) o[j] = r[j];
    }
};

// Block operand: VEC-wide asynchronous copies of a row's values.
template <int VEC, int NR>
struct Stage {
    const float *base;
    unsigned rows, k;
    const float *p[NR];
    bool ok[NR];
    unsigned k0;
    __device__ __forceinline__ Stage(const float *b, unsigned r, unsigned kk) : base(b), rows(r), k(kk), k0(0) {}
    __device__ __forceinline__ void row(int i, unsigned r) { ok[i] = r < rows; p[i] = base + (size_t)(ok[i] ? r : 0u) * k; }
    __device__ __forceinline__ void at(unsigned kk) { k0 = kk; }
    __device__ __forceinline__ void copy(unsigned dst, int i) const {
        #pragma unroll
        for (unsigned e = 0; e < 4; e += VEC) {
            const bool in = ok[i] && k0 + e < k;
            fmablk::copy_async<VEC * 4>(dst + e * 4u, in ? p[i] + k0 + e : base, in);
        }
    }
};

struct BlockBarrier { __device__ __forceinline__ void operator()() const { __syncthreads(); } };

template <typename S, int VEC>
__global__ void __launch_bounds__(fmablk::THREADS, 2) matmul_blocks(const Args a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned m0 = blockIdx.x * S::BM, n0 = blockIdx.y * S::BN;
    Stage<VEC, S::RW> lw(a.w + (size_t)m0 * a.k, a.m - m0, a.k);
    Stage<VEC, S::RX> lx(a.x + (size_t)n0 * a.k, a.n_cols - n0, a.k);
    Finish fin{a, m0, n0};
    fmablk::block<S>(smem, threadIdx.x, a.k, lw, lx, BlockBarrier(), fin);
}

// A word for each of the calls that run matmul_split at the same time: a wait of that call's kernel ran out.  One word for all would have
// a call clear another's, and take the failure of another for its own.
constexpr unsigned CALLS = 1024;
__device__ unsigned split_failed[CALLS];
CallSlots<CALLS> call_slots;

template <int VEC>
struct Operands {
    Rows<VEC> w, x;
    __device__ __forceinline__ float4 operator()(bool weight, unsigned row, unsigned k) const { return weight ? w(row, k) : x(row, k); }
    __device__ __forceinline__ const float *at(bool weight, unsigned row, unsigned k) const { return (weight ? w.base : x.base) + (size_t)row * x.k + k; }
    __device__ __forceinline__ unsigned ld() const { return x.k; }
    __device__ __forceinline__ float4 piece(const float *p) const {
        if (VEC == 4) return __ldg(reinterpret_cast<const float4 *>(p));
        if (VEC == 2) {
            const float2 a = __ldg(reinterpret_cast<const float2 *>(p)), b = __ldg(reinterpret_cast<const float2 *>(p + 2));
            return make_float4(a.x, a.y, b.x, b.y);
        }
        return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
    }
};
// Bias, the common activations and the store of four outputs; rare activations go over the stored values afterwards, where nothing
// else is in registers.
struct FinishPiece {
    const Args &a;
    __device__ __forceinline__ bool rare() const { return a.act != NO_ACTIVATION && a.act != LINEAR && a.act != RELU && a.act != GELU; }
    __device__ __forceinline__ void operator()(unsigned n, unsigned m, const float4 &v) const {
        if (n >= a.n_cols || m >= a.m) return;
        float r[4] = {v.x, v.y, v.z, v.w};
        #pragma unroll
        for (unsigned j = 0; j < 4; j++) {
            if (a.bias && m + j < a.m) r[j] += __ldg(a.bias + m + j);
            if (a.act == RELU) r[j] = r[j] > 0.f ? r[j] : 0.f;
            else if (a.act == GELU) r[j] = 0.5f * r[j] * (1.f + erff(r[j] * 0.7071067811865475f));
        }
        float *o = a.out + (size_t)n * a.m + m;
        if (a.vec_out && m + 4u <= a.m) *reinterpret_cast<float4 *>(o) = make_float4(r[0], r[1], r[2], r[3]);
        else
            #pragma unroll
            for (unsigned j = 0; j < 4; j++) if (m + j < a.m) o[j] = r[j];
    }
    __device__ __forceinline__ void late(unsigned n, unsigned dn, unsigned cn, unsigned m, unsigned cm) const {
        if (!rare()) return;
        #pragma unroll 1
        for (unsigned i = 0; i < cn * cm * 4u; i++) {
            const unsigned col = n + i / (4u * cm) * dn, row = m + i / 4u % cm * 32u + i % 4u;
            if (col < a.n_cols && row < a.m) { float *o = a.out + (size_t)col * a.m + row; *o = activate_rare(*o, a.act); }
        }
    }
};
// Outputs of a block of N rows x 128 columns by FMA blocks, 256 threads of the CTA.  32 x 32 ones, because they have the smallest error (eight
// partial sums; k = 768, operands around 2^-100: 1.8e-7, as where the layer itself takes them; 64 x 64 with one slice 3.5e-7) and few
// registers: those of the 8 x 4 shapes cost the splitting loop of the same warps spills (4096 x 3072 x 3072: 542 us a call instead of
// 523).  4096 x 768 x 3072 with every block marked: 900 us, in 64 x 64 blocks 826.
template <int N, int VEC>
struct Again {
    typedef fmablk::Small S;
    static_assert(S::SMEM_BYTES <= split::Shape<N>::SMEM_BYTES && 2 * NOALLOC_MAX_TILES <= split::MAX_BLOCKS, "room");
    struct Barrier { __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 1, 256;" ::: "memory"); } };
    const Args &a;
    unsigned char *smem;
    __device__ __forceinline__ void operator()(unsigned tid, unsigned n0, unsigned m0) const {
        #pragma unroll 1
        for (unsigned i = 0; i < N / 8; i++) {
            const unsigned n = n0 + i % 4u * 32u, m = m0 + i / 4u * 32u;
            if (n >= a.n_cols || m >= a.m) continue;
            Stage<VEC, S::RW> lw(a.w + (size_t)m * a.k, a.m - m, a.k);
            Stage<VEC, S::RX> lx(a.x + (size_t)n * a.k, a.n_cols - n, a.k);
            Finish fin{a, m, n};
            fmablk::block<S>(smem, tid, a.k, lw, lx, Barrier(), fin);
        }
    }
};
template <int N, int VEC>
__global__ void __launch_bounds__(split::THREADS, 1) matmul_split(const Args a, int call) {
    extern __shared__ __align__(1024) unsigned char split_smem[];
    __shared__ split::Shared sh;
    const Operands<VEC> in{{a.w, a.m, a.k}, {a.x, a.n_cols, a.k}};
    const FinishPiece out{a};
    split::blocks<N>(split_smem, &sh, &split_failed[call], a.n_cols, a.m, a.k, in, out, Again<N, VEC>{a, split_smem});
}

// One weight row per warp, N columns (the last ones may be missing).
template <int N, int VEC>
__global__ void __launch_bounds__(fmablk::THREADS) matmul_rows(const Args a) {
    const unsigned m = blockIdx.x * (fmablk::THREADS / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (m >= a.m) return;
    const Rows<VEC> w{a.w, a.m, a.k}, x{a.x, a.n_cols, a.k};
    float acc[N];
    #pragma unroll
    for (int n = 0; n < N; n++) acc[n] = 0.f;
    constexpr unsigned STEP = 128;
    constexpr int U = N == 1 ? 8 : N <= 4 ? 4 : 2;                         // weight pieces in flight per lane
    for (unsigned k0 = lane * 4u; k0 < a.k; k0 += U * STEP) {
        float4 wv[U];
        #pragma unroll
        for (int u = 0; u < U; u++) wv[u] = w(m, k0 + u * STEP);
        #pragma unroll
        for (int u = 0; u < U; u++)
            #pragma unroll
            for (int n = 0; n < N; n++) {
                const float4 xv = x(n, k0 + u * STEP);
                acc[n] = fmaf(wv[u].x, xv.x, acc[n]); acc[n] = fmaf(wv[u].y, xv.y, acc[n]);
                acc[n] = fmaf(wv[u].z, xv.z, acc[n]); acc[n] = fmaf(wv[u].w, xv.w, acc[n]);
            }
    }
    float mine = 0.f;
    #pragma unroll
    for (int n = 0; n < N; n++) {
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[n] += __shfl_xor_sync(0xffffffffu, acc[n], o);
        if ((int)lane == n) mine = acc[n];
    }
    if (lane < N && lane < a.n_cols) a.out[(size_t)lane * a.m + m] = act_value(mine + (a.bias ? __ldg(a.bias + m) : 0.f), a.act);
}

template <typename S, int VEC>
void launch_blocks(const Args &a, cudaStream_t stream) {
    // the attribute is per device; asking for it on every call costs a fraction of the launch
    cudaFuncSetAttribute(matmul_blocks<S, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM_BYTES);
    matmul_blocks<S, VEC><<<dim3((a.m + S::BM - 1) / S::BM, (a.n_cols + S::BN - 1) / S::BN), fmablk::THREADS, S::SMEM_BYTES, stream>>>(a);
}

template <int N, int VEC>
void launch_split(const Args &a, unsigned sms, int call, cudaStream_t stream) {
    typedef split::Shape<N> S;
    const unsigned blocks = ((a.m + N - 1) / N) * ((a.n_cols + 127) / 128);
    cudaFuncSetAttribute(matmul_split<N, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM_BYTES);
    matmul_split<N, VEC><<<std::min(blocks, sms), split::THREADS, S::SMEM_BYTES, stream>>>(a, call);
}

template <int VEC>
void launch(const Args &a, MatmulKernel kernel, unsigned sms, int call, cudaStream_t stream) {
    if (a.n_cols <= 8) {
        const unsigned grid = (a.m + fmablk::THREADS / 32 - 1) / (fmablk::THREADS / 32);
        if (a.n_cols == 1) matmul_rows<1, VEC><<<grid, fmablk::THREADS, 0, stream>>>(a);
        else if (a.n_cols == 2) matmul_rows<2, VEC><<<grid, fmablk::THREADS, 0, stream>>>(a);
        else if (a.n_cols <= 4) matmul_rows<4, VEC><<<grid, fmablk::THREADS, 0, stream>>>(a);
        else matmul_rows<8, VEC><<<grid, fmablk::THREADS, 0, stream>>>(a);
        return;
    }
    switch (kernel) {
        case FMA_128x64: launch_blocks<fmablk::Large, VEC>(a, stream); break;
        case FMA_64x64: launch_blocks<fmablk::Medium, VEC>(a, stream); break;
        case FMA_32x32: launch_blocks<fmablk::Small, VEC>(a, stream); break;
        case SPLIT_128: launch_split<128, VEC>(a, sms, call, stream); break;
        case SPLIT_64: launch_split<64, VEC>(a, sms, call, stream); break;
    }
}

// Launches and waits.  Whether a wait of the call's kernel ran out is looked at only if the call took long enough for one.
cudaError_t run(const Args &a, int vec, MatmulKernel kernel, unsigned sms, int call, cudaStream_t stream, bool *failed) {
    const auto started = std::chrono::steady_clock::now();
    if (vec == 4) launch<4>(a, kernel, sms, call, stream);
    else if (vec == 2) launch<2>(a, kernel, sms, call, stream);
    else launch<1>(a, kernel, sms, call, stream);
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
    if (err != cudaSuccess || call < 0 || std::chrono::steady_clock::now() - started < std::chrono::nanoseconds(split::LIMIT_NS / 2)) return err;
    unsigned word = 0;
    const unsigned none = 0;
    err = cudaMemcpyFromSymbolAsync(&word, split_failed, sizeof word, call * sizeof word, cudaMemcpyDeviceToHost, stream);
    if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
    if (err != cudaSuccess || word == 0) return err;
    *failed = true;
    err = cudaMemcpyToSymbolAsync(split_failed, &none, sizeof none, call * sizeof none, cudaMemcpyHostToDevice, stream);
    return err == cudaSuccess ? cudaStreamSynchronize(stream) : err;
}

}  // namespace

extern "C" int aspen_b200_matmul_noalloc(const float *x_dev, const float *w_dev, const float *bias_dev, float *out_dev,
                                         unsigned int n_cols, unsigned int k, unsigned int m, int activation, void *cuda_stream) {
    if (!x_dev || !w_dev || !out_dev || n_cols == 0 || k == 0 || m == 0) {
        ASPEN_ERR("aspen_b200_matmul_noalloc: NULL buffer or empty shape\n");
        return -1;
    }
    if (activation < 0 || activation >= NUM_ACTIVATIONS) { ASPEN_ERR("aspen_b200_matmul_noalloc: unknown activation %d\n", activation); return -1; }
    // 64-bit: m or n_cols close to 2^32 must not wrap into a small tile count
    const unsigned long long tiles = (((unsigned long long)m + NOALLOC_TILE - 1) / NOALLOC_TILE) * (((unsigned long long)n_cols + NOALLOC_TILE - 1) / NOALLOC_TILE);
    if (tiles > NOALLOC_MAX_TILES) {
        ASPEN_ERR("aspen_b200_matmul_noalloc: %u x %u outputs need %llu tiles of 128 x 128; the limit is %u. "
                  "Use the regular API (it allocates) for larger layers.\n", m, n_cols, tiles, NOALLOC_MAX_TILES);
        return -2;
    }
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess || sms <= 0) { ASPEN_ERR("aspen_b200_matmul_noalloc: no current CUDA device (%s)\n", cudaGetErrorString(err)); return -3; }
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    const Args a{x_dev, w_dev, bias_dev, out_dev, n_cols, k, m, activation, m % 4 == 0 && reinterpret_cast<uintptr_t>(out_dev) % 16 == 0};
    const uintptr_t align = reinterpret_cast<uintptr_t>(x_dev) | reinterpret_cast<uintptr_t>(w_dev);
    const int vec = k % 4 == 0 && align % 16 == 0 ? 4 : k % 2 == 0 && align % 8 == 0 ? 2 : 1;
    MatmulKernel kernel = pick_matmul(n_cols, k, m, (unsigned)sms, vec);
    int call = -1;
    if (n_cols > 8 && kernel >= SPLIT_128 && (call = call_slots.take()) < 0) kernel = pick_matmul(n_cols, k, m, (unsigned)sms, vec, false);
    bool failed = false;
    err = run(a, vec, kernel, (unsigned)sms, call, stream, &failed);
    // a word that is set and could not be cleared keeps its number
    if (call >= 0 && !(failed && err != cudaSuccess)) call_slots.give(call);
    if (failed) { ASPEN_ERR("aspen_b200_matmul_noalloc: a wait of the kernel ran out\n"); return -3; }
    if (err != cudaSuccess) { ASPEN_ERR("aspen_b200_matmul_noalloc: %s\n", cudaGetErrorString(err)); return -3; }
    return 0;
}
