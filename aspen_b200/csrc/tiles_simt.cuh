// Tile kernels that run on the CUDA cores: the memory-bound layer types (residual, pooling,
// layernorm, softmax, yolo, append) and the fp32-FFMA validation variant of the contraction tiles.
// Every function is executed by `nthr` cooperating threads of one CTA (thread ids 0..nthr-1) on
// one ninst tile.  Semantics follow the reference tile kernels, src/tiled_kernels.c (cited per
// function); activations are read with L1 bypass because other SMs produce them during the same
// kernel.
#pragma once
#include "device_types.h"
#include "gemm_ffma.cuh"
#include "../../include/aspen_b200.h"

// Barrier among the worker threads of a CTA only (the control warp does not take part).
__device__ __forceinline__ void worker_barrier(unsigned nthr) { asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory"); }

__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float ldcg1(const float *p) { return __ldcg(p); }

// ref src/naive_kernels.c:11-57 (double-precision exp/tanh where the reference calls the double libm)
__device__ __forceinline__ float activate(float x, int act) {
    switch (act) {
        case RELU: return x > 0.f ? x : 0.f;
        case LEAKY_RELU: return x > 0.f ? x : (float)(0.1 * (double)x);
        case ELU: return x > 0.f ? x : (float)(0.1 * (exp((double)x) - 1.0));
        case SELU: return x > 0.f ? (float)(1.0507 * (double)x) : (float)(1.0507 * 1.67326 * (exp((double)x) - 1.0));
        case SIGMOID: return (float)(1.0 / (1.0 + exp(-(double)x)));
        case TANH: return (float)tanh((double)x);
        case GELU: return 0.5f * x * (1.f + erff(x * 0.7071067811865475f));
        case GELU_ACCURATE: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
        default: return x;   // NO_ACTIVATION, LINEAR
    }
}

// GELU for the tensor-core epilogue, where 128 values per thread go through it.  The library erff / tanhf
// cost an order of magnitude more there than the contraction's own main loop; these forms are accurate to a
// few 1e-7 (far inside the TF32 bound) and branch-free.  The fp32 validation mode keeps `activate`.
//   erf: Abramowitz & Stegun 7.1.26, |error| <= 1.5e-7;  tanh(u) = 1 - 2 / (1 + exp(2u)), u clamped to +-15.
__device__ __forceinline__ float gelu_erf_fast(float x) {
    const float z = fabsf(x) * 0.7071067811865475f;
    const float t = __fdividef(1.f, fmaf(0.3275911f, z, 1.f));
    float p = fmaf(1.061405429f, t, -1.453152027f);
    p = fmaf(p, t, 1.421413741f);
    p = fmaf(p, t, -0.284496736f);
    p = fmaf(p, t, 0.254829592f);
    const float erf_abs = 1.f - p * t * __expf(-z * z);
    return 0.5f * x * (1.f + copysignf(erf_abs, x));
}
__device__ __forceinline__ float gelu_tanh_fast(float x) {
    float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    u = fminf(fmaxf(u, -15.f), 15.f);
    const float th = 1.f - __fdividef(2.f, 1.f + __expf(2.f * u));
    return 0.5f * x * (1.f + th);
}

// The tensor cores read only the upper 19 bits of an fp32 operand (TF32), i.e. they truncate.
// Truncation is biased toward zero and the bias compounds over a deep network, so every layer whose
// output feeds a tensor-core layer stores values already rounded to nearest TF32; the later
// truncation is then exact.  (Weights are rounded the same way when they are uploaded.)
__device__ __forceinline__ float tf32_round(float x) {
    unsigned u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
    return __uint_as_float(u);
}
__device__ __forceinline__ float finish(float x, const LayerDev &L) { x = activate(x, L.act); return L.round_out ? tf32_round(x) : x; }
__device__ __forceinline__ float store_round(float x, const LayerDev &L) { return L.round_out ? tf32_round(x) : x; }

// Output pixel (flattened column index) -> batch and top-left input coordinate of its window.
struct PixelWin { int b, ih0, iw0; };
__device__ __forceinline__ PixelWin pixel_window(const LayerDev &L, unsigned col) {
    unsigned hw = L.OH * L.OW;
    unsigned b = col / hw, r = col - b * hw;
    unsigned oh = r / L.OW, ow = r - oh * L.OW;
    PixelWin w;
    w.b = (int)b;
    w.ih0 = (int)(oh * L.stride) - (int)L.pad;
    w.iw0 = (int)(ow * L.stride) - (int)L.pad;
    return w;
}
// Pointer to the channel vector of input pixel (b, ih, iw), or nullptr when it is padding.
__device__ __forceinline__ const float *input_pixel(const LayerDev &L, const PixelWin &w, int kh, int kw) {
    int ih = w.ih0 + kh, iw = w.iw0 + kw;
    if (ih < 0 || ih >= (int)L.IH || iw < 0 || iw >= (int)L.IW) return nullptr;
    return L.in0 + ((size_t)(w.b * (int)L.IH + ih) * L.IW + iw) * L.ld0;
}

// ref src/tiled_kernels.c:613-638.  Pure streaming (12 bytes per element): four independent 16-byte load pairs are in flight per
// thread before the first use.  ReLU and no activation have loops of their own: with every activation inlined at each element the
// loop outgrew the instruction cache (256 x 24 elements 9 - 17 us, now 2.0 - 2.6).
enum { ACT_NONE = 0, ACT_RELU = 1, ACT_OTHER = 2 };
template <int KIND>
static __device__ __noinline__ void residual_loop(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned h4 = ((T.pos_h | L.ld0 | L.ld1 | L.ldc) & 3u) ? 0u : T.tile_h >> 2, tail = T.tile_h - 4u * h4;      // whole aligned pieces, and the rest
    const unsigned tile_w = T.tile_w, pos_w = T.pos_w, pos_h = T.pos_h, total = tile_w * h4;
    const size_t ld0 = L.ld0, ld1 = L.ld1, ldc = L.ldc;
    const float *in0 = L.in0, *in1 = L.in1;
    float *out = L.out;
    const bool round = L.round_out != 0;
    const int act = L.act;
    auto one = [&](float x) {
        if (KIND == ACT_RELU) x = x > 0.f ? x : 0.f;
        if (KIND == ACT_OTHER) x = activate(x, act);
        return round ? tf32_round(x) : x;
    };
    constexpr int U = KIND == ACT_OTHER ? 1 : 4;
    for (unsigned i0 = tid; i0 < total; i0 += nthr * U) {
        float4 a[U], b[U];
        size_t off[U];
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned i = min(i0 + u * nthr, total - 1u), n = i / h4, m = pos_h + 4u * (i - n * h4);
            const size_t col = pos_w + n;
            a[u] = ldcg4(in0 + col * ld0 + m);
            b[u] = ldcg4(in1 + col * ld1 + m);
            off[u] = col * ldc + m;
        }
        #pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * nthr < total)
                *reinterpret_cast<float4 *>(out + off[u]) = make_float4(one(a[u].x + b[u].x), one(a[u].y + b[u].y), one(a[u].z + b[u].z), one(a[u].w + b[u].w));
    }
    for (unsigned i = tid; i < tile_w * tail; i += nthr) {
        const unsigned n = i / tail, m = pos_h + 4u * h4 + (i - n * tail);
        const size_t col = pos_w + n;
        out[col * ldc + m] = one(ldcg1(in0 + col * ld0 + m) + ldcg1(in1 + col * ld1 + m));
    }
}
static __device__ __forceinline__ void tile_residual(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    if (L.act == RELU) residual_loop<ACT_RELU>(L, T, tid, nthr);
    else if (L.act == NO_ACTIVATION || L.act == LINEAR) residual_loop<ACT_NONE>(L, T, tid, nthr);
    else residual_loop<ACT_OTHER>(L, T, tid, nthr);
}

// Max pooling with a small window, whole 16-byte pieces of channels: taps outside the image are moved to the nearest pixel inside,
// which the window contains as well, so all KH x KW loads of U outputs are unconditional and in flight together.  With a
// test per tap the loads went out a few at a time: 64 x 100352 outputs (3 x 3, stride 2), launched alone, 158 -> 40 us per SM.
template <int KH, int KW, int U>
static __device__ __noinline__ void tile_max_small(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned h4 = T.tile_h >> 2, total = T.tile_w * h4, pos_w = T.pos_w, pos_h = T.pos_h, hw = L.OH * L.OW, OW = L.OW;
    const int IH = (int)L.IH, IW = (int)L.IW, stride = (int)L.stride, pad = (int)L.pad, act = L.act;
    const size_t ld0 = L.ld0, ldc = L.ldc;
    const float *in = L.in0;
    float *out = L.out;
    const bool round = L.round_out != 0;
    for (unsigned i0 = tid; i0 < total; i0 += nthr * U) {
        float4 v[U][KH * KW];
        unsigned n[U], m[U];
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned i = min(i0 + u * nthr, total - 1u);       // past the end: the last piece again
            n[u] = pos_w + i / h4;
            m[u] = pos_h + 4u * (i % h4);
            const unsigned b = n[u] / hw, r = n[u] - b * hw, oh = r / OW, ow = r - oh * OW;
            const int y = (int)oh * stride - pad, x = (int)ow * stride - pad;
            const float *img = in + (size_t)b * IH * IW * ld0 + m[u];
            #pragma unroll
            for (int kh = 0; kh < KH; kh++) {
                const int ih = min(max(y + kh, 0), IH - 1);
                #pragma unroll
                for (int kw = 0; kw < KW; kw++) v[u][kh * KW + kw] = ldcg4(img + (size_t)(ih * IW + min(max(x + kw, 0), IW - 1)) * ld0);
            }
        }
        #pragma unroll
        for (int u = 0; u < U; u++) {
            float4 a = v[u][0];
            #pragma unroll
            for (int k = 1; k < KH * KW; k++) {
                const float4 x = v[u][k];
                a.x = a.x >= x.x ? a.x : x.x; a.y = a.y >= x.y ? a.y : x.y; a.z = a.z >= x.z ? a.z : x.z; a.w = a.w >= x.w ? a.w : x.w;
            }
            if (act != NO_ACTIVATION && act != LINEAR) { a.x = activate(a.x, act); a.y = activate(a.y, act); a.z = activate(a.z, act); a.w = activate(a.w, act); }
            if (round) { a.x = tf32_round(a.x); a.y = tf32_round(a.y); a.z = tf32_round(a.z); a.w = tf32_round(a.w); }
            if (i0 + u * nthr < total) *reinterpret_cast<float4 *>(out + (size_t)n[u] * ldc + m[u]) = a;
        }
    }
}

// Average pooling whose windows lie inside the image (global pools): sixteen taps in flight, summed in order.  Tested tap by tap, a
// 7 x 7 window took 20 us.
static __device__ __noinline__ void tile_avg_inside(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned h4 = T.tile_h >> 2, total = T.tile_w * h4, KW = L.KW, taps = L.KH * KW, IW = L.IW;
    const size_t ld0 = L.ld0;
    const float inv = 1.f / (float)taps;
    for (unsigned i = tid; i < total; i += nthr) {
        const unsigned n = T.pos_w + i / h4, m = T.pos_h + 4u * (i % h4);
        const PixelWin w = pixel_window(L, n);
        const float *img = L.in0 + ((size_t)(w.b * (int)L.IH + w.ih0) * IW + w.iw0) * ld0 + m;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned kw = 0;
        const float *p = img;
        for (unsigned t0 = 0; t0 < taps; t0 += 16u) {
            float4 v[16];
            #pragma unroll
            for (unsigned g = 0; g < 16; g++) {
                v[g] = t0 + g < taps ? ldcg4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
                p += ld0;
                if (++kw == KW) { kw = 0; p += (size_t)(IW - KW) * ld0; }
            }
            #pragma unroll
            for (unsigned g = 0; g < 16; g++) { a.x += v[g].x; a.y += v[g].y; a.z += v[g].z; a.w += v[g].w; }
        }
        float *o = L.out + (size_t)n * L.ldc + m;
        *reinterpret_cast<float4 *>(o) = make_float4(finish(a.x * inv, L), finish(a.y * inv, L), finish(a.z * inv, L), finish(a.w * inv, L));
    }
}

// Pooling of any window (ref src/tiled_kernels.c:411-501).  Max ignores padded taps (all padded -> -inf); average divides by
// the full window size, padding counted.  A thread owns four channels of an output pixel and works on two such
// items at a time; the window's taps are fetched nine at a time (a whole 3 x 3 window), all loads of both items
// issued before the first is used (a tap outside the image reads nothing and contributes the neutral element),
// so the tile is bound by bandwidth instead of one load latency per tap.
template <bool IS_MAX>
static __device__ __noinline__ void tile_pool(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned h4 = ((T.pos_h | L.ld0 | L.ldc) & 3u) ? 0u : T.tile_h >> 2, per_col = T.tile_h - 3u * h4;   // whole aligned pieces, and the rest
    const float inv = 1.f / (float)(L.KH * L.KW);
    const float init = IS_MAX ? -INFINITY : 0.f;
    const unsigned taps = L.KH * L.KW, total = T.tile_w * per_col;
    constexpr unsigned G = 9, U = 2;
    for (unsigned i0 = tid; i0 < total; i0 += nthr * U) {
        PixelWin w[U];
        unsigned m[U];
        size_t col[U];
        bool vec[U], live[U];
        float4 acc[U];
        #pragma unroll
        for (unsigned u = 0; u < U; u++) {
            const unsigned i = i0 + u * nthr;
            live[u] = i < total;
            const unsigned n = live[u] ? i / per_col : 0u, j = live[u] ? i - n * per_col : 0u;
            col[u] = T.pos_w + n;
            w[u] = pixel_window(L, (unsigned)col[u]);
            vec[u] = j < h4;
            m[u] = T.pos_h + (vec[u] ? 4 * j : 4 * h4 + (j - h4));
            acc[u] = make_float4(init, init, init, init);
        }
        unsigned kh = 0, kw = 0;
        for (unsigned t0 = 0; t0 < taps; t0 += G) {
            float4 v[U][G];
            #pragma unroll
            for (unsigned g = 0; g < G; g++) {
                const bool tap_ok = t0 + g < taps;
                #pragma unroll
                for (unsigned u = 0; u < U; u++) {
                    v[u][g] = make_float4(init, init, init, init);
                    if (tap_ok && live[u]) {
                        const float *src = input_pixel(L, w[u], (int)kh, (int)kw);
                        if (src) {
                            if (vec[u]) v[u][g] = ldcg4(src + m[u]);
                            else v[u][g].x = ldcg1(src + m[u]);
                        }
                    }
                }
                if (tap_ok && ++kw == L.KW) { kw = 0; kh++; }
            }
            #pragma unroll
            for (unsigned u = 0; u < U; u++) {
                #pragma unroll
                for (unsigned g = 0; g < G; g++) {
                    const float4 x = v[u][g];
                    if (IS_MAX) { acc[u].x = acc[u].x >= x.x ? acc[u].x : x.x; acc[u].y = acc[u].y >= x.y ? acc[u].y : x.y; acc[u].z = acc[u].z >= x.z ? acc[u].z : x.z; acc[u].w = acc[u].w >= x.w ? acc[u].w : x.w; }
                    else { acc[u].x += x.x; acc[u].y += x.y; acc[u].z += x.z; acc[u].w += x.w; }
                }
            }
        }
        #pragma unroll
        for (unsigned u = 0; u < U; u++) {
            if (!live[u]) continue;
            float4 a = acc[u];
            if (!IS_MAX) { a.x *= inv; a.y *= inv; a.z *= inv; a.w *= inv; }
            if (vec[u]) {
                float4 o = {finish(a.x, L), finish(a.y, L), finish(a.z, L), finish(a.w, L)};
                *reinterpret_cast<float4 *>(L.out + col[u] * L.ldc + m[u]) = o;
            } else {
                L.out[col[u] * L.ldc + m[u]] = finish(a.x, L);
            }
        }
    }
}

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ref src/tiled_kernels.c:743-783: one pass mean / E[x^2], eps 1e-6, gain and shift.  One warp per column.
// A column of up to 1024 features is read ONCE: each lane keeps its up to eight 16-byte pieces in registers (all
// loads issued before the first use), the warp reduces sum and sum of squares, and the normalised values are
// written from the registers.  Longer or unaligned columns take the two-pass loop.
static __device__ __noinline__ void tile_layernorm(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned warp = tid >> 5, lane = tid & 31, nwarp = nthr >> 5;
    const unsigned M = T.tile_h;
    const float *gain = L.weight + T.pos_h;
    const float *shift = L.bias ? L.bias + T.pos_h : nullptr;
    const bool aligned = ((L.ld0 | L.ldc | T.pos_h) & 3u) == 0u, in_regs = aligned && M <= 1024u && (M & 3u) == 0u;
    if (in_regs) {
        // a column of a warp at a time, all its loads (and, once, the gains' and shifts') in flight before the first use; two columns
        // at a time spill
        const unsigned tile_w = T.tile_w, pos_w = T.pos_w, pos_h = T.pos_h;
        const size_t ld0 = L.ld0, ldc = L.ldc;
        const float *in = L.in0 + pos_h;
        float *out = L.out + pos_h;
        const bool round = L.round_out != 0;
        float4 g[8], b[8];
        #pragma unroll
        for (unsigned q = 0; q < 8; q++) {
            const unsigned m = lane * 4u + q * 128u;
            g[q] = m < M ? __ldg(reinterpret_cast<const float4 *>(gain + m)) : make_float4(0.f, 0.f, 0.f, 0.f);
            b[q] = m < M && shift ? __ldg(reinterpret_cast<const float4 *>(shift + m)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (unsigned n = warp; n < tile_w; n += nwarp) {
            float4 v[8];
            const float *x = in + (size_t)(pos_w + n) * ld0;
            #pragma unroll
            for (unsigned q = 0; q < 8; q++) {
                const unsigned m = lane * 4u + q * 128u;
                v[q] = m < M ? ldcg4(x + m) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            float s = 0.f, ss = 0.f;
            #pragma unroll
            for (unsigned q = 0; q < 8; q++) {
                const float4 t = v[q];
                s += t.x + t.y + t.z + t.w;
                ss += t.x * t.x + t.y * t.y + t.z * t.z + t.w * t.w;
            }
            s = warp_sum(s);
            ss = warp_sum(ss);
            const float mean = s / (float)M, var = ss / (float)M - mean * mean, inv = 1.f / sqrtf(var + 1e-6f);
            float *y = out + (size_t)(pos_w + n) * ldc;
            #pragma unroll
            for (unsigned q = 0; q < 8; q++) {
                const unsigned m = lane * 4u + q * 128u;
                if (m < M) {
                    const float4 t = v[q];
                    float4 o = {(t.x - mean) * inv * g[q].x, (t.y - mean) * inv * g[q].y, (t.z - mean) * inv * g[q].z, (t.w - mean) * inv * g[q].w};
                    if (shift) { o.x += b[q].x; o.y += b[q].y; o.z += b[q].z; o.w += b[q].w; }
                    if (round) { o.x = tf32_round(o.x); o.y = tf32_round(o.y); o.z = tf32_round(o.z); o.w = tf32_round(o.w); }
                    *reinterpret_cast<float4 *>(y + m) = o;
                }
            }
        }
        return;
    }
    for (unsigned n = warp; n < T.tile_w; n += nwarp) {
        const float *x = L.in0 + (size_t)(T.pos_w + n) * L.ld0 + T.pos_h;
        float *y = L.out + (size_t)(T.pos_w + n) * L.ldc + T.pos_h;
        float s = 0.f, ss = 0.f;
        const unsigned M4 = aligned ? M & ~3u : 0u;
        for (unsigned m = lane * 4; m < M4; m += 128) {
            float4 v = ldcg4(x + m);
            s += v.x + v.y + v.z + v.w;
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        for (unsigned m = M4 + lane; m < M; m += 32) { float v = ldcg1(x + m); s += v; ss += v * v; }
        s = warp_sum(s);
        ss = warp_sum(ss);
        float mean = s / (float)M;
        float var = ss / (float)M - mean * mean;
        float inv = 1.f / sqrtf(var + 1e-6f);
        for (unsigned m = lane * 4; m < M4; m += 128) {
            float4 v = ldcg4(x + m);
            float4 g = *reinterpret_cast<const float4 *>(gain + m);
            float4 o = {(v.x - mean) * inv * g.x, (v.y - mean) * inv * g.y, (v.z - mean) * inv * g.z, (v.w - mean) * inv * g.w};
            if (shift) { float4 b = *reinterpret_cast<const float4 *>(shift + m); o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w; }
            o.x = store_round(o.x, L); o.y = store_round(o.y, L); o.z = store_round(o.z, L); o.w = store_round(o.w, L);
            *reinterpret_cast<float4 *>(y + m) = o;
        }
        for (unsigned m = M4 + lane; m < M; m += 32) {
            float o = (ldcg1(x + m) - mean) * inv * gain[m];
            if (shift) o += shift[m];
            y[m] = store_round(o, L);
        }
    }
}

// ref src/tiled_kernels.c:640-673: max-subtracted softmax down each column.  One warp per column.
static __device__ __noinline__ void tile_softmax(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned warp = tid >> 5, lane = tid & 31, nwarp = nthr >> 5;
    const unsigned M = T.tile_h;
    for (unsigned n = warp; n < T.tile_w; n += nwarp) {
        const float *x = L.in0 + (size_t)(T.pos_w + n) * L.ld0 + T.pos_h;
        float *y = L.out + (size_t)(T.pos_w + n) * L.ldc + T.pos_h;
        float mx = -INFINITY;
        for (unsigned m = lane; m < M; m += 32) mx = fmaxf(mx, ldcg1(x + m));
        mx = warp_max(mx);
        float s = 0.f;
        for (unsigned m = lane; m < M; m += 32) s += expf(ldcg1(x + m) - mx);
        s = warp_sum(s);
        for (unsigned m = lane; m < M; m += 32) y[m] = store_round(expf(ldcg1(x + m) - mx) / s, L);
    }
}

// ref src/tiled_kernels.c:675-709: box decode of one detection head.
static __device__ __noinline__ void tile_yolo(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned C = L.p_out_c;
    const unsigned a_num = L.p_in_c / C, hw = L.IH * L.IW;
    for (unsigned i = tid; i < T.tile_w * C; i += nthr) {
        unsigned n = i / C, j = i - n * C;
        unsigned w_pos = T.pos_w + n;
        unsigned bidx = w_pos / (hw * a_num), b_num = w_pos % (hw * a_num);
        unsigned aidx = b_num / hw, wh = b_num % hw;
        unsigned hidx = wh / L.IW, widx = wh % L.IW;
        unsigned cidx = T.pos_h + aidx * C;
        const float *in = L.in0 + (size_t)(bidx * hw + hidx * L.IW + widx) * L.ld0 + cidx;
        float *out = L.out + (size_t)w_pos * L.ldc + T.pos_h;
        float v = ldcg1(in + j), o;
        if (j == 0) o = (1.0f / (1.0f + expf(-v)) + (float)widx) * (float)L.p_stride;
        else if (j == 1) o = (1.0f / (1.0f + expf(-v)) + (float)hidx) * (float)L.p_stride;
        else if (j == 2) o = expf(v) * L.anchors[2 * aidx];
        else if (j == 3) o = expf(v) * L.anchors[2 * aidx + 1];
        else o = 1.0f / (1.0f + expf(-v));
        out[j] = store_round(o, L);
    }
}

// ref src/tiled_kernels.c:711-741: nearest-neighbour upsample of PARENT_0 concatenated with PARENT_1.
static __device__ __noinline__ void tile_append(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned c1 = L.p_in_c, c2 = L.p_out_c - L.p_in_c, C = c1 + c2;
    const unsigned w2 = L.OW, w1 = L.IW, s = L.p_stride;
    for (unsigned i = tid; i < T.tile_w * C; i += nthr) {
        unsigned n = i / C, c = i - n * C;
        unsigned w_pos = T.pos_w + n;
        unsigned widx2 = w_pos % w2, hidx2 = w_pos / w2;
        unsigned widx1 = widx2 / s, hidx1 = hidx2 / s;
        float v = c < c1 ? ldcg1(L.in0 + (size_t)(hidx1 * w1 + widx1) * L.ld0 + c)
                         : ldcg1(L.in1 + (size_t)(hidx2 * w2 + widx2) * L.ld1 + (c - c1));
        L.out[(size_t)w_pos * L.ldc + c] = store_round(v, L);
    }
}

// ---- fp32 FFMA contraction tiles (validation mode) -----------------------------------------
// out[col n][row m] = epilogue( sum_k  W(m, k) * X(n, k) ), fp32 multiply-add.
//   conv     ref src/tiled_kernels.c:161-297   X(n,k): input pixel taps (kh, kw, ic), zero padding
//   matmul   ref src/tiled_kernels.c:299-409   X(n,k): parent column n
//   connected ref src/tiled_kernels.c:502-612  X(n,k): flattened sample n
//   k-attn   ref src/tiled_kernels.c:784-932   W = keys, X = queries of one (batch, head); then
//                                              mask (-1e10), scale 1/sqrt(hd), exp, column normalise
//   v-attn   ref src/tiled_kernels.c:934-1038  W(m,k) = V[token k][feature m], X = probabilities
struct GemmView {
    const float *wbase;   // row m of W starts at wbase + m * wld (k contiguous) unless w_transposed
    size_t wld;
    bool w_transposed;    // v-attn: W(m,k) = wbase[k * wld + m]
    const float *xbase;   // non-conv: row n of X starts at xbase + n * xld
    size_t xld;
    unsigned K;
    bool conv;
};

__device__ __forceinline__ GemmView gemm_view(const LayerDev &L, const TileDev &T) {
    GemmView g;
    g.conv = false; g.w_transposed = false;
    switch (L.type) {
        case CONV_LAYER:
            g.wbase = L.weight + (size_t)T.pos_h * L.Kpad; g.wld = L.Kpad; g.xbase = L.in0; g.xld = L.ld0; g.K = L.K; g.conv = true;
            break;
        case MATMUL_LAYER:
            g.wbase = L.weight + (size_t)T.pos_h * L.Kpad; g.wld = L.Kpad; g.xbase = L.in0 + (size_t)T.pos_w * L.ld0; g.xld = L.ld0; g.K = L.K;
            break;
        case FC_LAYER:   // a convolution whose window is the whole input image (geometry set at upload)
            g.wbase = L.weight + (size_t)T.pos_h * L.Kpad; g.wld = L.Kpad; g.xbase = L.in0; g.xld = L.ld0; g.K = L.K; g.conv = true;
            break;
        case K_ATTENTION_LAYER: {
            unsigned b = T.pos_w / (L.seq * L.heads), head = (T.pos_w % (L.seq * L.heads)) / L.seq, q0 = T.pos_w % L.seq;
            g.wbase = L.in1 + (size_t)(b * L.seq + T.pos_h) * L.ld1 + head * L.hd; g.wld = L.ld1;
            g.xbase = L.in0 + (size_t)(b * L.seq + q0) * L.ld0 + head * L.hd; g.xld = L.ld0; g.K = L.hd;
            break;
        }
        default: {   // V_ATTENTION_LAYER
            unsigned b = T.pos_w / L.seq, head = T.pos_h / L.hd, q0 = T.pos_w % L.seq;
            g.wbase = L.in1 + (size_t)b * L.seq * L.ld1 + T.pos_h; g.wld = L.ld1; g.w_transposed = true;
            g.xbase = L.in0 + (size_t)((b * L.heads + head) * L.seq + q0) * L.ld0; g.xld = L.ld0; g.K = L.seq;
            break;
        }
    }
    return g;
}

// The stored tile once more, transposed, for an attention_v layer that reads its values (LayerDev::vt_out).  The values of a projection
// on the tensor cores are written by its epilogue; this is for layers of any other kind.  Consecutive threads write consecutive
// tokens of a feature.
static __device__ __noinline__ void tile_transposed_copy(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned tile_w = T.tile_w, total = tile_w * T.tile_h, pos_w = T.pos_w, pos_h = T.pos_h, seq = L.seq, vt_seq = L.vt_seq;
    const size_t ldc = L.ldc, vt_ld = L.vt_ld;
    const float *in = L.out;
    float *out = L.vt_out;
    worker_barrier(nthr);
    for (unsigned i = tid; i < total; i += nthr) {
        const unsigned m = pos_h + i / tile_w, col = pos_w + i % tile_w, b = col / seq;
        out[(size_t)m * vt_ld + (size_t)b * vt_seq + (col - b * seq)] = ldcg1(in + (size_t)col * ldc + m);
    }
}

// Layer-0 tile: the uploaded input becomes the columns of the layer's activation matrix that the tile covers: scatter into the column
// stride, rounding, embedding rows of token ids, and the zero-padded copy of a small image.  Sources are read through L2: the
// host's DMA may have written them while this kernel was running.
static __device__ void tile_input(const InputDev &I, const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned H = L.H;
    if (I.ids) {
        // four pieces of rows in flight: each needs its id first
        const unsigned m4 = T.tile_h >> 2, total = T.tile_w * m4, pos_w = T.pos_w, pos_h = T.pos_h;
        const bool round = I.round != 0;
        const size_t ldc = L.ldc;
        float *out = L.out;
        for (unsigned i0 = tid; i0 < total; i0 += 4u * nthr) {
            unsigned t[4], j[4];
            int id[4];
            float4 v[4], p[4];
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned i = min(i0 + u * nthr, total - 1u), c = i / m4;
                t[u] = pos_w + c;
                j[u] = pos_h + (i - c * m4) * 4u;
                id[u] = __ldcg(I.ids + t[u]);
            }
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                id[u] = id[u] < 0 ? 0 : (id[u] >= (int)I.emb_vocab ? (int)I.emb_vocab - 1 : id[u]);
                v[u] = __ldg(reinterpret_cast<const float4 *>(I.emb_tok + (size_t)id[u] * H + j[u]));
                if (I.emb_pos) p[u] = __ldg(reinterpret_cast<const float4 *>(I.emb_pos + (size_t)(t[u] % I.emb_seq) * H + j[u]));
                else p[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                if (I.emb_pos) { v[u].x += p[u].x; v[u].y += p[u].y; v[u].z += p[u].z; v[u].w += p[u].w; }
                if (round) { v[u].x = tf32_round(v[u].x); v[u].y = tf32_round(v[u].y); v[u].z = tf32_round(v[u].z); v[u].w = tf32_round(v[u].w); }
                if (i0 + u * nthr < total) *reinterpret_cast<float4 *>(out + (size_t)t[u] * ldc + j[u]) = v[u];
            }
        }
        return;
    }
    if (I.padded && I.stage && H <= 4u && T.pos_h == 0u) {
        // an image of three channels, columns four floats apart: four pixels are three 16-byte loads, two such groups in flight
        if (H == 3u && L.ldc == 4u && ((T.tile_w | T.pos_w) & 3u) == 0u) {
            const unsigned hw = I.IH * I.IW, IW = I.IW, PH = I.PH, PW = I.PW, pad = I.pad, groups = T.tile_w >> 2, pos_w = T.pos_w;
            const bool round = I.round != 0;
            float4 *padded = reinterpret_cast<float4 *>(I.padded), *out = reinterpret_cast<float4 *>(L.out);
            const float *stage = I.stage;
            for (unsigned g0 = tid; g0 < groups; g0 += 2u * nthr) {
                float f[2][12];
                #pragma unroll
                for (int u = 0; u < 2; u++) {
                    const unsigned g = min(g0 + u * nthr, groups - 1u);
                    #pragma unroll
                    for (int q = 0; q < 3; q++) {
                        const float4 t = ldcg4(stage + (size_t)(pos_w + 4u * g) * 3u + 4 * q);
                        f[u][4 * q] = t.x; f[u][4 * q + 1] = t.y; f[u][4 * q + 2] = t.z; f[u][4 * q + 3] = t.w;
                    }
                }
                #pragma unroll
                for (int u = 0; u < 2; u++) {
                    const unsigned g = g0 + u * nthr;
                    if (g >= groups) break;
                    const unsigned w = pos_w + 4u * g;
                    unsigned b = w / hw, r = w - b * hw, ih = r / IW, iw = r - ih * IW;
                    #pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float4 v = make_float4(f[u][3 * q], f[u][3 * q + 1], f[u][3 * q + 2], 0.f);
                        if (round) { v.x = tf32_round(v.x); v.y = tf32_round(v.y); v.z = tf32_round(v.z); }
                        out[w + q] = v;
                        padded[((size_t)b * PH + ih + pad) * PW + iw + pad] = v;
                        if (++iw == IW) { iw = 0; if (++ih == I.IH) { ih = 0; b++; } }
                    }
                }
            }
            return;
        }
        // an image: one thread per pixel reads its (up to four) channels once and writes both copies
        const unsigned hw = I.IH * I.IW;
        for (unsigned c = tid; c < T.tile_w; c += nthr) {
            const unsigned w = T.pos_w + c, b = w / hw, r = w - b * hw, ih = r / I.IW, iw = r - ih * I.IW;
            const float *src = I.stage + (size_t)w * H;
            float *dst = L.out + (size_t)w * L.ldc;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            v.x = ldcg1(src);
            if (H > 1u) v.y = ldcg1(src + 1);
            if (H > 2u) v.z = ldcg1(src + 2);
            if (H > 3u) v.w = ldcg1(src + 3);
            if (I.round) { v.x = tf32_round(v.x); v.y = tf32_round(v.y); v.z = tf32_round(v.z); v.w = tf32_round(v.w); }
            dst[0] = v.x;
            if (H > 1u) dst[1] = v.y;
            if (H > 2u) dst[2] = v.z;
            if (H > 3u) dst[3] = v.w;
            reinterpret_cast<float4 *>(I.padded)[((size_t)b * I.PH + ih + I.pad) * I.PW + iw + I.pad] = v;
        }
        return;
    }
    if ((I.stage || I.round) && ((T.tile_h | T.pos_h | L.ldc | H) & 3u) == 0u) {
        // 16-byte pieces: consecutive threads take consecutive pieces of a column
        const unsigned m4 = T.tile_h >> 2;
        for (unsigned i = tid; i < T.tile_w * m4; i += nthr) {
            const unsigned c = i / m4, m = T.pos_h + (i - c * m4) * 4u;
            const size_t w = T.pos_w + c;
            float *dst = L.out + w * L.ldc + m;
            float4 v = I.stage ? ldcg4(I.stage + w * H + m) : ldcg4(dst);
            if (I.round) { v.x = tf32_round(v.x); v.y = tf32_round(v.y); v.z = tf32_round(v.z); v.w = tf32_round(v.w); }
            *reinterpret_cast<float4 *>(dst) = v;
        }
    } else if (I.stage || I.round)
        for (unsigned i = tid; i < T.tile_w * T.tile_h; i += nthr) {
            const unsigned c = i / T.tile_h, m = T.pos_h + (i - c * T.tile_h);
            const size_t w = T.pos_w + c;
            float *dst = L.out + w * L.ldc + m;
            float v = I.stage ? ldcg1(I.stage + w * H + m) : ldcg1(dst);
            *dst = I.round ? tf32_round(v) : v;
        }
    if (I.padded && T.pos_h == 0u)
        for (unsigned c = tid; c < T.tile_w; c += nthr) {
            const size_t w = T.pos_w + c, hw = (size_t)I.IH * I.IW, b = w / hw, r = w - b * hw;
            const unsigned ih = (unsigned)(r / I.IW), iw = (unsigned)(r - (size_t)ih * I.IW);
            const float *src = I.stage ? I.stage + w * H : L.out + w * L.ldc;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            v.x = ldcg1(src);
            if (I.IC > 1) v.y = ldcg1(src + 1);
            if (I.IC > 2) v.z = ldcg1(src + 2);
            if (I.IC > 3) v.w = ldcg1(src + 3);
            if (I.round) { v.x = tf32_round(v.x); v.y = tf32_round(v.y); v.z = tf32_round(v.z); v.w = tf32_round(v.w); }
            reinterpret_cast<float4 *>(I.padded)[(b * I.PH + ih + I.pad) * I.PW + iw + I.pad] = v;
        }
}

// ---- contraction tiles in fp32 ------------------------------------------------------------------
// Operand loaders of gemm_ffma.cuh over a layer's matrices, one for each way an operand lies in memory: a loader that chose at run
// time kept the addresses of every way in registers, and the blocks spilled.
template <int NR>
struct DenseRows {            // rows of k contiguous values, in 16-byte pieces: weights (zero padded to Kpad), keys, queries, tokens
    const float *base;
    unsigned rows, k_end, k0;
    const float *p[NR];
    __device__ __forceinline__ DenseRows(const float *b, unsigned r, unsigned ke) : base(b), rows(r), k_end(ke), k0(0) {}
    __device__ __forceinline__ void row(int i, unsigned r, size_t ld) { p[i] = r < rows ? base + (size_t)r * ld : nullptr; }
    __device__ __forceinline__ void at(unsigned k) { k0 = k; }
    __device__ __forceinline__ void copy(unsigned dst, int i) const {
        const bool in = p[i] != nullptr && k0 < k_end;
        fmablk::copy_async<16>(dst, in ? p[i] + k0 : base, in);
    }
};
template <int NR>
struct WeightRows : DenseRows<NR> {
    size_t ld;
    __device__ __forceinline__ WeightRows(const GemmView &g, unsigned r, unsigned ke) : DenseRows<NR>(g.wbase, r, ke), ld(g.wld) {}
    __device__ __forceinline__ void row(int i, unsigned r) { DenseRows<NR>::row(i, r, ld); }
};
template <int NR>
struct TokenRows : DenseRows<NR> {
    size_t ld;
    __device__ __forceinline__ TokenRows(const LayerDev &, const GemmView &g, unsigned, unsigned cols) : DenseRows<NR>(g.xbase, cols, g.K), ld(g.xld) {}
    __device__ __forceinline__ void row(int i, unsigned r) { DenseRows<NR>::row(i, r, ld); }
};
template <int NR>
struct PixelRows {            // taps of output pixels, channels in 16-byte pieces
    const float *in0;
    unsigned K, IC, KW, IH, IW, ld0, pos, cols, k0, ic;
    Divisor by_ic, by_kw;
    int kh, kw;
    const LayerDev &L;
    const float *img[NR];     // the pixel's sample; nullptr: no such pixel
    int y[NR], x[NR];
    __device__ __forceinline__ PixelRows(const LayerDev &l, const GemmView &g, unsigned po, unsigned c)
        : in0(l.in0), K(g.K), IC(l.IC), KW(l.KW), IH(l.IH), IW(l.IW), ld0(l.ld0), pos(po), cols(c), k0(0), ic(0),
          by_ic(l.by_ic), by_kw(l.by_kw), kh(0), kw(0), L(l) {}
    __device__ __forceinline__ void row(int i, unsigned r) {
        const PixelWin w = pixel_window(L, pos + (r < cols ? r : 0u));
        img[i] = r < cols ? in0 + (size_t)w.b * IH * IW * ld0 : nullptr;
        y[i] = w.ih0; x[i] = w.iw0;
    }
    __device__ __forceinline__ void at(unsigned k) {
        k0 = k;
        const unsigned tap = div_by_2_up(k, by_ic);            // whole pieces: at least four channels
        ic = k - tap * IC;
        kh = (int)div_by(tap, by_kw);
        kw = (int)(tap - (unsigned)kh * KW);
    }
    __device__ __forceinline__ void copy(unsigned dst, int i) const {
        const unsigned ih = (unsigned)(y[i] + kh), iw = (unsigned)(x[i] + kw);       // outside the image: negative or too large
        const bool in = img[i] != nullptr && k0 < K && ih < IH && iw < IW;
        fmablk::copy_async<16>(dst, in ? img[i] + (size_t)((ih * IW + iw) * ld0 + ic) : in0, in);
    }
};
// The odd cases, value by value: transposed attention values, channel counts or heads that are no multiple of four.
template <int NR>
struct AnyWeightRows {
    const GemmView &g;
    unsigned rows, k_end, k0, at_row[NR];
    bool ok[NR];
    __device__ __forceinline__ AnyWeightRows(const GemmView &v, unsigned r, unsigned ke) : g(v), rows(r), k_end(ke), k0(0) {}
    __device__ __forceinline__ void row(int i, unsigned r) { ok[i] = r < rows; at_row[i] = ok[i] ? r : 0u; }
    __device__ __forceinline__ void at(unsigned k) { k0 = k; }
    __device__ __forceinline__ void copy(unsigned dst, int i) const {
        #pragma unroll 1
        for (unsigned e = 0; e < 4; e++) {
            const bool in = ok[i] && k0 + e < k_end;
            const size_t off = g.w_transposed ? (size_t)(k0 + e) * g.wld + at_row[i] : (size_t)at_row[i] * g.wld + k0 + e;
            fmablk::copy_async<4>(dst + e * 4u, g.wbase + (in ? off : 0), in);
        }
    }
};
template <int NR>
struct AnyRows {
    const LayerDev &L;
    const GemmView &g;
    unsigned pos, cols, k0, at_row[NR];
    __device__ __forceinline__ AnyRows(const LayerDev &l, const GemmView &v, unsigned po, unsigned c) : L(l), g(v), pos(po), cols(c), k0(0) {}
    __device__ __forceinline__ void row(int i, unsigned r) { at_row[i] = r; }
    __device__ __forceinline__ void at(unsigned k) { k0 = k; }
    __device__ __forceinline__ void copy(unsigned dst, int i) const {
        #pragma unroll 1
        for (unsigned e = 0; e < 4; e++) {
            const unsigned k = k0 + e;
            const float *src = nullptr;
            if (at_row[i] < cols && k < g.K) {
                if (g.conv) {
                    const unsigned tap = k / L.IC;
                    src = input_pixel(L, pixel_window(L, pos + at_row[i]), (int)(tap / L.KW), (int)(tap % L.KW));
                    if (src) src += k - tap * L.IC;
                } else src = g.xbase + (size_t)at_row[i] * g.xld + k;
            }
            fmablk::copy_async<4>(dst + e * 4u, src ? src : L.in0, src != nullptr);
        }
    }
};
// Activations other than ReLU, and the softmax of the scores, are applied to the stored tile afterwards: inlined for each of a
// thread's outputs their double-precision forms made the block's code many times the instruction cache.
__device__ __forceinline__ bool late_activation(const LayerDev &L) {
    return L.type != V_ATTENTION_LAYER && L.type != K_ATTENTION_LAYER && L.act != NO_ACTIVATION && L.act != LINEAR && L.act != RELU;
}
// Bias, ReLU, store of a block's outputs.  Everything it needs is copied here: a load through L, or of a bias that a store
// might have changed, would wait for the store before it.
struct StoreTile {
    const float *bias;
    float *out;
    size_t ldc;
    unsigned tile_h, tile_w, pos_h, m0, n0;
    int act;
    bool round;
    __device__ __forceinline__ StoreTile(const LayerDev &L, const TileDev &T, unsigned m, unsigned n)
        : bias(L.type == V_ATTENTION_LAYER || L.type == K_ATTENTION_LAYER ? nullptr : L.bias), out(L.out + (size_t)T.pos_w * L.ldc + T.pos_h), ldc(L.ldc),
          tile_h(T.tile_h), tile_w(T.tile_w), pos_h(T.pos_h), m0(m), n0(n), act(L.type == V_ATTENTION_LAYER ? (int)NO_ACTIVATION : L.act),
          round(L.round_out != 0 && L.type != K_ATTENTION_LAYER && !late_activation(L)) {
        if (T.slices > 1u) {      // the sums of a part of k, as they are
            ldc = (T.tile_h + 3u) & ~3u;
            out = T.part + (size_t)T.slice * tile_w * ldc;
            bias = nullptr; act = NO_ACTIVATION; round = false;
        }
    }
    __device__ __forceinline__ void operator()(unsigned mi, unsigned ni, const float *v) const {
        const unsigned m = m0 + mi, n = n0 + ni;
        if (n >= tile_w || m >= tile_h) return;
        float r[4];
        #pragma unroll
        for (unsigned j = 0; j < 4; j++) {
            float x = v[j];
            if (bias && m + j < tile_h) x += __ldg(bias + pos_h + m + j);
            if (act == RELU) x = x > 0.f ? x : 0.f;
            if (round) x = tf32_round(x);
            r[j] = x;
        }
        float *o = out + (size_t)n * ldc + m;
        if (m + 4u <= tile_h && (reinterpret_cast<uintptr_t>(o) & 15u) == 0u) *reinterpret_cast<float4 *>(o) = make_float4(r[0], r[1], r[2], r[3]);
        else
            #pragma unroll
            for (unsigned j = 0; j < 4; j++) if (m + j < tile_h) o[j] = r[j];
    }
};
struct WorkerBarrier { __device__ __forceinline__ void operator()() const { worker_barrier(fmablk::THREADS); } };

template <typename S, template <int> class W, template <int> class X>
static __device__ __noinline__ void ffma_blocks(const LayerDev &L, const TileDev &T, unsigned tid, unsigned char *scratch) {
    const GemmView g = gemm_view(L, T);
    const bool is_k = L.type == K_ATTENTION_LAYER, weights = !is_k && L.type != V_ATTENTION_LAYER;
    for (unsigned n0 = 0; n0 < T.tile_w; n0 += S::BN)
        for (unsigned m0 = 0; m0 < T.tile_h; m0 += S::BM) {
            GemmView b = g;
            b.wbase += g.w_transposed ? (size_t)m0 : (size_t)m0 * g.wld;
            if (!g.conv) b.xbase += (size_t)n0 * g.xld;
            const unsigned k1 = min(g.K, T.k1);
            b.K = k1;
            W<S::RW> lw(b, T.tile_h - m0, T.k1 >= g.K && weights ? L.Kpad : k1);
            X<S::RX> lx(L, b, T.pos_w + n0, T.tile_w - n0);
            StoreTile out(L, T, m0, n0);
            fmablk::block<S>(scratch, tid, k1, lw, lx, WorkerBarrier(), out, T.k0);
        }
}
template <typename S>
static __device__ __forceinline__ void ffma_shape(const LayerDev &L, const TileDev &T, unsigned tid, unsigned char *scratch) {
    if (L.type == CONV_LAYER || L.type == FC_LAYER) ffma_blocks<S, WeightRows, PixelRows>(L, T, tid, scratch);
    else ffma_blocks<S, WeightRows, TokenRows>(L, T, tid, scratch);
}

// A layer of at most 8 columns (the connected layers and the classifier of one image, a few tokens) reads its weights once and does
// next to nothing else: a warp takes a weight row, its lanes stride over k with eight 16-byte loads in flight, the dot
// products end in a warp reduction.  As an MMA tile the 256 x 4096 layer of the CIFAR net took 23 us for its one column, in
// chunks of 0.19 us one after the other on 8 SMs; as dot products of 16 rows on 32 tiles of eight warps, two rows each, 3.6 us,
// and the net's pass 95 -> 73 us.  Products and sums are fp32.
template <int N>
static __device__ __noinline__ void gemv_columns(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned warp = tid >> 5, lane = tid & 31u, nwarp = nthr >> 5, tile_h = T.tile_h, tile_w = T.tile_w, K = L.K;
    const size_t wld = L.Kpad, xld = L.x_ld, ldc = L.ldc;
    const float *weight = L.weight + (size_t)T.pos_h * wld, *in = L.in0 + (size_t)T.pos_w * xld, *bias = L.bias ? L.bias + T.pos_h : nullptr;
    float *out = L.out + (size_t)T.pos_w * ldc + T.pos_h;
    const int act = L.act;
    const bool round = L.round_out != 0;
    constexpr int U = N <= 4 ? 8 : 4;
    for (unsigned m = warp; m < tile_h; m += nwarp) {
        const float *w = weight + (size_t)m * wld;
        float acc[N];
        #pragma unroll
        for (int n = 0; n < N; n++) acc[n] = 0.f;
        for (unsigned k0 = lane * 4u; k0 < K; k0 += U * 128u) {
            float4 wv[U];
            #pragma unroll
            for (int u = 0; u < U; u++) wv[u] = k0 + u * 128u < K ? __ldg(reinterpret_cast<const float4 *>(w + k0 + u * 128u)) : make_float4(0.f, 0.f, 0.f, 0.f);
            #pragma unroll
            for (int n = 0; n < N; n++) {
                const float *x = in + (size_t)min((unsigned)n, tile_w - 1u) * xld + k0;
                #pragma unroll
                for (int u = 0; u < U; u++) {
                    const float4 xv = k0 + u * 128u < K ? ldcg4(x + u * 128u) : make_float4(0.f, 0.f, 0.f, 0.f);
                    acc[n] = fmaf(wv[u].x, xv.x, acc[n]); acc[n] = fmaf(wv[u].y, xv.y, acc[n]);
                    acc[n] = fmaf(wv[u].z, xv.z, acc[n]); acc[n] = fmaf(wv[u].w, xv.w, acc[n]);
                }
            }
        }
        float mine = 0.f;
        #pragma unroll
        for (int n = 0; n < N; n++) {
            acc[n] = warp_sum(acc[n]);
            if ((int)lane == n) mine = acc[n];
        }
        if (lane < tile_w) {
            mine = activate(mine + (bias ? __ldg(bias + m) : 0.f), act);
            out[(size_t)lane * ldc + m] = round ? tf32_round(mine) : mine;
        }
    }
}
static __device__ __forceinline__ void tile_gemv(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    if (T.tile_w == 1u) gemv_columns<1>(L, T, tid, nthr);
    else if (T.tile_w == 2u) gemv_columns<2>(L, T, tid, nthr);
    else if (T.tile_w <= 4u) gemv_columns<4>(L, T, tid, nthr);
    else gemv_columns<8>(L, T, tid, nthr);
}

// A tile that sums a part of k has stored its sums: whether it is the last one of its set.  All worker threads.
__device__ __forceinline__ bool arrives_last(const TileDev &T, unsigned tid, unsigned nthr, unsigned *last) {
    worker_barrier(nthr);
    if (tid == 0) {
        asm volatile("fence.acq_rel.gpu;" ::: "memory");        // release: the sums, through the barrier
        const unsigned before = atomicAdd(T.arrived, 1u);
        asm volatile("fence.acq_rel.gpu;" ::: "memory");        // acquire: the others'
        *(volatile unsigned *)last = before % T.slices == T.slices - 1u ? 1u : 0u;
    }
    worker_barrier(nthr);
    return *(volatile unsigned *)last != 0u;
}
// The parts' sums added in order (so a run's bits do not depend on which tile came last), bias, activation and store.  fp32 mode: nothing is
// rounded to TF32.
static __device__ __noinline__ void finish_parts(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr) {
    const unsigned tile_h = T.tile_h, h4 = (tile_h + 3u) >> 2, total = T.tile_w * h4, slices = T.slices;
    const size_t step = (size_t)T.tile_w * h4 * 4u;
    const float *part = T.part, *bias = L.bias ? L.bias + T.pos_h : nullptr;
    float *out = L.out + (size_t)T.pos_w * L.ldc + T.pos_h;
    const size_t ldc = L.ldc;
    const bool late = late_activation(L), relu = !late && L.act == RELU;
    for (unsigned i = tid; i < total; i += nthr) {
        const unsigned n = i / h4, m = (i - n * h4) * 4u;
        float4 a[8];
        #pragma unroll
        for (unsigned s = 0; s < 8; s++) a[s] = ldcg4(part + min(s, slices - 1u) * step + (size_t)i * 4u);
        float f[4] = {a[0].x, a[0].y, a[0].z, a[0].w};
        #pragma unroll
        for (unsigned s = 1; s < 8; s++)
            if (s < slices) { f[0] += a[s].x; f[1] += a[s].y; f[2] += a[s].z; f[3] += a[s].w; }
        float *o = out + (size_t)n * ldc + m;
        #pragma unroll
        for (unsigned j = 0; j < 4; j++) {
            if (bias && m + j < tile_h) f[j] += __ldg(bias + m + j);
            if (relu) f[j] = f[j] > 0.f ? f[j] : 0.f;
        }
        if (m + 4u <= tile_h && (reinterpret_cast<uintptr_t>(o) & 15u) == 0u) *reinterpret_cast<float4 *>(o) = make_float4(f[0], f[1], f[2], f[3]);
        else
            #pragma unroll
            for (unsigned j = 0; j < 4; j++) if (m + j < tile_h) o[j] = f[j];
    }
    if (late) worker_barrier(nthr);
}

// Tile in fp32 (ref src/tiled_kernels.c:21-490, 784-1038).  FULL: the fp32 mode, 96 KB of staging; the shape of the blocks
// follows the tile (a shape larger than the tile would compute padding).  Otherwise the few layers of a tensor-core graph without an
// operand form: scores of heads that are no multiple of four features or of more than 512 keys, values of such heads, convolutions
// past an im2col map's limits.
template <bool FULL>
static __device__ void tile_gemm_ffma(const LayerDev &L, const TileDev &T, unsigned tid, unsigned nthr, unsigned char *scratch, unsigned *last) {
    if (L.gemv) { tile_gemv(L, T, tid, nthr); return; }
    const bool pieces = L.a_vec4 != 0 && L.type != V_ATTENTION_LAYER;
    if (!FULL) {
        // The staging is the epilogue's transposing buffers, one per warp: a warp may still be storing the tensor-core tile before when
        // another comes here, and the warps have met since (worker_loop).
        if (pieces) ffma_shape<fmablk::Tight>(L, T, tid, scratch);
        else ffma_blocks<fmablk::Tight, AnyWeightRows, AnyRows>(L, T, tid, scratch);
    } else if (!pieces) ffma_blocks<fmablk::Small, AnyWeightRows, AnyRows>(L, T, tid, scratch);
    else if (T.tile_h > 64 && T.tile_w > 32) ffma_shape<fmablk::Large>(L, T, tid, scratch);
    else if (T.tile_h > 32 && T.tile_w > 32) ffma_shape<fmablk::Medium>(L, T, tid, scratch);
    else ffma_shape<fmablk::Small>(L, T, tid, scratch);
    const unsigned tile_h = T.tile_h, tile_w = T.tile_w;
    if (T.slices > 1u) {
        if (!arrives_last(T, tid, nthr, last)) return;
        finish_parts(L, T, tid, nthr);
    }
    float *tile = L.out + (size_t)T.pos_w * L.ldc + T.pos_h;
    if (L.type == K_ATTENTION_LAYER) {
        // mask, / sqrt(hd), exp, every column normalised by its sum (no max subtraction, as the reference)
        const unsigned warp = tid >> 5, lane = tid & 31, nwarp = nthr >> 5, q0 = T.pos_w % L.seq;
        const float scale = sqrtf((float)L.hd);
        for (unsigned n = warp; n < tile_w; n += nwarp) {
            float *o = tile + (size_t)n * L.ldc, s = 0.f;
            for (unsigned m = lane; m < tile_h; m += 32) {
                const float x = L.masked && T.pos_h + m > q0 + n ? -1e10f : ldcg1(o + m);
                s += o[m] = expf(x / scale);
            }
            s = warp_sum(s);
            for (unsigned m = lane; m < tile_h; m += 32) o[m] = store_round(o[m] / s, L);
        }
    } else if (late_activation(L)) {
        const int act = L.act;
        const size_t ldc = L.ldc;
        for (unsigned i = tid; i < tile_w * tile_h; i += nthr) {
            float *o = tile + (size_t)(i / tile_h) * ldc + i % tile_h;
            *o = store_round(activate(ldcg1(o), act), L);
        }
    }
}
