// Contraction tiles on the 5th-generation tensor cores (sm_100a): conv, matmul, connected,
// K-attention and V-attention ninst tiles as TF32 tcgen05.mma with fp32 accumulators in TMEM.
//
// Orientation.  A ninst tile is out[column n][row m] (n: pixels / tokens, m: channels / keys /
// features, m contiguous in memory).  The MMA is issued as D[128 x N] with
//     MMA-M (128 TMEM lanes)  <- 128 consecutive tile columns n   (operand "X": activations)
//     MMA-N (<=256 TMEM cols) <- tile rows m                      (operand "W": weights / keys / V)
// so an accumulator lane is one output column n.  The epilogue transposes 32 x 32 pieces through shared memory, after which
// consecutive lanes store consecutive m; the K-attention softmax (a reduction over m) sums a lane's own column, half of the
// pieces in each of the two warps of a query quarter.
//
// Roles.  A tile is a sequence of 128 x (<= 256) blocks, and four kinds of warps walk the same sequence, each at its own pace
// and across tile boundaries; nothing but mbarriers connects them:
//     warp A, warp B   TMA boxes of the X / W operand into a ring of stages (32 fp32 of k a chunk, up to four chunks a stage)
//     warp MMA         four tcgen05.mma (k = 8 each) per chunk, accumulators alternate between two halves of TMEM
//     8 worker warps   epilogue: TMEM -> registers -> bias, activation, residual add, softmax -> memory; they also run the
//                      memory-bound tiles
// so the operands of the next block (or of the next tile, once the scheduler has posted one) stream in and are multiplied
// while the previous block is written out.
// What bounds the k loop.  The instruction streams of the three issuing warps, for narrow tiles: issued from one lane's own branch a
// wait and a box take 0.17 us whatever the box holds, since TMA and MMA take their operands from uniform registers and a value of one
// lane has to be brought there each time.  So the whole warp walks with values that the compiler knows to be uniform, and one lane
// issues (BERT 1 x 37 875 -> 799 us a pass, ResNet-50 + VGG-16 x 16 1859 -> 1719, ResNet-50 x 32 1465 -> 1398); two warps feed
// the ring, narrow tiles take several chunks a stage, and the loops hold no division.  A chunk of a block of 256 rows takes
// 0.30 - 0.37 us (all SMs at work, operands in L2), the rate of the measured dense TF32 peak.
//
// Staging.  Both operands are K-major, 32 fp32 (128 bytes) per row and k-chunk, in the 128-byte swizzled shared-memory
// layout UMMA descriptors and TMA share.  A narrow layer (few tokens, few pixels) stages only the columns it has; the MMA reads
// 128 rows all the same, whatever lies there: those accumulator lanes have no reader.  The ring is cut into stages of four
// chunks for tiles of up to 64 rows (2 stages of 96 KB), two up to 128 (3 of 64 KB), one above (4 of 48 KB); when the cut
// changes between two tiles both producers first wait until the old stages have been read.
//
// Every wait is bounded: when a time budget runs out the thread records an error and raises the abort flag, every role
// leaves its loop, producers let their copies land, and the CTA frees its TMEM and exits.  (The workers' barriers: worker_loop.h.)
#pragma once
#include "tiles_simt.cuh"

namespace tc {

constexpr unsigned MAX_STAGES = 8;
constexpr unsigned RING_BYTES = 192u * 1024u;
constexpr unsigned NW = 256;                       // worker threads
constexpr unsigned WARP_A = 0, WARP_MMA = 1, WARP_SCHED = 2, WARP_B = 3, WARP_WORK = 4;   // workers: warps 4 .. 11 (warp % 4 = TMEM lane quarter)
constexpr unsigned THREADS = 128 + NW;
constexpr unsigned TMEM_COLS = 512;
constexpr unsigned BLOCK_ROWS = 256;               // rows m of a block: one half of TMEM
constexpr unsigned EPI_BYTES = (NW / 32) * 4096;   // a 4 KB transposing buffer per worker warp
constexpr unsigned SLOTS = 4;                      // ring of posted tiles

// A posted tile: everything the roles need, so none of them waits for a load from global memory.
struct Slot {
    LayerDev layer;
    TileDev tile;
    unsigned live, nasm;                           // live 0: leave
    const unsigned char *maps;                     // the graph's tensor maps
    const InputDev *input;
};

// What the scheduler needs of a graph to hand out and retire its tiles; the first ones of a launch are kept in shared memory,
// which takes an L2 round trip off both.
struct GraphRef {
    const LayerDev *layers;
    const TileDev *tiles;
    const uint2 *children;
    unsigned *dep;
    const unsigned char *maps;
    const InputDev *input;
    unsigned *svc;
    unsigned n_exec;
};
constexpr unsigned CACHED_GRAPHS = 12;

struct Shared {
    GraphRef graphs[CACHED_GRAPHS];
    unsigned long long full[MAX_STAGES], empty[MAX_STAGES];    // stage filled (both producers) / read by the MMAs
    unsigned long long acc_full[2], acc_empty[2];              // accumulator half complete / read by the workers
    unsigned long long posted[SLOTS], finished[SLOTS];         // scheduler -> roles: the slot is filled / roles -> scheduler
    unsigned long long fed[SLOTS];                             // W producer -> scheduler: the tile's last box is on its way
    unsigned long long ready[SLOTS];                           // scheduler -> roles: the tile's parents are complete
    unsigned long long prof_mark;                              // time accounting: when the workers' last step ended
    unsigned tmem_base;
    unsigned last;                                             // the workers' tile is the last of its set (arrives_last)
    Slot slots[SLOTS];
};
static_assert(sizeof(Shared) <= 3072, "Shared must fit beside the ring");

// ---- PTX wrappers ----------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    unsigned one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0u;
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Non-blocking probe (try_wait may suspend the thread for a hardware-defined time; a polling loop
// that has other things to look at uses this one).
__device__ __forceinline__ bool mbar_test_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false (and marks the run aborted) when the time budget runs out.  The one-thread roles are bound by the
// length of their instruction stream, so the common case is four instructions; clock, budget and abort flag are only looked at
// after some ten thousand try_waits (each suspends the thread for a while in hardware), out of the loop's way.
__device__ __forceinline__ bool mbar_wait_slow(unsigned long long *bar, unsigned parity, CtrlDev *ctrl, StatusHost *status, unsigned where) {
    unsigned long long t0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    const unsigned long long budget = ctrl->pipe_ns;
    for (unsigned spin = 1;; spin++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 0u) {
            if (*(volatile unsigned *)&ctrl->abort) return false;
            unsigned long long now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (now - t0 > budget) break;
        }
    }
    if (atomicCAS(&ctrl->abort, 0u, (unsigned)ASPEN_B200_ERR_PIPE) == 0u) {
        status->info0 = where;
        status->info1 = blockIdx.x;
        status->status = ASPEN_B200_ERR_PIPE;
        __threadfence_system();
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, CtrlDev *ctrl, StatusHost *status, unsigned where) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u32 c;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "@p bra DONE;\n\t"
                 "mov.u32 c, 0;\n"
                 "AGAIN:\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "@p bra DONE;\n\t"
                 "add.u32 c, c, 1;\n\t"
                 "setp.lt.u32 q, c, 10000;\n\t"
                 "@q bra AGAIN;\n"
                 "DONE:\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (__builtin_expect(ok != 0u, 1)) return true;
    return mbar_wait_slow(bar, parity, ctrl, status, where);
}

// A role's wait for the next tile (Shared::posted) or for its parents (Shared::ready).  The scheduler always posts an exit marker
// eventually (end of run, stop, stall, abort); the time bound only guards against that logic failing.
__device__ __forceinline__ bool wait_slot(unsigned long long *bar, unsigned parity, CtrlDev *ctrl, StatusHost *status) {
    #pragma unroll 1
    for (unsigned spin = 0; spin < 1024u; spin++)
        if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    const unsigned long long budget = 2ull * ctrl->stall_ns + 4ull * ctrl->pipe_ns + 1000000000ull;
    for (unsigned spin = 1;; spin++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 63u) == 0u) {
            __nanosleep(64);
            unsigned long long now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (now - t0 > budget) break;
        }
    }
    if (atomicCAS(&ctrl->abort, 0u, (unsigned)ASPEN_B200_ERR_PIPE) == 0u) {
        status->info0 = 7; status->info1 = blockIdx.x; status->status = ASPEN_B200_ERR_PIPE;
        __threadfence_system();
    }
    return false;
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(unsigned dst, const void *tmap, int x, int y, unsigned long long *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tma_load_3d(unsigned dst, const void *tmap, int x, int y, int z, unsigned long long *bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

// 128 (box) output pixels from (x, y, sample n) on, 32 channels from c on, of the tap (kw, kh); coordinates are input pixels
__device__ __forceinline__ void tma_load_im2col(unsigned dst, const void *tmap, int c, int x, int y, int n, unsigned kw, unsigned kh, unsigned long long *bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6], {%7, %8};"
                 ::"r"(dst), "l"(tmap), "r"(c), "r"(x), "r"(y), "r"(n), "r"(smem_u32(bar)), "h"((unsigned short)kw), "h"((unsigned short)kh) : "memory");
}

__device__ __forceinline__ void tmem_alloc(unsigned *holder, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(unsigned long long *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// K-major, 128-byte swizzle, 8-row groups 1024 bytes apart; version 1 (sm_100) in bits 46-47.  Only the low word, which holds
// the address, changes: leading byte offset (unused for swizzled K-major) in bits 16-29.
constexpr unsigned UMMA_DESC_HIGH = (1024u >> 4) | 1u << 14 | 2u << 29;
__device__ __forceinline__ unsigned umma_desc_low(unsigned smem_addr) { return (smem_addr >> 4) | 1u << 16; }
// The four k = 8 steps of one stage.
__device__ __forceinline__ void tc_mma_stage(unsigned d_tmem, unsigned alow, unsigned blow, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n\t.reg .pred p, t;\n\t.reg .b64 a, b;\n\t.reg .b32 al, bl;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, %4, %4;\n\t"
                 "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, p;\n\t"
                 "add.u32 al, %1, 2;\n\tadd.u32 bl, %2, 2;\n\tmov.b64 a, {al, %5};\n\tmov.b64 b, {bl, %5};\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, t;\n\t"
                 "add.u32 al, %1, 4;\n\tadd.u32 bl, %2, 4;\n\tmov.b64 a, {al, %5};\n\tmov.b64 b, {bl, %5};\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, t;\n\t"
                 "add.u32 al, %1, 6;\n\tadd.u32 bl, %2, 6;\n\tmov.b64 a, {al, %5};\n\tmov.b64 b, {bl, %5};\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, t;\n\t}"
                 ::"r"(d_tmem), "r"(alow), "r"(blow), "r"(idesc), "r"(accumulate), "r"(UMMA_DESC_HIGH) : "memory");
}
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float *v) {
    unsigned *r = reinterpret_cast<unsigned *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_st32(unsigned taddr, const float *v) {
    const unsigned *r = reinterpret_cast<const unsigned *>(v);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// D fp32, A/B tf32, both K-major, M = 128, N = n.
__device__ __forceinline__ unsigned umma_idesc(unsigned n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}



// How the X operand of a layer reaches shared memory (chosen on the host, LayerDev::a_kind):
//   A_TMA      boxes straight from the parent's [columns][rows] matrix: matmul, 1x1 stride-1 convolution, attention, connected
//              layers over an unpadded parent.  One box per k-chunk, or per stage where the map has the chunk as a third dimension
//   A_IM2COL   any other convolution: TMA im2col boxes.  The parent is a (channel, iw, ih, sample) tensor; one chunk is 32
//              channels of one tap for 128 consecutive output pixels, wherever they cross the end of an image row or of a
//              sample; taps outside the image and channels past the last arrive as zeros (the weights hold every tap in whole
//              chunks).  No im2col matrix exists.  A connected layer over padded columns is a window as large as its image.
//              A convolution on an image of at most 4 channels (the 7x7 stem) reads a zero-padded [sample][row][pixel][4] copy of
//              it: a row of the window is 4 * KW consecutive floats there, the tensor's columns are the output's (a stride apart,
//              overlapping), and KH rows of 28 floats take 7 chunks where 49 taps of 3 channels would take 49.
//   A_HEAD     attention scores with heads that are no multiple of 32 features: the parent is a (feature, head, column) tensor for
//              queries and keys alike, one box per k-chunk, zeros past the head's last feature
// The W operand -- weights, attention keys (PARENT_1's matrix) or the transposed copy of the attention values -- arrives in one
// box per stage.  Layers that fit none of these run as fp32 FMA tiles (tile_gemm_ffma).

// Box coordinates of column 0 / row 0 of a tile (x in chunks of 32), and, for attention values behind a causal mask, the keys its
// first block of queries can see: the probabilities after them are zeros and are not multiplied.
struct Origin {
    int ax, ay, bx, by;
    unsigned seen;
    __device__ __forceinline__ unsigned chunks(unsigned all, unsigned n0) const { return seen ? min(all, (seen + n0 + 31u) >> 5) : all; }
};

__device__ __forceinline__ Origin origin(const LayerDev &L, const TileDev &T) {
    Origin g;
    g.ax = 0; g.ay = (int)T.pos_w; g.bx = 0; g.by = (int)T.pos_h; g.seen = 0;
    if (L.type == K_ATTENTION_LAYER) {
        const unsigned per = L.seq * L.heads, b = T.pos_w / per, r = T.pos_w - b * per, head = r / L.seq, q0 = r - head * L.seq;
        g.ax = g.bx = (int)(L.a_kind == A_HEAD ? head : head * (L.hd >> 5));
        g.ay = (int)(b * L.seq + q0); g.by = (int)(b * L.seq + T.pos_h);
    } else if (L.type == V_ATTENTION_LAYER) {
        const unsigned b = T.pos_w / L.seq, head = T.pos_h / L.hd, q0 = T.pos_w - b * L.seq;
        g.ay = (int)((b * L.heads + head) * L.seq + q0);
        g.bx = (int)(b * (L.vt_seq >> 5));
        if (L.masked) g.seen = q0 + 128u;
    }
    return g;
}

// A value that all lanes of a converged warp hold: the compiler keeps what is computed from it in uniform registers, where the operands of
// TMA and MMA instructions have to be.
__device__ __forceinline__ unsigned uniform(unsigned v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
template <typename T>
__device__ __forceinline__ const T *uniform(const T *p) { return reinterpret_cast<const T *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), 0)); }
__device__ __forceinline__ Origin uniform(const Origin &g) {
    Origin u;
    u.ax = uniform(g.ax); u.ay = uniform(g.ay); u.bx = uniform(g.bx); u.by = uniform(g.by); u.seen = uniform(g.seen);
    return u;
}

// Ring position of one role.  `uses` holds, per stage, the parity of the number of times this role has used it.
struct Ring {
    unsigned s = 0, uses = 0, stage_bytes = 0, stages = 1;
    __device__ __forceinline__ void step() { uses ^= 1u << s; if (++s == stages) s = 0; }
    __device__ __forceinline__ unsigned parity() const { return (uses >> s) & 1u; }
};

// A wait of a whole warp: its lanes give up together.
__device__ __forceinline__ bool warp_wait(unsigned long long *bar, unsigned parity, CtrlDev *ctrl, StatusHost *status, unsigned where) {
    #pragma unroll 1
    for (unsigned tries = 0; tries < 10000u; tries++)
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait_slow(bar, parity, ctrl, status, where));
}

// Producer side of a change of the ring's cut: every stage must have been read.
__device__ __forceinline__ bool recut(Ring &r, const LayerDev &L, Shared *sh, CtrlDev *ctrl, StatusHost *status) {
    const unsigned stage_bytes = uniform(L.stage_bytes);
    if (stage_bytes == r.stage_bytes) return true;
    if (r.stage_bytes)
        for (unsigned i = 0; i < r.stages; i++)
            if (!warp_wait(&sh->empty[i], ((r.uses >> i) & 1u) ^ 1u, ctrl, status, 8)) return false;
    r.s = 0; r.stage_bytes = stage_bytes; r.stages = uniform((unsigned)L.stages);
    return true;
}

// The slot's parents are complete (false: gave up, or the scheduler has withdrawn the tile).
__device__ __forceinline__ bool wait_ready(const Slot &sl, unsigned long long *ready, unsigned parity, CtrlDev *ctrl, StatusHost *status) {
    return __all_sync(0xffffffffu, wait_slot(ready, parity, ctrl, status) && sl.live != 0u);
}

// The three roles below are one warp each: all lanes walk, and one (the same one each time) issues.
// ---- X operand producer -----------------------------------------------------------------------------------------------
__device__ __forceinline__ bool produce_a(const Slot &sl, unsigned long long *ready, unsigned ready_parity, unsigned ring, Ring &r, Shared *sh, CtrlDev *ctrl,
                                          StatusHost *status) {
    const LayerDev &L = sl.layer;
    const Origin g = uniform(origin(L, sl.tile));
    const unsigned char *map = uniform(sl.maps + (size_t)L.amap * 128);
    if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    if (!recut(r, L, sh, ctrl, status) || !wait_ready(sl, ready, ready_parity, ctrl, status)) return false;
    // activations were written with ordinary (generic proxy) stores; TMA reads them through the async proxy
    asm volatile("fence.proxy.async.global;" ::: "memory");
    const unsigned kind = uniform((unsigned)L.a_kind), tile_w = uniform(sl.tile.tile_w), tile_h = uniform(sl.tile.tile_h), per = uniform((unsigned)L.per_stage),
                   chunk_bytes = uniform((unsigned)L.a_rows) * 128u;
    if (kind == A_IM2COL) {
        const unsigned pos_w = uniform(sl.tile.pos_w), OW = uniform(L.OW), hw = uniform(L.OH) * OW, KW = uniform((unsigned)L.tap_kw), C = uniform(L.tap_c),
                       sx = uniform((unsigned)L.tap_sx), sy = uniform((unsigned)L.tap_sy), chunks = uniform(L.chunks);
        const int pad = (int)uniform((unsigned)L.tap_pad);
        for (unsigned n0 = 0; n0 < tile_w; n0 += 128u) {
            const unsigned n = pos_w + n0, pn = n / hw, q = n - pn * hw, py = q / OW, px = q - py * OW;      // first output pixel of the block
            const int x0 = (int)(px * sx) - pad, y0 = (int)(py * sy) - pad;
            for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS) {
                unsigned kh = 0, kw = 0, c = 0;      // tap and first channel of the next chunk; c runs fastest
                for (unsigned ch = 0; ch < chunks; ch += per) {
                    const unsigned count = min(per, chunks - ch);
                    unsigned dst = ring + r.s * r.stage_bytes;
                    if (!warp_wait(&sh->empty[r.s], r.parity() ^ 1u, ctrl, status, 2)) return false;
                    const bool issue = elect_one();
                    if (issue) mbar_arrive_expect_tx(&sh->full[r.s], count * chunk_bytes);
                    for (unsigned j = 0; j < count; j++, dst += chunk_bytes) {
                        if (issue) tma_load_im2col(dst, map, (int)c, x0, y0, (int)pn, kw, kh, &sh->full[r.s]);
                        c += 32u;
                        if (c == C) { c = 0; if (++kw == KW) { kw = 0; kh++; } }
                    }
                    r.step();
                }
            }
        }
        return true;
    }
    const bool multi = uniform((unsigned)L.a_multi) != 0u;
    const unsigned all_chunks = uniform(L.chunks);
    for (unsigned n0 = 0; n0 < tile_w; n0 += 128u) {
        const unsigned chunks = g.chunks(all_chunks, n0);
        const int y = g.ay + (int)n0;
        for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS) {
            if (multi) {
                for (unsigned ch = 0; ch < chunks; ch += per) {
                    if (!warp_wait(&sh->empty[r.s], r.parity() ^ 1u, ctrl, status, 2)) return false;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&sh->full[r.s], per * chunk_bytes);
                        tma_load_3d(ring + r.s * r.stage_bytes, map, 0, y, g.ax + (int)ch, &sh->full[r.s]);
                    }
                    r.step();
                }
                continue;
            }
            for (unsigned ch = 0; ch < chunks; ch += per) {
                const unsigned count = min(per, chunks - ch);
                unsigned dst = ring + r.s * r.stage_bytes;
                if (!warp_wait(&sh->empty[r.s], r.parity() ^ 1u, ctrl, status, 2)) return false;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh->full[r.s], count * chunk_bytes);
                    for (unsigned j = 0; j < count; j++, dst += chunk_bytes) {
                        if (kind == A_HEAD) tma_load_3d(dst, map, (int)(ch + j) * 32, g.ax, y, &sh->full[r.s]);
                        else tma_load_2d(dst, map, (g.ax + (int)(ch + j)) * 32, y, &sh->full[r.s]);
                    }
                }
                r.step();
            }
        }
    }
    return true;
}

// ---- W operand producer -----------------------------------------------------------------------------------------------
// Weights depend on no parent: a tile's first stages are filled while it still waits for them.  A stage beyond the ring's is
// free only after the tile's own MMAs, so its (shorter bounded) wait starts behind the parents'.
__device__ __forceinline__ bool produce_b(const Slot &sl, unsigned long long *ready, unsigned ready_parity, unsigned ring, Ring &r, Shared *sh, CtrlDev *ctrl,
                                          StatusHost *status) {
    const LayerDev &L = sl.layer;
    const Origin g = uniform(origin(L, sl.tile));
    const unsigned char *map = uniform(sl.maps + (size_t)L.wmap * 128);
    if (!recut(r, L, sh, ctrl, status)) return false;
    unsigned lead = r.stages;
    if (L.type == K_ATTENTION_LAYER || L.type == V_ATTENTION_LAYER) {
        if (!wait_ready(sl, ready, ready_parity, ctrl, status)) return false;
        asm volatile("fence.proxy.async.global;" ::: "memory");
        lead = ~0u;
    }
    const unsigned tile_w = uniform(sl.tile.tile_w), tile_h = uniform(sl.tile.tile_h), per = uniform((unsigned)L.per_stage), box = uniform((unsigned)L.b_rows) * 128u,
                   bytes = per * box, b_off = per * uniform((unsigned)L.a_rows) * 128u, all_chunks = uniform(L.chunks);
    if (L.a_kind == A_HEAD) {
        for (unsigned n0 = 0; n0 < tile_w; n0 += 128u)
            for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS)
                for (unsigned ch = 0; ch < all_chunks; ch += per) {
                    const unsigned n = min(per, all_chunks - ch);
                    if (!warp_wait(&sh->empty[r.s], r.parity() ^ 1u, ctrl, status, 9)) return false;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&sh->full[r.s], n * box);
                        for (unsigned j = 0; j < n; j++)
                            tma_load_3d(ring + r.s * r.stage_bytes + b_off + j * box, map, (int)(ch + j) * 32, g.bx, g.by + (int)mp, &sh->full[r.s]);
                    }
                    r.step();
                }
        return true;
    }
    for (unsigned n0 = 0; n0 < tile_w; n0 += 128u)
        for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS)
            for (unsigned ch = 0, chunks = g.chunks(all_chunks, n0); ch < chunks; ch += per) {
                if (lead-- == 0u && !wait_ready(sl, ready, ready_parity, ctrl, status)) return false;
                if (!warp_wait(&sh->empty[r.s], r.parity() ^ 1u, ctrl, status, 9)) return false;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh->full[r.s], bytes);
                    tma_load_3d(ring + r.s * r.stage_bytes + b_off, map, 0, g.by + (int)mp, g.bx + (int)ch, &sh->full[r.s]);
                }
                r.step();
            }
    return true;
}

// ---- MMA issuer -------------------------------------------------------------------------------------------------------
// `half`: accumulator half of the next block; `acc_uses`: parity of the uses of each half.
__device__ __forceinline__ bool issue_mma(const Slot &sl, unsigned ring, Ring &r, unsigned &half, unsigned &acc_uses, Shared *sh, CtrlDev *ctrl, StatusHost *status) {
    const LayerDev &L = sl.layer;
    const unsigned stage_bytes = uniform(L.stage_bytes);
    if (stage_bytes != r.stage_bytes) { r.s = 0; r.stage_bytes = stage_bytes; r.stages = uniform((unsigned)L.stages); }
    const unsigned tmem = uniform(sh->tmem_base), tile_w = uniform(sl.tile.tile_w), tile_h = uniform(sl.tile.tile_h), per = uniform((unsigned)L.per_stage);
    const Origin g = uniform(origin(L, sl.tile));
    const unsigned a_rows = uniform((unsigned)L.a_rows), b_rows = uniform((unsigned)L.b_rows), all_chunks = uniform(L.chunks);
    const unsigned b_off = per * a_rows * 128u, a_step = (a_rows * 128u) >> 4, b_step = (b_rows * 128u) >> 4;
    for (unsigned n0 = 0; n0 < tile_w; n0 += 128u)
        for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS) {
            const unsigned idesc = umma_idesc((min(BLOCK_ROWS, tile_h - mp) + 15u) & ~15u), d = tmem + half * BLOCK_ROWS;
            if (!warp_wait(&sh->acc_empty[half], ((acc_uses >> half) & 1u) ^ 1u, ctrl, status, 6)) return false;
            acc_uses ^= 1u << half;
            tc_fence_after();
            for (unsigned ch = 0, chunks = g.chunks(all_chunks, n0); ch < chunks; ch += per) {
                const unsigned n = min(per, chunks - ch), sA = ring + r.s * r.stage_bytes;
                unsigned alow = umma_desc_low(sA), blow = umma_desc_low(sA + b_off);
                if (!warp_wait(&sh->full[r.s], r.parity(), ctrl, status, 3)) return false;
                tc_fence_after();
                if (elect_one()) {
                    tc_mma_stage(d, alow, blow, idesc, ch);
                    for (unsigned j = 1; j < n; j++) {
                        alow += a_step;
                        blow += b_step;
                        tc_mma_stage(d, alow, blow, idesc, 1u);
                    }
                    tc_commit(&sh->empty[r.s]);
                    if (ch + per >= chunks) tc_commit(&sh->acc_full[half]);
                }
                r.step();
            }
            half ^= 1u;
        }
    return true;
}

// ---- worker warps: epilogue ---------------------------------------------------------------------------------------------
// A block is handled in 32 x 32 pieces (32 tile columns, one per lane, x 32 rows m).  tcgen05.ld gives a lane 32 consecutive m
// of ITS column, but global memory wants consecutive m from consecutive lanes, so a piece is transposed through a 4 KB
// buffer of the warp (XOR-swizzled 16-byte quads, conflict free both ways).  After that lane l holds rows 4 (l % 8) .. + 3 of
// the columns l / 8 + 4 i, i = 0 .. 7: bias (one 16-byte load for the piece), activation, residual add and rounding happen
// there, and every load or store instruction covers four full 128-byte lines.
struct Piece {
    float4 x[8];
};
__device__ __forceinline__ void transpose(float *stage, const float *v, Piece &p) {
    const unsigned lane = threadIdx.x & 31u, quad = lane & 7u, n0 = lane >> 3;
    float4 *st = reinterpret_cast<float4 *>(stage);
    #pragma unroll
    for (unsigned j = 0; j < 8; j++) st[lane * 8u + (j ^ (lane & 7u))] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    __syncwarp();
    #pragma unroll
    for (unsigned i = 0; i < 8; i++) p.x[i] = st[(i * 4u + n0) * 8u + (quad ^ ((i * 4u + n0) & 7u))];
    __syncwarp();
}
__device__ __forceinline__ void untranspose(float *stage, const Piece &p, float *v) {
    const unsigned lane = threadIdx.x & 31u, quad = lane & 7u, n0 = lane >> 3;
    float4 *st = reinterpret_cast<float4 *>(stage);
    #pragma unroll
    for (unsigned i = 0; i < 8; i++) st[(i * 4u + n0) * 8u + (quad ^ ((i * 4u + n0) & 7u))] = p.x[i];
    __syncwarp();
    #pragma unroll
    for (unsigned j = 0; j < 8; j++) {
        const float4 t = st[lane * 8u + (j ^ (lane & 7u))];
        v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
    }
    __syncwarp();
}
// Whole pieces (all 32 columns and rows exist) take a path without tests, so the eight loads or stores issue back to back.
__device__ __forceinline__ void store_piece(const Piece &p, float *out /*(n = 0, m = 0)*/, size_t ld, unsigned n_valid, unsigned m_valid) {
    const unsigned lane = threadIdx.x & 31u, m = (lane & 7u) * 4u, n0 = lane >> 3;
    float *dst = out + (size_t)n0 * ld + m;
    const size_t step = 4u * ld;
    if (n_valid == 32u && m_valid == 32u) {
        #pragma unroll
        for (unsigned i = 0; i < 8; i++) { *reinterpret_cast<float4 *>(dst) = p.x[i]; dst += step; }
    } else {
        #pragma unroll
        for (unsigned i = 0; i < 8; i++) {
            if (i * 4u + n0 < n_valid) {
                if (m + 4u <= m_valid) *reinterpret_cast<float4 *>(dst) = p.x[i];
                else {
                    if (m < m_valid) dst[0] = p.x[i].x;
                    if (m + 1u < m_valid) dst[1] = p.x[i].y;
                    if (m + 2u < m_valid) dst[2] = p.x[i].z;
                }
            }
            dst += step;
        }
    }
}
// The other operand of a fused residual add.  A warp asks for it two of its pieces ahead (the first ones before the
// accumulator is waited for), so it lands under the main loop or under the previous pieces' stores: one piece ahead measured
// 142 us for a 256 x 768 tile with k = 64 (every piece waits for HBM), two ahead 74, and 51 once rare activations had left the loop.
__device__ __forceinline__ void load_piece(Piece &p, const float *in, size_t ld, unsigned n_valid, unsigned m_valid) {
    const unsigned lane = threadIdx.x & 31u, m = (lane & 7u) * 4u, n0 = lane >> 3;
    const float *src = in + (size_t)n0 * ld + m;
    const size_t step = 4u * ld;
    if (n_valid == 32u && m_valid == 32u) {
        #pragma unroll
        for (unsigned i = 0; i < 8; i++) { p.x[i] = ldcg4(src); src += step; }
    } else {
        #pragma unroll
        for (unsigned i = 0; i < 8; i++) {
            p.x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i * 4u + n0 < n_valid) {
                if (m + 4u <= m_valid) p.x[i] = ldcg4(src);
                else {
                    if (m < m_valid) p.x[i].x = ldcg1(src);
                    if (m + 1u < m_valid) p.x[i].y = ldcg1(src + 1);
                    if (m + 2u < m_valid) p.x[i].z = ldcg1(src + 2);
                }
            }
            src += step;
        }
    }
}
// bias of this lane's four rows, m = first of them, `valid` rows exist from there
__device__ __forceinline__ float4 load_bias(const float *bias, int valid) {
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) {
        if (valid >= 4 && (reinterpret_cast<uintptr_t>(bias) & 15u) == 0u) b = __ldg(reinterpret_cast<const float4 *>(bias));
        else {
            if (valid > 0) b.x = __ldg(bias);
            if (valid > 1) b.y = __ldg(bias + 1);
            if (valid > 2) b.z = __ldg(bias + 2);
            if (valid > 3) b.w = __ldg(bias + 3);
        }
    }
    return b;
}
__device__ __forceinline__ void round_piece(Piece &p) {
    #pragma unroll
    for (unsigned i = 0; i < 8; i++) { p.x[i].x = tf32_round(p.x[i].x); p.x[i].y = tf32_round(p.x[i].y); p.x[i].z = tf32_round(p.x[i].z); p.x[i].w = tf32_round(p.x[i].w); }
}

// Activations of the tensor-core epilogue.  ReLU, leaky ReLU and the two GELUs are branch-free single precision on the registers.
__device__ __forceinline__ float act_inline(float x, int act) {
    switch (act) {
        case RELU: return fmaxf(x, 0.f);
        case GELU: return gelu_erf_fast(x);
        case GELU_ACCURATE: return gelu_tanh_fast(x);
        default: return x > 0.f ? x : fmaf(x, 0.1f, x * (float)(0.1 - (double)0.1f));   // LEAKY_RELU: 0.1 in two parts, rounded once
    }
}
template <int ACT>
__device__ __forceinline__ void act_piece(Piece &p) {
    #pragma unroll
    for (unsigned i = 0; i < 8; i++) {
        p.x[i].x = act_inline(p.x[i].x, ACT); p.x[i].y = act_inline(p.x[i].y, ACT); p.x[i].z = act_inline(p.x[i].z, ACT); p.x[i].w = act_inline(p.x[i].w, ACT);
    }
}
// The others are the reference's double-precision forms (`activate`): in single precision exp(x) - 1 cancels.  Their code once, in a
// loop over the lane's 32 values in its warp's buffer: inlined for each value it would be many times the instruction cache.
static __device__ __noinline__ void act_buffer(float *mine, int act) {
    #pragma unroll 1
    for (unsigned e = 0; e < 32; e++) mine[e * 32u] = activate(mine[e * 32u], act);
}
__device__ __forceinline__ void activate_piece(Piece &p, int act, float *stage) {
    switch (act) {
        case NO_ACTIVATION: case LINEAR: break;
        case RELU: act_piece<RELU>(p); break;
        case GELU: act_piece<GELU>(p); break;
        case GELU_ACCURATE: act_piece<GELU_ACCURATE>(p); break;
        case LEAKY_RELU: act_piece<LEAKY_RELU>(p); break;
        default: {
            float *mine = stage + (threadIdx.x & 31u);
            #pragma unroll
            for (unsigned i = 0; i < 8; i++) { mine[i * 128u] = p.x[i].x; mine[i * 128u + 32u] = p.x[i].y; mine[i * 128u + 64u] = p.x[i].z; mine[i * 128u + 96u] = p.x[i].w; }
            act_buffer(mine, act);
            #pragma unroll
            for (unsigned i = 0; i < 8; i++) p.x[i] = make_float4(mine[i * 128u], mine[i * 128u + 32u], mine[i * 128u + 64u], mine[i * 128u + 96u]);
            __syncwarp();      // the buffer's next use is another lane's
        }
    }
}

// Block (n0, mp) of the tile, all eight worker warps: warp w has the TMEM lanes (tile columns) of quarter w % 4 and the pieces
// w / 4, w / 4 + 2, ... of the rows.
// A function of its own that takes values: a reference to the caller's state, or a register too many, would put state into
// local memory, and with the ring in shared memory hardly any L1 is left, so every access to it goes to L2.  The slot's
// fields are read once: the compiler may not keep them in registers across the stores.
template <bool RES>
static __device__ __noinline__ bool epilogue_block(const Slot &sl, unsigned n0, unsigned mp, unsigned half, unsigned acc_parity, float *stage, Shared *sh,
                                                   CtrlDev *ctrl, StatusHost *status) {
    const LayerDev &L = sl.layer;
    const unsigned lane = threadIdx.x & 31u, warp = (threadIdx.x >> 5) - WARP_WORK, lane0 = (warp & 3u) * 32u, first = warp >> 2;
    const unsigned cols_left = sl.tile.tile_w - n0, n_valid = cols_left > lane0 ? min(32u, cols_left - lane0) : 0u;     // columns of this warp
    const unsigned rows = min(BLOCK_ROWS, sl.tile.tile_h - mp), pieces = (rows + 31u) >> 5;
    const unsigned acc = sh->tmem_base + half * BLOCK_ROWS + (lane0 << 16);
    const size_t col0 = sl.tile.pos_w + n0 + lane0, ldc = L.ldc, ld_res = L.res_ld_in, ld_out2 = L.res_ld_out;
    const unsigned m0 = sl.tile.pos_h + mp, quad = (lane & 7u) * 4u;
    const bool plain = L.type == V_ATTENTION_LAYER, rnd = L.round_out != 0, rnd2 = L.res_round != 0, live = n_valid && first < pieces;
    const bool own = !RES || L.res_elide == 0;
    const int act = plain ? (int)NO_ACTIVATION : L.act, act2 = L.res_act;
    const float *bias = plain ? nullptr : L.bias, *rin = L.res_in + col0 * ld_res + m0;
    float *out = L.out + col0 * ldc + m0, *out2 = L.res_out + col0 * ld_out2 + m0;
    float *vt = RES ? nullptr : L.vt_out;
    const size_t vt_ld = L.vt_ld;
    if (vt) {
        const unsigned col = (unsigned)col0 + lane, seq = L.seq, bt = col / seq;
        vt += (size_t)m0 * vt_ld + (size_t)bt * L.vt_seq + (col - bt * seq);
    }
    Piece p, r, r2;
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) {
        if (RES) {
            load_piece(r, rin + first * 32u, ld_res, n_valid, min(32u, rows - first * 32u));
            if (first + 2u < pieces) load_piece(r2, rin + (first + 2u) * 32u, ld_res, n_valid, min(32u, rows - (first + 2u) * 32u));
        }
        b = load_bias(bias ? bias + m0 + first * 32u + quad : nullptr, (int)(rows - first * 32u) - (int)quad);
    }
    bool ok = mbar_wait(&sh->acc_full[half], acc_parity, ctrl, status, 4);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    if (ok && live)
        for (unsigned c = first; c < pieces; c += 2u) {
            const unsigned valid = min(32u, rows - c * 32u), m = c * 32u;
            float v[32];
            tmem_ld32(acc + m, v);
            if (c + 2u >= pieces) {
                // last read of the accumulator by this warp
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->acc_empty[half]);
            }
            transpose(stage, v, p);
            #pragma unroll
            for (unsigned i = 0; i < 8; i++) { p.x[i].x += b.x; p.x[i].y += b.y; p.x[i].z += b.z; p.x[i].w += b.w; }
            if (bias && c + 2u < pieces) b = load_bias(bias + m0 + m + 64u + quad, (int)(rows - (c + 2u) * 32u) - (int)quad);
            activate_piece(p, act, stage);
            if (rnd) round_piece(p);
            if (own) store_piece(p, out + m, ldc, n_valid, valid);
            if (!RES && vt) {
                // transposed copy for an attention_v consumer: back to one column per lane, so that each of the 32 stores of a
                // warp covers consecutive words of a feature's row
                untranspose(stage, p, v);
                if (lane < n_valid) {
                    float *t = vt + (size_t)m * vt_ld;
                    #pragma unroll
                    for (unsigned j = 0; j < 32; j++) { if (j < valid) *t = v[j]; t += vt_ld; }
                }
            }
            if (RES) {
                // fused residual layer (ref src/tiled_kernels.c:503-541 computes it as a layer of its own): out2 = act(value +
                // other), same piece.  The value itself is stored only if something else reads it.
                #pragma unroll
                for (unsigned i = 0; i < 8; i++) {
                    p.x[i].x += r.x[i].x; p.x[i].y += r.x[i].y; p.x[i].z += r.x[i].z; p.x[i].w += r.x[i].w;
                    r.x[i] = r2.x[i];
                }
                if (c + 4u < pieces) load_piece(r2, rin + (c + 4u) * 32u, ld_res, n_valid, min(32u, rows - (c + 4u) * 32u));
                activate_piece(p, act2, stage);
                if (rnd2) round_piece(p);
                store_piece(p, out2 + m, ld_out2, n_valid, valid);
            }
        }
    else {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->acc_empty[half]);
    }
    return ok;
}

__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, %0;" ::"r"(NW) : "memory"); }

// K-attention: scores -> mask -> / sqrt(hd) -> exp, normalised by the column sum, no maximum subtracted (ref
// src/tiled_kernels.c:859-876).  All keys of 128 queries are in TMEM at once: one block, or two (both accumulator halves) for
// more than 256 keys.  The two warps of a query quarter take alternate pieces and add their sums; the exponentials go back
// to TMEM, so each is computed once.  `parity`: acc_full parity of each half.
// `ok` false: the warp has given up before; it only meets the others at the barriers.
static __device__ __noinline__ bool softmax_block(const Slot &sl, unsigned n0, unsigned half, unsigned parity, bool ok, unsigned char *epi, Shared *sh, CtrlDev *ctrl,
                                                  StatusHost *status) {
    const LayerDev &L = sl.layer;
    const unsigned tile_w = sl.tile.tile_w, tile_h = sl.tile.tile_h, pos_w = sl.tile.pos_w, pos_h = sl.tile.pos_h;
    const bool masked = L.masked != 0, rnd = L.round_out != 0;
    const size_t ldc = L.ldc;
    const unsigned lane = threadIdx.x & 31u, warp = (threadIdx.x >> 5) - WARP_WORK, lane0 = (warp & 3u) * 32u, first = warp >> 2;
    const unsigned cols_left = tile_w - n0, n_valid = cols_left > lane0 ? min(32u, cols_left - lane0) : 0u;
    const unsigned two = tile_h > BLOCK_ROWS ? 1u : 0u;
    float *stage = reinterpret_cast<float *>(epi + warp * 4096u), *other = reinterpret_cast<float *>(epi + (warp ^ 4u) * 4096u);
    float *out = L.out + (size_t)(pos_w + n0 + lane0) * ldc + pos_h;
    const unsigned acc = sh->tmem_base + (lane0 << 16);
    const float scale = 1.4426950408889634f / sqrtf((float)L.hd);
    const unsigned q = pos_w % L.seq + n0 + lane0 + lane;
    ok = ok && mbar_wait(&sh->acc_full[half], (parity >> half) & 1u, ctrl, status, 4);
    if (two) ok = ok && mbar_wait(&sh->acc_full[half ^ 1u], (parity >> (half ^ 1u)) & 1u, ctrl, status, 4);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const bool live = ok && n_valid;
    // Keys past the last query of the warp are masked for all its columns: nothing to compute, and nothing to store -- the matrix
    // is zero from the start, and nothing else ever writes there.
    const unsigned last = q - lane + 32u, seen = masked ? min(tile_h, last - min(last, pos_h)) : tile_h, seen_pieces = (seen + 31u) >> 5;
    float v[32], sum = 0.f;
    Piece p;
    if (live)
        for (unsigned c = first; c < seen_pieces; c += 2u) {
            const unsigned at = acc + (half ^ (c >> 3)) * BLOCK_ROWS + (c & 7u) * 32u;
            tmem_ld32(at, v);
            #pragma unroll
            for (unsigned j = 0; j < 32; j++) {
                const unsigned m = c * 32u + j;
                const bool in = m < tile_h && !(masked && pos_h + m > q);
                v[j] = in ? exp2f(v[j] * scale) : 0.f;
                sum += v[j];
            }
            tmem_st32(at, v);
        }
    stage[lane] = sum;
    worker_sync();
    sum += other[lane];
    worker_sync();
    const float inv_sum = 1.f / sum;
    if (live)
        for (unsigned c = first; c < seen_pieces; c += 2u) {
            tmem_ld32(acc + (half ^ (c >> 3)) * BLOCK_ROWS + (c & 7u) * 32u, v);
            #pragma unroll
            for (unsigned j = 0; j < 32; j++) v[j] *= inv_sum;
            transpose(stage, v, p);
            if (rnd) round_piece(p);
            store_piece(p, out + c * 32u, ldc, n_valid, min(32u, tile_h - c * 32u));
        }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
        mbar_arrive(&sh->acc_empty[half]);
        if (two) mbar_arrive(&sh->acc_empty[half ^ 1u]);
    }
    return ok;
}

// A contraction tile in the worker warps.  `half`: accumulator half of the next block; `acc_uses`: parity of the uses of each half.
__device__ __forceinline__ bool epilogue_tile(const Slot &sl, unsigned &half, unsigned &acc_uses, unsigned char *epi, Shared *sh, CtrlDev *ctrl, StatusHost *status) {
    const unsigned tile_w = sl.tile.tile_w, tile_h = sl.tile.tile_h;
    float *stage = reinterpret_cast<float *>(epi + ((threadIdx.x >> 5) - WARP_WORK) * 4096u);
    const bool softmax = sl.layer.type == K_ATTENTION_LAYER, res = sl.layer.res_out != nullptr;
    bool ok = true;
    for (unsigned n0 = 0; n0 < tile_w; n0 += 128u) {
        if (softmax) {
            ok = softmax_block(sl, n0, half, acc_uses, ok, epi, sh, ctrl, status);
            if (tile_h > BLOCK_ROWS) acc_uses ^= 3u;
            else { acc_uses ^= 1u << half; half ^= 1u; }
            continue;
        }
        for (unsigned mp = 0; mp < tile_h; mp += BLOCK_ROWS) {
            const unsigned parity = (acc_uses >> half) & 1u;
            if (!(res ? epilogue_block<true>(sl, n0, mp, half, parity, stage, sh, ctrl, status)
                      : epilogue_block<false>(sl, n0, mp, half, parity, stage, sh, ctrl, status))) return false;
            acc_uses ^= 1u << half;
            half ^= 1u;
        }
    }
    return ok;
}

}  // namespace tc
