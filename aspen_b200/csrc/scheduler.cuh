// Persistent device-side dataflow scheduler: the B200 counterpart of the reference's DSE worker
// loop (dse_schedule, ref src/dse.c:20-108) and ready pool (ref src/rpool.c:390-685).
//
// One CTA per SM stays resident for a whole launch.  A launch per run hands its tiles out in a fixed order (`ordered_warp`: claim the
// next one, wait for its counter); in service mode, where passes of several graphs are at different stages, the scheduler warp
//   pops a ready tile      (rpool_fetch_ninsts)     ticket = atomicAdd(head); wait for queue[ticket]
//   lets the CTA run it    (switch on layer type, ref src/dse.c:39-79)
//   updates the children   (update_children_but_prioritize_dse_target, ref src/dse.c:363-401):
//                          atomicAdd on each child's dependency counter; a child whose last parent
//                          this was becomes ready; the first such child is kept as this CTA's next
//                          tile (depth first, no queue round trip), the others are pushed
//   accounts completion    one counter per graph; its last tile ends the graph's pass (ref src/dse.c:80-106)
// There is no kernel boundary and no barrier between layers: a tile fires as soon as its own
// parent tiles are complete.
//
// Passes.  The host asks for pass number p of a graph by writing p to the graph's SVC_TARGET word.  A scheduler
// warp that finds an idle graph with target != started claims it (CAS on SVC_IDLE) and pushes its layer-0 tiles; those
// prepare the input, everything else follows from the dependency counters.  The warp that retires the last tile of a
// pass writes the pass number to the graph's mapped host word and marks the graph idle.
//   A launch per run (dse_group_run by default): one pass of each graph that owes one; the kernel leaves when they are complete.
//   Service mode: the kernel stays resident while the host keeps asking (the counterpart of the reference's DSE threads,
//   which run from dse_group_run to dse_group_stop and serve whatever rpool_add_nasm brings, ref src/dse.c:20-108,
//   215-232).  It leaves -- without error -- when no pass is running or asked for and the host has asked it to
//   stop, when nothing has run for idle_ns, or when the queue of this launch is used up; the host launches it
//   again if work is left.
// The counters are never reset between the passes of a launch: a pass only starts when the previous one of its graph is
// complete, so a child is ready whenever its counter reaches a multiple of the count it waits for.
//
// The queue is a ticket ring with room for a fixed number of passes, so it never wraps; 0 = slot not yet filled.  A popper
// that holds a ticket whose slot is still empty waits -- bounded: when no tile anywhere completes for
// `stall_ns` it records ASPEN_B200_ERR_STALL, raises the abort flag and every CTA leaves.
//
// Latency.  From the last store of a tile to the first load of the tile it makes ready lie the scheduler's round trips to
// L2 (about 0.4 us each): fence, child counters, fence, and -- through the queue -- tail, slot, the popper's poll, the
// descriptors.  What can be known earlier is fetched earlier: a tile's child list while the tile runs; queue entries and
// child lists name the layer and the graph, so that a tile's descriptor and its layer's are read side by side.
//
// Memory ordering: tile data is written by the worker threads; their mbarrier arrivals order it before the
// scheduler warp's fence.acq_rel.gpu + relaxed atomicAdd on the child counter (release).  The CTA
// whose increment completes the count fences again after the atomic (acquiring every earlier
// parent's data through the counter's RMW chain) before it publishes or keeps the child.
#pragma once
#include "tiles_tc.cuh"
#include "worker_loop.h"

namespace sched {

constexpr unsigned PROF_LAYERS = 256;
constexpr unsigned PROF_SLOTS = 2 + 2 * PROF_LAYERS + 2;

// A ready tile: low word = local tile id + 1 (0: none), high word = graph << 16 | layer.
typedef unsigned long long Entry;
__host__ __device__ __forceinline__ Entry make_entry(unsigned tile, unsigned g, unsigned layer) { return (Entry)(tile + 1u) | ((Entry)((g << 16) | layer) << 32); }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ Entry ld_acquire(const Entry *p) {
    Entry v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(Entry *p, Entry v) { asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory"); }
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ tc::GraphRef graph_ref(const NasmDev &G) {
    return {G.layers, G.tiles, reinterpret_cast<const uint2 *>(G.children), G.dep, (const unsigned char *)G.wmaps, &G.input, G.svc, G.n_exec};
}
__device__ __forceinline__ tc::GraphRef graph_ref(const tc::Shared *sh, const NasmDev *nasms, unsigned g) {
    return g < tc::CACHED_GRAPHS ? sh->graphs[g] : graph_ref(nasms[g]);
}

// Child update of a completed tile; called by the whole (converged) scheduler warp.  An edge is (child tile, layer << 16 |
// count the child waits for); `e` holds this lane's first edge, fetched while the tile ran.
// Returns a child this CTA should run next (only when want_keep), or 0.
static __device__ __forceinline__ Entry complete_children(const tc::GraphRef &G, unsigned g, uint2 e, unsigned child_off, unsigned child_cnt, CtrlDev *ctrl, Entry *queue, unsigned cap, bool want_keep) {
    const unsigned lane = threadIdx.x & 31u;
    const uint2 *edges = G.children + child_off;
    unsigned *dep = G.dep;
    fence_gpu();                                         // release: this tile's output
    Entry next = 0;
    for (unsigned base = 0; base < child_cnt; base += 32u) {
        const unsigned idx = base + lane;
        bool ready = false;
        if (idx < child_cnt) {
            if (base) e = edges[idx];
            const unsigned now = atomicAdd(&dep[e.x], 1u) + 1u;
            ready = now % (e.y & 0xffffu) == 0u;
        }
        unsigned mask = __ballot_sync(0xffffffffu, ready);
        if (mask == 0u) continue;
        fence_gpu();                                     // acquire the other parents' outputs (through the counters), then publish
        const Entry mine = make_entry(e.x, g, e.y >> 16);
        if (want_keep && next == 0) {
            const unsigned first = __ffs(mask) - 1u;
            next = __shfl_sync(0xffffffffu, mine, first);
            mask &= ~(1u << first);
            if (lane == first) ready = false;
        }
        const unsigned n_push = __popc(mask);
        if (n_push) {
            unsigned pos = 0;
            if (lane == 0) pos = atomicAdd(&ctrl->tail, n_push);
            pos = __shfl_sync(0xffffffffu, pos, 0);
            if (ready) {
                const unsigned rank = __popc(mask & ((1u << lane) - 1u));
                if (pos + rank < cap) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&queue[pos + rank]), "l"(mine) : "memory");   // behind the fence
            }
        }
    }
    return next;
}

// Looks at every graph, a lane a graph; starts the next pass where one is asked for.  Whole (converged) warp.
// Returns bit 0: some graph has a pass in progress, bit 1: a pass is asked for but this launch's queue has no room left,
// bit 2: this warp started a pass.
static __device__ unsigned svc_scan(const NasmDev *nasms, unsigned n_nasm, CtrlDev *ctrl, Entry *queue, const tc::Shared *sh) {
    const unsigned lane = threadIdx.x & 31u;
    unsigned st = 0;
    for (unsigned g0 = 0; g0 < n_nasm; g0 += 32u) {
        const unsigned g = g0 + lane;
        unsigned go = 0;
        if (g < n_nasm) {
            unsigned *svc = graph_ref(sh, nasms, g).svc;
            if (ld_acquire(&svc[SVC_IDLE]) == 0u) go = 1u;
            else if (ld_acquire_sys(&svc[SVC_TARGET]) == ld_acquire(&svc[SVC_STARTED])) {
                // nothing asked for -- or another warp has claimed the pass between the two reads
                go = ld_acquire(&svc[SVC_IDLE]) == 0u ? 1u : 0u;
            } else {
                // (room for a pass of every graph: no graph has more than one in progress)
                if (ld_relaxed(&ctrl->tail) + ctrl->total > ctrl->cap) go = 2u;
                else if (atomicCAS(&svc[SVC_IDLE], 1u, 0u) == 1u) {
                    // only the holder of the claim changes SVC_STARTED: look again now that it is ours
                    const unsigned started = ld_relaxed(&svc[SVC_STARTED]);
                    if (ld_acquire_sys(&svc[SVC_TARGET]) != started) {
                        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&svc[SVC_STARTED]), "r"(started + 1u) : "memory");
                        go = 4u;
                    } else asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&svc[SVC_IDLE]), "r"(1u) : "memory");
                } else go = 1u;
            }
        }
        __syncwarp();
        st |= __reduce_or_sync(0xffffffffu, go);
        for (unsigned mask = __ballot_sync(0xffffffffu, go == 4u); mask; mask &= mask - 1u) {
            const unsigned mine = g0 + __ffs(mask) - 1u, n_input = nasms[mine].n_input;
            unsigned pos = 0;
            if (lane == 0) pos = atomicAdd(&ctrl->tail, n_input);
            pos = __shfl_sync(0xffffffffu, pos, 0);
            for (unsigned i = lane; i < n_input; i += 32u)
                if (pos + i < ctrl->cap) st_release(&queue[pos + i], make_entry(i, mine, 0));
        }
    }
    return st;
}

// `t` tiles of graph g have completed since the launch: every n_exec-th completion ends a pass.  Whole warp.
static __device__ void end_of_pass(const NasmDev *nasms, unsigned n_nasm, unsigned g, unsigned t, CtrlDev *ctrl, Entry *queue, const tc::Shared *sh) {
    const NasmDev &G = nasms[g];
    if ((threadIdx.x & 31u) == 0) {
        __threadfence_system();
        *G.completed = ld_relaxed(&G.svc[SVC_BASE]) + t / G.n_exec;          // mapped host word: number of the pass that is complete
        __threadfence_system();
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&G.svc[SVC_IDLE]), "r"(1u) : "memory");
    }
    __syncwarp();
    // the next pass of this graph may already be asked for; with nothing left and the host's request to stop, everybody leaves
    if (svc_scan(nasms, n_nasm, ctrl, queue, sh) == 0u && (threadIdx.x & 31u) == 0u && ld_relaxed(&ctrl->svc_stop) != 0u) atomicExch(&ctrl->svc_close, 1u);
}

// Arms a launch: empty queue, zero counters, every graph idle at the pass count the host has seen complete.  The pass numbers
// travel as arguments (a launch of the same graphs then needs no copy); more than ARM_GRAPHS graphs take several launches,
// the first of which (g0 = 0) also resets the queue and the control words.
constexpr unsigned ARM_GRAPHS = 32;
struct ArmArgs {
    unsigned g0, n, n_nasm, cap, total, svc_stop, ahead, ordered;
    unsigned long long stall_ns, pipe_ns, idle_ns;
    unsigned base[ARM_GRAPHS], target[ARM_GRAPHS];
};
static __global__ void arm_kernel(const NasmDev *nasms, CtrlDev *ctrl, Entry *queue, const ArmArgs a) {
    const unsigned stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (a.g0 == 0 && !a.ordered)
        for (unsigned i = t0; i < a.cap; i += stride) queue[i] = 0u;
    for (unsigned g = 0; g < a.n; g++) {
        const NasmDev &G = nasms[a.g0 + g];
        unsigned *dep = G.dep;
        for (unsigned i = t0, n = G.n_counters; i < n; i += stride) dep[i] = 0u;
        if (t0 == 0) {
            G.svc[SVC_STARTED] = G.svc[SVC_BASE] = a.base[g];
            G.svc[SVC_TARGET] = a.target[g];
            G.svc[SVC_IDLE] = 1u; G.svc[SVC_COUNT] = 0u;
        }
    }
    if (t0 == 0 && a.g0 == 0) {
        ctrl->head = 0u; ctrl->tail = 0u; ctrl->done = 0u; ctrl->total = a.total; ctrl->cap = a.cap; ctrl->n_nasm = a.n_nasm;
        ctrl->abort = 0u; ctrl->stop = 0u; ctrl->stall_ns = a.stall_ns; ctrl->pipe_ns = a.pipe_ns;
        ctrl->svc_stop = a.svc_stop; ctrl->svc_close = 0u; ctrl->idle_ns = a.idle_ns; ctrl->ahead = a.ahead; ctrl->ordered = a.ordered;
    }
}

// A tile that runs on the worker warps alone; `wt`: worker thread 0 .. tc::NW-1, `scratch`: the shared memory of fp32 blocks.
template <bool TENSOR_CORES>
static __device__ __noinline__ void worker_tile(const tc::Slot &sl, unsigned wt, unsigned char *scratch, unsigned *last) {
    const LayerDev &L = sl.layer;
    const TileDev &T = sl.tile;
    switch (L.type) {
        case CONV_LAYER: case FC_LAYER: case MATMUL_LAYER: case K_ATTENTION_LAYER: case V_ATTENTION_LAYER:
            tile_gemm_ffma<!TENSOR_CORES>(L, T, wt, tc::NW, scratch, last);
            break;
        case RESIDUAL_LAYER: tile_residual(L, T, wt, tc::NW); break;
        case MAXPOOL_LAYER:
            // whole 16-byte pieces, and every window holds a pixel of the image
            if (((T.tile_h | T.pos_h | L.ld0 | L.ldc) & 3u) == 0u && L.KH == L.KW && L.pad < L.KH && (L.OH - 1u) * L.stride < L.IH + L.pad &&
                (L.OW - 1u) * L.stride < L.IW + L.pad && (L.KH == 2u || L.KH == 3u)) {
                if (L.KH == 2u) tile_max_small<2, 2, 4>(L, T, wt, tc::NW);
                else tile_max_small<3, 3, 2>(L, T, wt, tc::NW);
            } else tile_pool<true>(L, T, wt, tc::NW);
            break;
        case AVGPOOL_LAYER:
            if (((T.tile_h | T.pos_h | L.ld0 | L.ldc) & 3u) == 0u && L.pad == 0u && (L.OH - 1u) * L.stride + L.KH <= L.IH && (L.OW - 1u) * L.stride + L.KW <= L.IW)
                tile_avg_inside(L, T, wt, tc::NW);
            else tile_pool<false>(L, T, wt, tc::NW);
            break;
        case LAYERNORM_LAYER: tile_layernorm(L, T, wt, tc::NW); break;
        case SOFTMAX_LAYER: tile_softmax(L, T, wt, tc::NW); break;
        case YOLO_LAYER: tile_yolo(L, T, wt, tc::NW); break;
        case APPEND_LAYER: tile_append(L, T, wt, tc::NW); break;
        case INPUT_LAYER: tile_input(*sl.input, L, T, wt, tc::NW); break;
        default: break;
    }
    if (TENSOR_CORES && L.vt_out) tile_transposed_copy(L, T, wt, tc::NW);
}

// ---- the persistent kernel -------------------------------------------------------------------
// The SCHEDULER warp hands tiles to the other roles (tiles_tc.cuh) through SLOTS slots in shared memory; slot k = sequence
// number % SLOTS.  It copies the tile's descriptor and its layer's into the slot and arrives on posted[k]; every role takes
// the slots in order, at its own pace, and arrives on finished[k] when it is done with the slot (the worker warps: when all
// stores of the tile are made).  The scheduler then updates the children (a first child that became ready is kept as this
// CTA's next tile), does the completion accounting, and may use the slot again.
// The fp32 kernel has no producers: its scheduler is warp 0, its workers follow, and nobody shares the registers.
template <bool TENSOR_CORES> __host__ __device__ constexpr unsigned threads() { return TENSOR_CORES ? tc::THREADS : 32u + tc::NW; }
// dynamic shared memory: operand ring and transposing buffers (tensor cores), or the staging of the fp32 blocks
constexpr unsigned FFMA_BYTES = 96u * 1024u;
template <bool TENSOR_CORES> __host__ __device__ constexpr unsigned work_bytes() { return TENSOR_CORES ? tc::RING_BYTES + tc::EPI_BYTES : FFMA_BYTES; }

// Fills slot k with a tile and hands it to the roles (whole warp).  The tile's and the layer's descriptors are independent
// loads; both and the graph's addresses are constant while the kernel runs.
static __device__ __forceinline__ void post(tc::Shared *sh, unsigned k, const tc::GraphRef &G, Entry entry) {
    tc::Slot &sl = sh->slots[k];
    const unsigned lane = threadIdx.x & 31u, g = (unsigned)(entry >> 48), layer = (unsigned)(entry >> 32) & 0xffffu, tile = (unsigned)entry - 1u;
    constexpr unsigned LW = sizeof(LayerDev) / 4, TW = sizeof(TileDev) / 4;
    static_assert(LW == 64 && TW <= 32, "copied in words");
    const unsigned *lsrc = reinterpret_cast<const unsigned *>(G.layers + layer), *tsrc = reinterpret_cast<const unsigned *>(G.tiles + tile);
    const unsigned l0 = __ldg(lsrc + lane), l1 = __ldg(lsrc + 32u + lane);
    unsigned tw = 0;
    if (lane < TW) tw = __ldg(tsrc + lane);
    reinterpret_cast<unsigned *>(&sl.layer)[lane] = l0;
    reinterpret_cast<unsigned *>(&sl.layer)[32u + lane] = l1;
    if (lane < TW) reinterpret_cast<unsigned *>(&sl.tile)[lane] = tw;
    if (lane == 0) { sl.live = 1u; sl.nasm = g; sl.maps = G.maps; sl.input = G.input; }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&sh->posted[k]);
}
static __device__ __forceinline__ void post_ready(tc::Shared *sh, unsigned k) {
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) tc::mbar_arrive(&sh->ready[k]);
}
// The marker behind the last tile.
static __device__ __forceinline__ void post_exit(tc::Shared *sh, unsigned k) {
    if ((threadIdx.x & 31u) == 0) { sh->slots[k].live = 0u; tc::mbar_arrive(&sh->posted[k]); tc::mbar_arrive(&sh->ready[k]); }
}

static __device__ __noinline__ void scheduler_warp(const NasmDev *nasms, CtrlDev *ctrl, Entry *queue, StatusHost *status, tc::Shared *sh, unsigned long long *my_prof) {
    const unsigned lane = threadIdx.x & 31u, n_nasm = ctrl->n_nasm;
    unsigned issued = 0, retired = 0;           // tiles posted to / retired from the slots: at most two apart
    uint2 edge0 = make_uint2(0u, 1u), edge1 = edge0;   // this lane's first child edge of the tiles in the slots (by parity)
    unsigned acct_nasm = 0;                     // completion accounting still to do
    bool acct = false;
    Entry kept = 0;                             // a child made ready by a tile this CTA completed
    unsigned ticket = ASPEN_TILE_NONE;          // a queue position we hold and wait on
    bool closed = false;                        // no further tiles will be issued (end of run, stop)
    bool no_tickets = false;                    // the queue has no unowned position left; kept children still run
    const unsigned cap = ctrl->cap, ahead = ctrl->ahead;
    const unsigned *watch = lane == 1u ? &ctrl->abort : lane == 2u ? &ctrl->stop : lane == 3u ? &ctrl->svc_close : &ctrl->done;
    unsigned last_done = 0;
    unsigned long long t_progress = __shfl_sync(0xffffffffu, global_ns(), 0), t_mark = t_progress;
    const unsigned long long window = ctrl->stall_ns;
    unsigned idle_spins = 30u, turn = 0, flags = 0, done = 0, ahead_turn = 0, q_tail = 0, q_head = 0;   // the first idle turns already look for a pass to start
    while (true) {
        bool progressed = false;
        // Control words (lanes 1 - 4) and the slot we wait on (lane 0) are read together: one L2 round trip a turn.  With a tile
        // in work the control words are sampled every 64th turn: what the turn is then waiting for is the tile.
        unsigned word = 0;
        Entry slot = 0;
        const bool sample = issued == retired || (turn++ & 63u) == 0u;
        if (sample && lane >= 1u && lane <= 4u) word = ld_relaxed(watch);
        if (ticket != ASPEN_TILE_NONE && lane == 0u) slot = ld_acquire(&queue[ticket]);
        if (sample) {
            flags = __ballot_sync(0xffffffffu, lane >= 1u && lane <= 3u && word != 0u);
            done = __shfl_sync(0xffffffffu, word, 4);
            if (flags & 2u) break;               // aborted: roles leave their tiles unfinished, nothing more will be retired
            if (flags) closed = true;
        }
        // 1. retire the oldest tile in flight once every role has finished it
        if (issued > retired) {
            const unsigned k = retired % tc::SLOTS;
            unsigned ok = lane == 0 ? (unsigned)tc::mbar_test_wait(&sh->finished[k], (retired / tc::SLOTS) & 1u) : 0u;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (ok) {
                __syncwarp();                    // a shuffle orders no memory: what lane 0 has observed holds for the lanes that release it
                if (my_prof && lane == 0) t_mark = global_ns();
                const tc::Slot &sl = sh->slots[k];
                const unsigned g = sl.nasm;
                const Entry child = complete_children(graph_ref(sh, nasms, g), g, (retired & 1u) ? edge1 : edge0, sl.tile.child_off, sl.tile.child_cnt, ctrl, queue, cap, kept == 0);
                if (child) kept = child;
                if (my_prof && lane == 0) my_prof[1] += global_ns() - t_mark;
                acct_nasm = g;
                acct = true;
                retired++;
                progressed = true;
            }
        }
        // 2. find the next tile
        Entry next = 0;
        if (!closed && issued - retired < 2u) {
            if (kept) { next = kept; kept = 0; }
            else if (!no_tickets) {
                // An idle CTA queues up for the next ready tile.  A busy one (one tile in work) lines up a second only when at
                // least `ahead` ready tiles wait unclaimed: its operands then stream in under the first one's epilogue, and
                // the completion of the first runs beside the second.  A ticket held for a tile that is not there yet would
                // keep that tile from an idle SM.
                bool take = ticket == ASPEN_TILE_NONE && issued == retired;
                if (ahead != 0u && !take && ticket == ASPEN_TILE_NONE) {
                    // asked for in one turn, looked at some turns later: the turns in between do not wait for it
                    if ((ahead_turn & 7u) == 0u && lane == 0) { q_tail = ld_relaxed(&ctrl->tail); q_head = ld_relaxed(&ctrl->head); }
                    if ((ahead_turn & 7u) == 7u) take = __shfl_sync(0xffffffffu, (int)(q_tail - q_head), 0) >= (int)ahead;
                    ahead_turn++;
                }
                if (take) {
                    unsigned t = lane == 0 ? atomicAdd(&ctrl->head, 1u) : 0u;
                    ticket = __shfl_sync(0xffffffffu, t, 0);
                    if (ticket >= cap) { ticket = ASPEN_TILE_NONE; no_tickets = true; }   // every tile that can be pushed has an owner
                }
                else if (ticket != ASPEN_TILE_NONE) {
                    next = __shfl_sync(0xffffffffu, slot, 0);
                    if (next) ticket = ASPEN_TILE_NONE;
                }
            }
        }
        // 3. post it: one tile in work, one behind it
        if (next) {
            const unsigned k = issued % tc::SLOTS;
            const tc::GraphRef G = graph_ref(sh, nasms, (unsigned)(next >> 48));
            post(sh, k, G, next);
            post_ready(sh, k);
            const tc::Slot &sl = sh->slots[k];
            uint2 e = make_uint2(0u, 1u);
            if (lane < sl.tile.child_cnt) e = __ldg(G.children + sl.tile.child_off + lane);
            if (issued & 1u) edge1 = e; else edge0 = e;
            issued++;
            progressed = true;
        }
        // 4. completion accounting, behind everything that another tile may be waiting for
        if (acct) {
            unsigned t = 0;
            const tc::GraphRef G = graph_ref(sh, nasms, acct_nasm);
            if (lane == 0) { atomicAdd(&ctrl->done, 1u); t = atomicAdd(&G.svc[SVC_COUNT], 1u) + 1u; }
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t % G.n_exec == 0u) end_of_pass(nasms, n_nasm, acct_nasm, t, ctrl, queue, sh);
            // With every SM busy nobody is idle for long enough to look for passes asked for since; every 32nd tile somebody does.
            // (Looked for by idle SMs alone, a graph's next pass began when another's ended: bursts of 12 requests of ResNet-50 x 32
            // 17.4 ms and now 14.9, of 32 of x 4 8.9 and 7.8, of 16 of BERT 16 x 128 21.9 and 20.3.)
            else if ((retired & 31u) == (blockIdx.x & 31u)) svc_scan(nasms, n_nasm, ctrl, queue, sh);
            acct = false;
        }
        // 5. end of launch / stall detection
        if (issued == retired) {
            if (closed) break;
            if (no_tickets && kept == 0) break;   // can never get work again
        }
        if (progressed || done != last_done) {
            unsigned long long now = lane == 0 ? global_ns() : 0ull;
            last_done = done; t_progress = __shfl_sync(0xffffffffu, now, 0); idle_spins = 0;
            continue;
        }
        if (((++idle_spins) & 31u) == 0u) {
            unsigned long long now = lane == 0 ? global_ns() : 0ull;
            now = __shfl_sync(0xffffffffu, now, 0);
            unsigned svc = 1u;
            if (issued == retired && !closed) {
                // an idle CTA looks for passes to start, and decides when the kernel has nothing left to wait for
                svc = svc_scan(nasms, n_nasm, ctrl, queue, sh);
                if (svc & 4u) t_progress = now;
                else if (!(svc & 1u)) {
                    unsigned leave = (svc & 2u) ? 1u : 0u;
                    if (lane == 0 && !leave) leave = (ld_relaxed(&ctrl->svc_stop) != 0u || now - t_progress > ctrl->idle_ns) ? 1u : 0u;
                    leave = __shfl_sync(0xffffffffu, leave, 0);
                    if (leave) {
                        if (lane == 0) atomicExch(&ctrl->svc_close, 1u);
                        closed = true;
                    }
                }
            }
            if (now - t_progress > window && issued == retired && (svc & 1u)) {
                // nothing running here, nothing completed anywhere for a whole window: the graph cannot progress
                if (lane == 0 && atomicCAS(&ctrl->abort, 0u, (unsigned)ASPEN_B200_ERR_STALL) == 0u) {
                    status->info0 = ticket; status->info1 = done; status->status = ASPEN_B200_ERR_STALL;
                    __threadfence_system();
                }
                closed = true;
            }
            if (my_prof && lane == 0 && issued == retired) my_prof[0] += 1ull;   // idle polls with nothing in flight
        }
        __nanosleep(20u);
    }
    post_exit(sh, issued % tc::SLOTS);
}

// A launch in a fixed order.  Every tile of the launch is in `order`, parents before children; a CTA claims the next position,
// posts that tile at once and waits for its counter itself.  Against the ready queue this takes the counter's answer, the queue's
// tail, its entry and the descriptors off the way from a tile's last store to its child's first load (what is left: one fence,
// one reduction, one poll), and a tile's weights stream into the ring while it waits.  What it gives up is the choice among ready
// tiles: a claimed tile waits for its own parents while another could run.  The order is that of a simulated run
// (plan.cpp: claim_order), so that a tile's turn comes when its parents are about done.  Device time of a pass, queue and order:
// CIFAR net x 1 68 and 49 us, BERT 1 x 37 1128 and 878, ResNet-50 x 1 fp32 1126 and 1022, x 32 1541 and 1466, GPT-2 8 x 512 2520
// and 2461, ResNet-50 + VGG-16 x 16 2132 and 1832.
// Claims are contiguous and a tile's parents lie before it, so whatever is claimed completes; a CTA asked to stop only
// claims no more.
static __device__ __noinline__ void ordered_warp(const NasmDev *nasms, CtrlDev *ctrl, const Entry *order, StatusHost *status, tc::Shared *sh, unsigned long long *my_prof) {
    const unsigned lane = threadIdx.x & 31u, count = ctrl->cap;
    const unsigned *watch = lane == 1u ? &ctrl->abort : lane == 2u ? &ctrl->stop : &ctrl->done;
    const unsigned long long window = ctrl->stall_ns;
    unsigned issued = 0, running = 0, retired = 0;     // tiles posted / whose parents are complete / completed: at most two apart
    uint2 edge0 = make_uint2(0u, 1u), edge1 = edge0;   // this lane's first child edge of the tiles in the slots (by parity)
    enum { NOTHING, TICKET, ENTRY } claim = NOTHING;   // what has been asked for; looked at in a later turn
    unsigned ticket = 0, need = 0, counted = 0, count_nasm = 0, turn = 0, last_done = 0;
    const unsigned *dep = nullptr;                     // of the posted tile that waits for its parents
    Entry entry = 0;
    const bool ahead = ctrl->ahead != 0u;
    bool closed = false, out = false, accounting = false, aborted = false;
    unsigned long long t_progress = __shfl_sync(0xffffffffu, global_ns(), 0), t_mark = t_progress;
    // the pass's last tile ends it
    auto account = [&]() {
        const NasmDev &G = nasms[count_nasm];
        if (lane == 0 && counted == G.n_exec) {
            __threadfence_system();
            *G.completed = ld_relaxed(&G.svc[SVC_BASE]) + 1u;
            __threadfence_system();
        }
        __syncwarp();
        accounting = false;
    };
    while (true) {
        bool progressed = false;
        // 1. retire the oldest running tile once every role has finished it
        if (running > retired) {
            const unsigned k = retired % tc::SLOTS;
            unsigned ok = lane == 0 ? (unsigned)tc::mbar_test_wait(&sh->finished[k], (retired / tc::SLOTS) & 1u) : 0u;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (ok) {
                __syncwarp();                    // a shuffle orders no memory: what lane 0 has observed holds for the lanes that release it
                if (my_prof && lane == 0) t_mark = global_ns();
                const tc::Slot &sl = sh->slots[k];
                const unsigned g = sl.nasm, cnt = sl.tile.child_cnt;
                const tc::GraphRef G = graph_ref(sh, nasms, g);
                uint2 e = (retired & 1u) ? edge1 : edge0;
                fence_gpu();                     // release: this tile's output
                for (unsigned idx = lane; idx < cnt; idx += 32u) {
                    if (idx >= 32u) e = __ldg(G.children + sl.tile.child_off + idx);
                    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(G.dep + e.x) : "memory");
                }
                if (my_prof && lane == 0) my_prof[1] += global_ns() - t_mark;
                if (accounting) account();
                // the count of the pass is looked at in a later turn
                if (lane == 0) {
                    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&ctrl->done) : "memory");
                    counted = atomicAdd(&G.svc[SVC_COUNT], 1u) + 1u;
                }
                count_nasm = g;
                accounting = progressed = true;
                retired++;
            }
        }
        // 2. the tile that waits for its parents; with nothing else to do the counter is read as fast as it can be
        if (issued > running) {
            unsigned v = 0;
            const bool idle = running == retired;
            if (lane == 0) v = idle ? ld_acquire(dep) : ld_relaxed(dep);
            const bool there = __shfl_sync(0xffffffffu, (int)(v - need), 0) >= 0;
            if (there) {
                if (!idle) fence_gpu();          // acquire the parents' outputs
                post_ready(sh, running % tc::SLOTS);
                running++;
                progressed = true;
            }
        }
        // 3. claim the next tile
        bool want = claim == NOTHING && issued == running && issued - retired < 2u && !out && !closed;
        if (want && issued != retired) {
            // A busy CTA claims ahead when the tile in work has all its weights, so that the next one's stream in under its epilogue --
            // but only where several graphs share the launch and work is plenty: alone, the tile it holds back would often be
            // ready for an idle CTA (ResNet-50 x 32 1466 us a pass without, 1487 with; ResNet-50 and VGG-16 x 16 1995 and 1832).
            unsigned fed = 0;
            if (ahead && sh->slots[retired % tc::SLOTS].layer.tc) {
                if (lane == 0) fed = (unsigned)tc::mbar_test_wait(&sh->fed[retired % tc::SLOTS], (retired / tc::SLOTS) & 1u);
                fed = __shfl_sync(0xffffffffu, fed, 0);
            }
            want = fed != 0u;
        }
        if (want) {
            if (lane == 0) ticket = atomicAdd(&ctrl->head, 1u);
            claim = TICKET;
        } else if (claim == TICKET) {
            ticket = __shfl_sync(0xffffffffu, ticket, 0);
            out = ticket >= count;
            claim = out ? NOTHING : ENTRY;
            if (!out) entry = __ldg(order + ticket);
        } else if (claim == ENTRY) {
            const unsigned k = issued % tc::SLOTS;
            const tc::GraphRef G = graph_ref(sh, nasms, (unsigned)(entry >> 48));
            post(sh, k, G, entry);
            const tc::Slot &sl = sh->slots[k];
            need = sl.tile.need;
            dep = G.dep + ((unsigned)entry - 1u);
            uint2 e = make_uint2(0u, 1u);
            if (lane < sl.tile.child_cnt) e = __ldg(G.children + sl.tile.child_off + lane);
            if (issued & 1u) edge1 = e; else edge0 = e;
            issued++;
            claim = NOTHING;
        }
        // 4. completion accounting, behind everything that another tile may be waiting for
        if (accounting && !progressed) account();
        if (issued == retired && claim == NOTHING && (out || closed) && !accounting) break;
        // 5. control words and stall detection
        if (progressed) continue;
        if ((++turn & 31u) == 0u) {
            unsigned word = lane >= 1u && lane <= 3u ? ld_relaxed(watch) : 0u;
            const unsigned flags = __ballot_sync(0xffffffffu, lane >= 1u && lane <= 2u && word != 0u), done = __shfl_sync(0xffffffffu, word, 3);
            unsigned long long now = lane == 0 ? global_ns() : 0ull;
            now = __shfl_sync(0xffffffffu, now, 0);
            if (flags & 2u) { aborted = true; break; }       // roles leave their tiles unfinished, nothing more will be retired
            if (flags & 4u) closed = true;
            if (done != last_done || running > retired) { last_done = done; t_progress = now; }
            else if (now - t_progress > window) {
                // nothing running here, nothing completed anywhere for a whole window: the graph cannot progress
                if (lane == 0 && atomicCAS(&ctrl->abort, 0u, (unsigned)ASPEN_B200_ERR_STALL) == 0u) {
                    status->info0 = (unsigned)entry - 1u; status->info1 = done; status->status = ASPEN_B200_ERR_STALL;
                    __threadfence_system();
                }
                aborted = true;
                break;
            }
            if (my_prof && lane == 0 && running == retired) my_prof[0] += 1ull;   // idle polls with nothing in flight
        }
        if (issued == running) __nanosleep(20u);
    }
    if (aborted && issued > running) {                   // the waiting tile is withdrawn
        if (lane == 0) sh->slots[running % tc::SLOTS].live = 0u;
        post_ready(sh, running % tc::SLOTS);
    }
    post_exit(sh, issued % tc::SLOTS);
}

// The loops of the one-warp roles, all their state inside: a reference to it would put it into local memory.
template <unsigned ROLE>
static __device__ __forceinline__ void one_warp_role(unsigned char *smem, tc::Shared *sh, CtrlDev *ctrl, StatusHost *status) {
    const unsigned ring = tc::smem_u32(smem);
    tc::Ring r;
    unsigned half = 0, acc_uses = 0;
    for (unsigned seq = 0;; seq++) {
        const unsigned k = seq % tc::SLOTS;
        const unsigned parity = (seq / tc::SLOTS) & 1u;
        if (!__all_sync(0xffffffffu, tc::wait_slot(&sh->posted[k], parity, ctrl, status))) break;
        const tc::Slot &sl = sh->slots[k];
        if (!tc::uniform(sl.live)) break;
        if (tc::uniform((unsigned)sl.layer.tc)) {
            bool ok;
            if (ROLE == tc::WARP_A) ok = tc::produce_a(sl, &sh->ready[k], parity, ring, r, sh, ctrl, status);
            else if (ROLE == tc::WARP_B) ok = tc::produce_b(sl, &sh->ready[k], parity, ring, r, sh, ctrl, status);
            else ok = tc::wait_ready(sl, &sh->ready[k], parity, ctrl, status) && tc::issue_mma(sl, ring, r, half, acc_uses, sh, ctrl, status);
            if (!ok) break;
        }
        __syncwarp();
        if ((threadIdx.x & 31u) == 0u) {
            if (ROLE == tc::WARP_B) tc::mbar_arrive(&sh->fed[k]);
            tc::mbar_arrive(&sh->finished[k]);
        }
    }
    if (*(volatile unsigned *)&ctrl->abort) {
        // copies and MMAs of this CTA may still be in flight; they take microseconds
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
}

// What a worker warp does at each step of worker_loop.  It keeps next to nothing across a tile -- the tiles are calls, and what does not
// fit the registers that they leave would come back by an L2 round trip.
template <bool TENSOR_CORES>
struct WorkerWarp {
    CtrlDev *ctrl;
    StatusHost *status;
    unsigned long long *prof;                    // of all CTAs, or nullptr
    unsigned half = 0, acc_uses = 0;

    __device__ __forceinline__ static unsigned char *smem() { extern __shared__ __align__(1024) unsigned char work[]; return work; }
    __device__ __forceinline__ static tc::Shared *sh() { return reinterpret_cast<tc::Shared *>(smem() + work_bytes<TENSOR_CORES>()); }
    __device__ __forceinline__ static unsigned wt() { return threadIdx.x - (TENSOR_CORES ? tc::WARP_WORK : 1u) * 32u; }     // worker thread 0 .. tc::NW - 1
    __device__ __forceinline__ static tc::Slot &slot(unsigned seq) { return sh()->slots[seq % tc::SLOTS]; }
    // time since the last call, for the accounting of the CTA (one thread)
    __device__ __forceinline__ static unsigned long long lap() {
        const unsigned long long now = global_ns(), t = now - sh()->prof_mark;
        sh()->prof_mark = now;
        return t;
    }
    __device__ __forceinline__ bool posted(unsigned seq) {
        return __all_sync(0xffffffffu, tc::wait_slot(&sh()->ready[seq % tc::SLOTS], (seq / tc::SLOTS) & 1u, ctrl, status));
    }
    __device__ __forceinline__ bool live(unsigned seq) const { return slot(seq).live != 0u; }
    __device__ __forceinline__ bool meets(unsigned seq) const { return slot(seq).layer.meets != 0u; }
    __device__ __forceinline__ bool agree(bool yes) const {
        unsigned all;
        __syncwarp();
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                     : "=r"(all) : "r"(yes ? 1u : 0u), "r"(tc::NW) : "memory");
        return all != 0u;
    }
    __device__ __forceinline__ bool run(unsigned seq) {
        if (prof && wt() == 0) prof[(size_t)blockIdx.x * PROF_SLOTS + PROF_SLOTS - 1] += lap();
        bool ok = true;
        if (TENSOR_CORES && slot(seq).layer.tc) ok = tc::epilogue_tile(slot(seq), half, acc_uses, smem() + tc::RING_BYTES, sh(), ctrl, status);
        else worker_tile<TENSOR_CORES>(slot(seq), wt(), smem() + (TENSOR_CORES ? tc::RING_BYTES : 0u), &sh()->last);
        if (prof && wt() == 0) {
            unsigned long long *mine = prof + (size_t)blockIdx.x * PROF_SLOTS + 2 + slot(seq).tile.layer % PROF_LAYERS;
            mine[0] += lap(); mine[PROF_LAYERS] += 1ull;
        }
        return ok;
    }
    __device__ __forceinline__ void finished(unsigned seq) const {
        __syncwarp();
        if ((threadIdx.x & 31u) == 0u) tc::mbar_arrive(&sh()->finished[seq % tc::SLOTS]);      // release (CTA scope): this warp's stores of the tile
    }
};

// Registers move from the first warpgroup to the two of workers: 128 x 104 + 256 x 200 = 384 x 168, what the launch holds.
constexpr int ROLE_REGISTERS = 104, WORKER_REGISTERS = 200;
static_assert(128 * ROLE_REGISTERS + 256 * WORKER_REGISTERS <= 384 * 168, "register split");

template <bool TENSOR_CORES>
__global__ void __launch_bounds__(threads<TENSOR_CORES>(), 1)
scheduler_kernel(const NasmDev *nasms, CtrlDev *ctrl, Entry *queue /* or, ctrl->ordered, the order of the launch */, StatusHost *status, unsigned long long *prof) {
    extern __shared__ __align__(1024) unsigned char smem[];      // stages need 1024-byte alignment for the 128-byte swizzle
    tc::Shared *sh = reinterpret_cast<tc::Shared *>(smem + work_bytes<TENSOR_CORES>());
    const unsigned tid = threadIdx.x, warp = tc::uniform(tid >> 5);
    constexpr unsigned sched_warp = TENSOR_CORES ? tc::WARP_SCHED : 0u, first_worker = TENSOR_CORES ? tc::WARP_WORK : 1u;

    if (tid == 0) {
        sh->prof_mark = global_ns();
        for (unsigned s = 0; s < tc::MAX_STAGES; s++) { tc::mbar_init(&sh->full[s], 2u); tc::mbar_init(&sh->empty[s], 1u); }
        for (unsigned h = 0; h < 2; h++) { tc::mbar_init(&sh->acc_full[h], 1u); tc::mbar_init(&sh->acc_empty[h], tc::NW / 32u); }
        for (unsigned k = 0; k < tc::SLOTS; k++) { tc::mbar_init(&sh->fed[k], 1u); tc::mbar_init(&sh->posted[k], 1u); tc::mbar_init(&sh->ready[k], 1u); tc::mbar_init(&sh->finished[k], tc::NW / 32u + (TENSOR_CORES ? 3u : 0u)); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_proxy_async_smem();
    }
    if (TENSOR_CORES) {
        if (warp == tc::WARP_MMA) tc::tmem_alloc(&sh->tmem_base, tc::TMEM_COLS);
        tc::tc_fence_before();
    }
    for (unsigned g = tid, n = min(tc::CACHED_GRAPHS, ctrl->n_nasm); g < n; g += threads<TENSOR_CORES>()) sh->graphs[g] = graph_ref(nasms[g]);
    __syncthreads();
    if (TENSOR_CORES) tc::tc_fence_after();

    // Optional time accounting per CTA: [0] scheduler idle polls, [1] completion + child update (ns),
    // [2 + layer] ns the workers spent on tiles of that layer (index modulo PROF_LAYERS),
    // [2 + PROF_LAYERS + layer] tile counts, [PROF_SLOTS - 1] ns the workers waited for a tile.
    // The first four warps need few registers, the workers many: a spill costs an L2 round trip here, because the ring leaves
    // almost no L1 (with 168 registers for everybody the epilogue of a 256 x 128 block took 12 us instead of 6).
    if (TENSOR_CORES) {
        if (warp >= first_worker) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(WORKER_REGISTERS));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ROLE_REGISTERS));
    }
    if (warp == sched_warp) {
        unsigned long long *mine = prof ? prof + (size_t)blockIdx.x * PROF_SLOTS : nullptr;
        if (ctrl->ordered) ordered_warp(nasms, ctrl, queue, status, sh, mine);
        else scheduler_warp(nasms, ctrl, queue, status, sh, mine);
    } else if (warp >= first_worker) {
        WorkerWarp<TENSOR_CORES> w{ctrl, status, prof};
        worker_loop(w);
    } else if (TENSOR_CORES) {
        if (warp == tc::WARP_A) one_warp_role<tc::WARP_A>(smem, sh, ctrl, status);
        else if (warp == tc::WARP_B) one_warp_role<tc::WARP_B>(smem, sh, ctrl, status);
        else one_warp_role<tc::WARP_MMA>(smem, sh, ctrl, status);
    }
    __syncwarp();
    if (TENSOR_CORES) tc::tc_fence_before();
    __syncthreads();
    if (TENSOR_CORES && warp == tc::WARP_MMA) { tc::tc_fence_after(); tc::tmem_dealloc(sh->tmem_base, tc::TMEM_COLS); }
}

}  // namespace sched
