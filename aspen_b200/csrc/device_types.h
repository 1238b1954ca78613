// Flattened device image of a tile graph (nasm) and the scheduler's control block.
// Shared by the host uploader (engine.cu) and the kernels.
#pragma once
#include <cstdint>

#include "index_div.h"

// Layer types / activations use the ABI enum values of include/aspen_b200.h.

// How the X operand (activations) of a contraction layer reaches shared memory on the tensor-core path; see tiles_tc.cuh.
enum { A_NONE = 0, A_TMA = 1, A_IM2COL = 2, A_HEAD = 3 };

// The scheduler copies a descriptor on the way from a ready tile to its first load: two words a lane, two lines.  (79 words with flags a
// word each: BERT 1 x 37, 96 short layers, 1193 us a pass instead of 1187; ResNet-50 x 32 served 17.92 ms instead of 17.80.)
struct alignas(128) LayerDev {
    float *out;               // own activation matrix: column-major, H rows contiguous, W columns
    const float *in0, *in1;   // activations of PARENT_0, PARENT_1
    const float *weight;      // [rows][Kpad] fp32, K contiguous, zero padded; layernorm: gain[rows]
    const float *bias;        // [rows]
    const float *anchors;
    // A residual layer fused into this (convolution / matmul) layer's epilogue: besides its own output the tile
    // also writes res_out = act(own + res_in) for the same region.  res_out == nullptr: nothing fused.
    const float *res_in;
    float *res_out;
    // A layer whose output is the value operand of an attention_v layer also writes it transposed: row = feature, column
    // b * vt_seq + s (vt_seq = seq rounded up to 32, the columns in between are zero).  That copy is what the
    // attention tile's TMA reads as a K-major operand.  nullptr: no copy.  (attention_v itself: vt_seq of that copy.)
    float *vt_out;
    unsigned vt_ld, vt_seq;
    unsigned res_ld_in, res_ld_out;
    unsigned ldc, H, W;       // column stride (floats; of every layer a multiple of 4), logical rows, columns
    unsigned ld0, H0, ld1, H1;
    unsigned K, Kpad;
    unsigned IC, IH, IW, OH, OW, KH, KW, stride, pad;     // conv / pool geometry
    unsigned seq, heads, hd;                             // attention
    unsigned p_out_c, p_in_c, p_stride;                  // yolo / append raw cfg parameters
    unsigned x_ld;            // gemv: distance between the columns
    int wmap;                 // tensor map of the W-side operand (weights, PARENT_1 for attention keys, transposed values)
    int amap;                 // tensor map of the X-side operand (PARENT_0 activations)
    unsigned chunks;          // 32-deep chunks of the contraction
    unsigned stage_bytes;     // a stage of the operand ring
    Divisor by_ic, by_kw;     // division by IC, KW
    unsigned tap_c;           // A_IM2COL: channels of a tap, rounded up to whole chunks
    unsigned short a_rows;    // columns (MMA rows) of the X-side box: 128, or what a narrow layer has
    unsigned short b_rows;    // rows of the W-side box (one per stage): the tile's rows, at most 256
    unsigned char type;       // LAYER_TYPE
    unsigned char act;        // LAYER_ACT
    unsigned char tc;         // the layer's tiles run on the tensor cores
    unsigned char meets;      // its tiles have barriers of the worker warps: the softmax of scores, fp32 blocks, a stored tile read back (vt_out)
    unsigned char gemv;       // at most 8 columns, each one contiguous run of K values: dot products (tile_gemv)
    unsigned char masked;     // attention: causal
    unsigned char a_kind;     // A_*
    unsigned char a_multi;    // one X box covers all chunks of a stage (the map has a third dimension: the chunk)
    unsigned char per_stage;  // chunks of one stage
    unsigned char stages;
    unsigned char a_vec4;     // fp32 tiles: operand rows can be fetched in 16-byte pieces (IC % 4 == 0 ...)
    unsigned char round_out;  // store outputs rounded to TF32 (nearest): a tensor-core layer reads them
    unsigned char tap_kw, tap_sx, tap_sy, tap_pad;       // A_IM2COL: taps of a row, input pixels between two output pixels, padding
    unsigned char res_act, res_round;
    unsigned char res_elide;  // the layer's own (pre-add) output has no other reader and is not written
};
static_assert(sizeof(LayerDev) == 256, "two words a lane");

struct alignas(64) TileDev {        // two sectors, one load for the scheduler
    unsigned layer;
    unsigned pos_h, pos_w;    // position in the layer's output matrix
    unsigned tile_h, tile_w;  // clipped extents
    unsigned child_off, child_cnt;
    unsigned need;            // completions of parents that a pass of the tile waits for
    // Contractions in the fp32 mode: the values of k that the tile sums.  Where a layer's k is split, `slices` tiles of the same outputs
    // leave their sums in `part`, [slice][column][rows rounded up to 4], and count at `arrived`; the one that comes last adds them
    // in order and writes the outputs.
    unsigned k0, k1;
    unsigned slice, slices;
    float *part;
    unsigned *arrived;
};

// The layer-0 tiles run on the device and turn what the host uploaded into the layer's activation matrix, so a
// graph's next pass can start inside the running kernel.
struct InputDev {
    const float *stage;       // packed [column][rows] copy as uploaded; nullptr when the upload goes straight into layer 0
    const int *ids;           // token ids as uploaded (one per column), nullptr otherwise
    const float *emb_tok, *emb_pos;
    unsigned emb_vocab, emb_seq;
    float *padded;            // zero-padded [sample][PH][PW][4] copy of the image for a convolution on it, nullptr otherwise
    unsigned IC, IH, IW, PH, PW, pad;
    unsigned round;           // values are rounded to TF32 (nearest)
};

// words of NasmDev::svc
#define SVC_TARGET 0u         // written by the host: number of the last pass asked for
#define SVC_STARTED 1u        // number of the last pass started
#define SVC_IDLE 2u           // 1: no pass in progress
#define SVC_COUNT 3u          // tiles completed since the kernel was launched
#define SVC_BASE 4u           // passes complete when the kernel was launched
#define SVC_WORDS 8u

struct NasmDev {
    const LayerDev *layers;
    const TileDev *tiles;
    const unsigned *children;        // CSR payload: (local child tile id, layer << 16 | count that child waits for) pairs
    unsigned *dep;                   // [n_tiles] parents completed since the launch
    volatile unsigned *completed;    // mapped host word: number of the last complete pass
    const void *wmaps;               // CUtensorMap[]
    unsigned n_tiles;
    unsigned n_counters;             // words of dep: a counter per tile, and one per set of tiles with a split k
    unsigned *svc;                   // SVC_* words in device memory
    unsigned n_exec;                 // tiles that complete in one pass (every tile but the ones whose parents write their values)
    unsigned n_input;                // layer-0 tiles (local ids 0 .. n_input-1): the seeds of a pass
    InputDev input;
};

struct CtrlDev {
    unsigned head;           // next ticket to hand out
    unsigned tail;           // next free queue slot
    unsigned done;           // tiles completed
    unsigned total;          // tiles of one pass of every graph
    unsigned cap;            // queue capacity
    unsigned abort;          // set with a status code: everybody leaves
    unsigned stop;           // host request: leave after the current tile
    unsigned n_nasm;
    unsigned long long stall_ns;   // no-progress window after which a wait gives up
    unsigned long long pipe_ns;    // time budget of in-kernel pipeline waits
    unsigned svc_stop;       // host request: leave once no pass is running or asked for
    unsigned svc_close;      // set by the device: everybody leaves (no error)
    unsigned ordered;        // the tiles are handed out in a fixed order (scheduler.cuh) instead of as they become ready
    unsigned ahead;          // a busy CTA lines up a second tile when at least this many ready tiles wait unclaimed (0: never); in a fixed
                             // order: it claims one when the tile in work has its weights
    unsigned long long idle_ns;    // leave after this long without a pass in progress
};

struct StatusHost {          // mapped host memory
    volatile unsigned status;        // ASPEN_B200_ERR_*
    volatile unsigned info0, info1;  // where it gave up (tile id / barrier id)
};

#define ASPEN_TILE_NONE 0xffffffffu
