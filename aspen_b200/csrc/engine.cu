// Host side of the device engine: uploads weights and flattened tile graphs, owns the stream,
// launches the persistent scheduler, and moves inputs / results.  The only translation unit of
// the library that calls the CUDA runtime.  There is no CPU execution path: without a usable
// sm_100 device every entry point fails with an error.
#include "internal.h"
#include "scheduler.cuh"
#include "hostcopy.h"
#include "fp32.h"
#include "recent_sets.h"

#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <memory>
#include <mutex>
#include <sched.h>
#include <unordered_map>

#define CUDA_TRY(expr)                                                                          \
    do {                                                                                        \
        cudaError_t err__ = (expr);                                                             \
        if (err__ != cudaSuccess) {                                                             \
            ASPEN_ERR("CUDA error %s at %s: %s\n", cudaGetErrorName(err__), #expr, cudaGetErrorString(err__)); \
            return -1;                                                                          \
        }                                                                                       \
    } while (0)

struct Engine;
static int svc_halt(Engine *e);

static thread_local int g_device = -1;

extern "C" int aspen_b200_set_device(int device) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
        ASPEN_ERR("aspen_b200_set_device: device %d not available (%d visible)\n", device, n);
        return -1;
    }
    g_device = device;
    return cudaSetDevice(device) == cudaSuccess ? 0 : -1;
}

// Whether every layer's output stays readable after a run (the default), or outputs that only feed a residual add
// fused into their producer are left unwritten (1 = keep all, 0 = drop those).  Read when a graph's device image is built.
static thread_local int g_keep_hidden = -1;

extern "C" void aspen_b200_set_hidden_states(int keep) { g_keep_hidden = keep ? 1 : 0; }

static bool keep_hidden_states() {
    if (g_keep_hidden >= 0) return g_keep_hidden != 0;
    const char *v = getenv("ASPEN_B200_HIDDEN_STATES");
    return !(v && *v && atoi(v) == 0);
}

int engine_current_device() {
    if (g_device >= 0) return g_device;
    if (const char *v = getenv("ASPEN_B200_DEVICE")) {     // for callers that cannot call aspen_b200_set_device
        int n = 0, want = atoi(v);
        if (*v && cudaGetDeviceCount(&n) == cudaSuccess && want >= 0 && want < n) return want;
    }
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) return 0;
    return d;
}

// ---- device copies of a dnn's weights ----------------------------------------------------------
struct DeviceDnn {
    int device = 0;
    // per layer, per precision mode (0: rounded to TF32, 1: exact fp32)
    std::vector<float *> weight[2];
    std::vector<float *> bias;
    std::vector<float *> anchors;
    std::vector<unsigned> kpad;
    std::vector<float *> weight_boxes;  // A_IM2COL layers whose taps are not whole 32-value chunks: every tap zero padded (OperandForm::k)
    std::vector<unsigned> ic_pad;     // conv on the network input, connected layer, with IC % 4 != 0: channels padded to this many (0: not padded)
    bool have[2] = {false, false};
    float *emb_token = nullptr, *emb_position = nullptr;   // embedding tables, uploaded on first use
};

static float round_to_tf32(float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    if ((u & 0x7f800000u) == 0x7f800000u) return x;
    u += 0x00001000u;          // round to nearest, ties away: 13 mantissa bits are dropped
    u &= 0xffffe000u;
    memcpy(&x, &u, 4);
    return x;
}

static int upload_weights(aspen_dnn_t *dnn, int device, int precision, DeviceDnn **out) {
    if (device < 0 || device >= 16) { ASPEN_ERR("device index %d out of range\n", device); return -1; }
    DeviceDnn *dd = dnn->dev[device];
    if (!dd) {
        dd = new DeviceDnn();
        dd->device = device;
        dd->weight[0].assign(dnn->num_layers, nullptr);
        dd->weight[1].assign(dnn->num_layers, nullptr);
        dd->bias.assign(dnn->num_layers, nullptr);
        dd->anchors.assign(dnn->num_layers, nullptr);
        dd->kpad.assign(dnn->num_layers, 0);
        dd->ic_pad.assign(dnn->num_layers, 0);
        dd->weight_boxes.assign(dnn->num_layers, nullptr);
        dnn->dev[device] = dd;
    }
    *out = dd;
    if (dd->have[precision]) return 0;
    for (unsigned i = 0; i < dnn->num_layers; i++) {
        aspen_layer_t &l = dnn->layers[i];
        aspen_tensor_t *w = l.tensors[WEIGHT_TENSOR], *b = l.tensors[BIAS_TENSOR], *a = l.tensors[ANCHOR_TENSOR];
        if (w) {
            unsigned rows = layer_weight_rows(&l);
            unsigned k = l.type == LAYERNORM_LAYER ? 1 : layer_contraction_k(&l);
            // A convolution straight on the network input with an odd channel count (the 3-channel stem), and a connected layer
            // over padded columns: the parent's pad rows stay zero, so the device copy pads every tap to a multiple of 4 channels
            // with zero weights and the tile reads 16-byte pieces, or the whole sample as one row.
            unsigned ic = l.params[IN_C], icp = ic;
            if (ic % 4 != 0 && (l.type == FC_LAYER || (l.type == CONV_LAYER && l.parent_layers[PARENT_0] && l.parent_layers[PARENT_0]->type == INPUT_LAYER))) {
                icp = (unsigned)round_up(ic, 4);
                dd->ic_pad[i] = icp;
            }
            const unsigned taps = icp != ic ? k / ic : 1, kk = icp != ic ? taps * icp : k;
            unsigned kpad = l.type == LAYERNORM_LAYER ? 1 : (unsigned)round_up(kk, 32);
            dd->kpad[i] = kpad;
            std::vector<float> padded((size_t)rows * kpad, 0.f);
            const float *src = (const float *)w->data;
            for (unsigned r = 0; r < rows; r++)
                for (unsigned c = 0; c < k; c++) {
                    float v = src[(size_t)r * k + c];
                    unsigned dc = icp != ic ? (c / ic) * icp + c % ic : c;
                    padded[(size_t)r * kpad + dc] = (precision == 0 && l.type != LAYERNORM_LAYER) ? round_to_tf32(v) : v;
                }
            CUDA_TRY(cudaMalloc(&dd->weight[precision][i], padded.size() * sizeof(float) + 256));
            CUDA_TRY(cudaMemcpy(dd->weight[precision][i], padded.data(), padded.size() * sizeof(float), cudaMemcpyHostToDevice));
            const OperandForm form = operand_form(&l, 0);
            if (precision == 0 && form.kind == A_IM2COL && (form.image || (ic % 32 != 0 && form.kh * form.kw > 1)) && !dd->weight_boxes[i]) {
                const unsigned window = k / ic, in_row = form.image ? l.params[WEIGHT_W] : 1, cp = (unsigned)round_up(form.c, 32);
                std::vector<float> boxes((size_t)rows * form.k(), 0.f);
                for (unsigned r = 0; r < rows; r++)
                    for (unsigned t = 0; t < window; t++)
                        for (unsigned c = 0; c < ic; c++)
                            boxes[(size_t)r * form.k() + t / in_row * cp + t % in_row * 4 + c] = round_to_tf32(src[(size_t)r * k + t * ic + c]);
                CUDA_TRY(cudaMalloc(&dd->weight_boxes[i], boxes.size() * sizeof(float) + 256));
                CUDA_TRY(cudaMemcpy(dd->weight_boxes[i], boxes.data(), boxes.size() * sizeof(float), cudaMemcpyHostToDevice));
            }
        }
        if (b && !dd->bias[i]) {
            CUDA_TRY(cudaMalloc(&dd->bias[i], (size_t)b->num_elements * sizeof(float) + 256));
            CUDA_TRY(cudaMemcpy(dd->bias[i], b->data, (size_t)b->num_elements * sizeof(float), cudaMemcpyHostToDevice));
        }
        if (a && !dd->anchors[i]) {
            CUDA_TRY(cudaMalloc(&dd->anchors[i], 8 * sizeof(float)));
            CUDA_TRY(cudaMemcpy(dd->anchors[i], a->data, 6 * sizeof(float), cudaMemcpyHostToDevice));
        }
    }
    dd->have[precision] = true;
    return 0;
}

void engine_release_dnn(aspen_dnn_t *dnn) {
    for (auto &dd : dnn->dev) {
        if (!dd) continue;
        int prev = 0;
        cudaGetDevice(&prev);
        cudaSetDevice(dd->device);
        for (int p = 0; p < 2; p++)
            for (float *ptr : dd->weight[p]) cudaFree(ptr);
        for (float *ptr : dd->bias) cudaFree(ptr);
        for (float *ptr : dd->weight_boxes) cudaFree(ptr);
        for (float *ptr : dd->anchors) cudaFree(ptr);
        cudaFree(dd->emb_token);
        cudaFree(dd->emb_position);
        cudaSetDevice(prev);
        delete dd;
        dd = nullptr;
    }
}

// ---- engine --------------------------------------------------------------------------------
struct MergedOrder {
    sched::Entry *tiles = nullptr;
    unsigned cap = 0;
};
static void free_order(MergedOrder &o) { cudaFree(o.tiles); }

struct Engine {
    int device = 0;
    int precision = 0;
    int num_sms = 0;
    unsigned n_ctas = 0;
    size_t smem_bytes = 0;
    cudaStream_t stream = nullptr, side = nullptr, io = nullptr;   // compute, stop flag, host transfers
    CtrlDev *ctrl = nullptr;
    StatusHost *status_h = nullptr;   // mapped host memory
    StatusHost *status_d = nullptr;
    sched::Entry *queue = nullptr;
    unsigned queue_cap = 0;
    // Several graphs in one launch (images, by DeviceNasm::serial): their tiles in the order they are handed out, 8 bytes each.  A program whose
    // launches take turns between sets finds each set's order (64: every set of six graphs).  Made anew for every launch it cost a call of
    // ResNet-50 + VGG-16 x 16 (1770 us) another 100; the CIFAR net in 56 sets of seven graphs, dse_group_run: 45 us with 8 sets kept, 10 with 64.
    RecentSets<MergedOrder, 64> orders;
    NasmDev *nasms_d = nullptr;
    unsigned nasms_cap = 0;
    std::vector<NasmDev> uploaded;    // what nasms_d holds
    unsigned long long stall_ns = 2000000000ull;
    unsigned long long pipe_ns = 1000000000ull;
    unsigned long long launches = 0;
    bool service = false;             // service mode: one kernel serves pass after pass of its graphs until dse_group_stop (see scheduler.cuh)
    bool uploading = false;           // inputs were copied on the compute stream since a launch or a read
    bool svc_live = false;            // a kernel was launched and has not yet been seen to end
    std::vector<nasm_t *> svc_graphs; // the graphs that kernel serves
    std::vector<nasm_t *> svc_pool;   // every graph of the group's rpool that has a device image: what the next launch serves
    unsigned long long idle_ns = 20000000ull;   // the kernel leaves after this long with no pass running
    cudaEvent_t svc_armed_ev = nullptr;
    unsigned svc_ahead = 32;          // see CtrlDev::ahead
    std::unique_ptr<HostCopy> copy;   // results into pageable memory
    unsigned long long *prof = nullptr;   // per-CTA time accounting, allocated when ASPEN_B200_PROFILE is set
};

struct DeviceNasm {
    Engine *e = nullptr;
    DeviceDnn *dd = nullptr;
    std::unique_ptr<nasm_t> plan;   // the tiles the device executes
    float *arena = nullptr;
    size_t arena_bytes = 0;
    std::vector<size_t> ldata_off;
    LayerDev *layers = nullptr;
    TileDev *tiles = nullptr;
    unsigned *children = nullptr, *dep = nullptr;
    void *wmaps = nullptr;
    NasmDev host;               // the graph's entry in a launch, but for its input
    unsigned long long serial = 0;      // no two images have the same
    ClaimOrder claims;
    std::vector<unsigned> tile_layer;
    sched::Entry *order = nullptr;      // claims of a launch of this graph alone
    bool round_input = false;   // tensor-core path: the input is rounded to TF32 by the layer-0 tiles
    unsigned *svc_d = nullptr;                               // SVC_* words
    unsigned *svc_done_h = nullptr, *svc_done_d = nullptr;   // mapped: number of the last complete pass
    unsigned svc_armed = 0;                                  // number of the last pass the host has asked for
    unsigned svc_chain = 0;                                  // timing loops: passes complete when the next launch starts
    bool svc_ids = false;                                    // the last input was token ids
    float *in_stage = nullptr;          // packed input as uploaded (strided layer 0), spread by the layer-0 tiles
    int *ids_stage = nullptr;           // token ids as uploaded
    std::vector<float *> scratch;       // transposed copies of attention value matrices (LayerDev::vt_out), shared probabilities
    // zero-padded [sample][PH][PW][4] copy of the input image (borders stay zero), written by the layer-0 tiles (OperandForm::image)
    float *padded_in = nullptr;
    unsigned pin_ph = 0, pin_pw = 0, pin_pad = 0, pin_ic = 0, pin_ih = 0, pin_iw = 0;
};

static bool env_u64(const char *name, unsigned long long *out) {
    const char *v = getenv(name);
    if (!v || !*v) return false;
    *out = strtoull(v, nullptr, 10);
    return true;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const int *,
                                   const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
template <typename Fn>
static Fn driver_fn(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? (Fn)p : nullptr;
}
static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = driver_fn<EncodeTiledFn>("cuTensorMapEncodeTiled");
    return fn;
}
static EncodeIm2colFn get_encode_im2col_fn() {
    static EncodeIm2colFn fn = driver_fn<EncodeIm2colFn>("cuTensorMapEncodeIm2col");
    return fn;
}

Engine *engine_create(int device, int precision, unsigned int /*num_dse_hint*/) {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device >= count) {
        cudaGetLastError();
        ASPEN_ERR("no CUDA device %d (%d visible); this library has no CPU execution path\n", device, count);
        return nullptr;
    }
    cudaDeviceProp prop;
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&prop, device) != cudaSuccess) {
        ASPEN_ERR("cannot select CUDA device %d\n", device);
        return nullptr;
    }
    if (prop.major != 10) {
        ASPEN_ERR("device %d is sm_%d%d; the kernels are built for sm_100a only\n", device, prop.major, prop.minor);
        return nullptr;
    }
    Engine *e = new Engine();
    e->device = device;
    e->precision = precision;
    e->num_sms = prop.multiProcessorCount;
    e->copy.reset(new HostCopy());
    unsigned long long v;
    e->n_ctas = (unsigned)e->num_sms;
    if (env_u64("ASPEN_B200_CTAS", &v) && v > 0 && v <= (unsigned long long)e->num_sms) e->n_ctas = (unsigned)v;
    if (env_u64("ASPEN_B200_STALL_MS", &v) && v > 0) e->stall_ns = v * 1000000ull;
    if (env_u64("ASPEN_B200_PIPE_MS", &v) && v > 0) e->pipe_ns = v * 1000000ull;
    e->smem_bytes = (precision == 0 ? sched::work_bytes<true>() : sched::work_bytes<false>()) + sizeof(tc::Shared);
    bool ok = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&e->side, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&e->io, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&e->ctrl, sizeof(CtrlDev)) == cudaSuccess && cudaMemset(e->ctrl, 0, sizeof(CtrlDev)) == cudaSuccess &&
              cudaHostAlloc(&e->status_h, sizeof(StatusHost), cudaHostAllocMapped) == cudaSuccess &&
              cudaHostGetDevicePointer(&e->status_d, e->status_h, 0) == cudaSuccess;
    if (ok) {
        memset((void *)e->status_h, 0, sizeof(StatusHost));
        ok = (precision == 0 ? cudaFuncSetAttribute(sched::scheduler_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e->smem_bytes)
                             : fp32_prepare(e->smem_bytes)) == cudaSuccess;
        ok = ok && cudaEventCreateWithFlags(&e->svc_armed_ev, cudaEventDisableTiming) == cudaSuccess;
        if (env_u64("ASPEN_B200_IDLE_MS", &v) && v > 0) e->idle_ns = v * 1000000ull;
        if (env_u64("ASPEN_B200_SVC_AHEAD", &v)) e->svc_ahead = (unsigned)v;
        if (env_u64("ASPEN_B200_SERVICE", &v)) e->service = v != 0;      // for programs that cannot call aspen_b200_dse_group_set_service
        e->copy->prepare(0);
    }
    if (ok && getenv("ASPEN_B200_PROFILE")) {
        size_t bytes = (size_t)e->n_ctas * sched::PROF_SLOTS * sizeof(unsigned long long);
        ok = cudaMalloc(&e->prof, bytes) == cudaSuccess && cudaMemset(e->prof, 0, bytes) == cudaSuccess;
    }
    if (ok && precision == 0 && (!get_encode_fn() || !get_encode_im2col_fn())) { ASPEN_ERR("driver has no cuTensorMapEncodeTiled / Im2col\n"); ok = false; }
    if (!ok) {
        ASPEN_ERR("engine_create: CUDA setup failed: %s\n", cudaGetErrorString(cudaGetLastError()));
        engine_destroy(e);
        return nullptr;
    }
    return e;
}

void engine_destroy(Engine *e) {
    if (!e) return;
    cudaSetDevice(e->device);
    svc_halt(e);
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (e->stream) cudaStreamDestroy(e->stream);
    if (e->side) cudaStreamDestroy(e->side);
    if (e->io) cudaStreamDestroy(e->io);
    if (e->svc_armed_ev) cudaEventDestroy(e->svc_armed_ev);
    cudaFree(e->ctrl);
    if (e->status_h) cudaFreeHost((void *)e->status_h);
    cudaFree(e->queue);
    e->orders.drop(0, free_order);
    cudaFree(e->nasms_d);
    cudaFree(e->prof);
    delete e;
}

int engine_status(Engine *e) { return e ? (int)e->status_h->status : ASPEN_B200_ERR_CUDA; }

template <typename T>
static int to_device(T **dst, const std::vector<T> &src) {
    size_t bytes = std::max<size_t>(src.size(), 1) * sizeof(T);
    CUDA_TRY(cudaMalloc(dst, bytes));
    if (!src.empty()) CUDA_TRY(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
    return 0;
}

static void fill_layer(const nasm_t *nasm, const DeviceNasm *dn, unsigned i, int precision, LayerDev &L) {
    const nasm_ldata_t &ld = nasm->ldata[i];
    const aspen_layer_t &l = *ld.layer;
    const unsigned *p = l.params;
    memset(&L, 0, sizeof L);
    L.type = l.type;
    L.act = l.activation;
    L.out = (float *)((char *)dn->arena + dn->ldata_off[i]);
    L.ldc = ld.out_mat_stride; L.H = ld.out_mat_dims[OUT_H]; L.W = ld.out_mat_dims[OUT_W];
    unsigned p0 = ld.parent_ldata_idx_arr[PARENT_0], p1 = ld.parent_ldata_idx_arr[PARENT_1];
    if (p0 != (unsigned)-1) {
        L.in0 = (const float *)((char *)dn->arena + dn->ldata_off[p0]);
        L.ld0 = nasm->ldata[p0].out_mat_stride; L.H0 = nasm->ldata[p0].out_mat_dims[OUT_H];
    }
    if (p1 != (unsigned)-1) {
        L.in1 = (const float *)((char *)dn->arena + dn->ldata_off[p1]);
        L.ld1 = nasm->ldata[p1].out_mat_stride; L.H1 = nasm->ldata[p1].out_mat_dims[OUT_H];
    }
    L.weight = dn->dd->weight[precision][i];
    L.bias = dn->dd->bias[i];
    L.anchors = dn->dd->anchors[i];
    L.K = layer_contraction_k(&l);
    L.Kpad = dn->dd->kpad[i];
    L.IC = p[IN_C]; L.IH = p[IN_H]; L.IW = p[IN_W]; L.OH = p[OUT_H]; L.OW = p[OUT_W];
    L.KH = p[WEIGHT_H]; L.KW = p[WEIGHT_W]; L.stride = p[STRIDE] ? p[STRIDE] : 1; L.pad = p[PADDING];
    if (l.type == FC_LAYER) { L.KH = p[IN_H]; L.KW = p[IN_W]; L.OH = 1; L.OW = 1; L.stride = 1; L.pad = 0; }
    if (dn->dd->ic_pad[i]) { L.IC = dn->dd->ic_pad[i]; L.K = L.KH * L.KW * L.IC; }
    L.by_ic = make_divisor(L.IC); L.by_kw = make_divisor(L.KW);
    L.seq = nasm->tr_seq_len; L.heads = p[NUM_HEAD]; L.hd = p[NUM_HEAD] ? p[NUM_HIDDEN] / p[NUM_HEAD] : 0; L.masked = p[MASKED] != 0;
    L.p_out_c = p[OUT_C]; L.p_in_c = p[IN_C]; L.p_stride = p[STRIDE];
    L.wmap = -1;
    L.amap = -1;
    switch (l.type) {
        case CONV_LAYER: case FC_LAYER: L.a_vec4 = (L.IC % 4 == 0) && (L.ld0 % 4 == 0); break;
        case MATMUL_LAYER: L.a_vec4 = (L.K % 4 == 0) && (L.ld0 % 4 == 0); break;
        case K_ATTENTION_LAYER: L.a_vec4 = (L.hd % 4 == 0) && (L.ld0 % 4 == 0) && (L.ld1 % 4 == 0); break;
        case V_ATTENTION_LAYER: L.a_vec4 = (L.seq % 4 == 0) && (L.ld0 % 4 == 0); break;
        default: L.a_vec4 = 0; break;
    }
    if (gemv_layer(ld) && L.a_vec4 && (l.type != FC_LAYER || L.ld0 == L.IC || L.KH * L.KW == 1)) {
        L.gemv = 1;
        L.x_ld = l.type == FC_LAYER ? L.KH * L.KW * L.ld0 : L.ld0;
    }
}

static void free_device_nasm(DeviceNasm *dn) {
    if (!dn) return;
    cudaFree(dn->arena); cudaFree(dn->layers); cudaFree(dn->tiles); cudaFree(dn->children); cudaFree(dn->dep); cudaFree(dn->wmaps); cudaFree(dn->order);
    if (dn->svc_done_h) cudaFreeHost(dn->svc_done_h);
    cudaFree(dn->svc_d);
    cudaFree(dn->in_stage); cudaFree(dn->ids_stage); cudaFree(dn->padded_in);
    for (float *p : dn->scratch) cudaFree(p);
    delete dn;
}

// Layer `i` follows from layer `from` through per-token layers, at least one of which reads whole columns.
static bool follows(const nasm_t *nasm, unsigned i, unsigned from, bool whole) {
    if (i == (unsigned)-1 || i < from) return false;
    if (i == from) return whole;
    const LAYER_TYPE t = nasm->ldata[i].layer->type;
    if (t != MATMUL_LAYER && t != LAYERNORM_LAYER && t != RESIDUAL_LAYER) return false;
    whole = whole || t != RESIDUAL_LAYER;
    return follows(nasm, nasm->ldata[i].parent_ldata_idx_arr[PARENT_0], from, whole) ||
           (t == RESIDUAL_LAYER && follows(nasm, nasm->ldata[i].parent_ldata_idx_arr[PARENT_1], from, whole));
}

// The graph as the device executes it: layer geometry (strides, tiles) and lists.
static const nasm_t *device_view(const nasm_t *nasm) { return nasm->dev->plan.get(); }

static int build_device_nasm(Engine *e, nasm_t *host_nasm) {
    DeviceNasm *dn = new DeviceNasm();
    dn->e = e;
    host_nasm->dev = dn;
    const char *keep_tiles = getenv("ASPEN_B200_PLAN");      // 0: execute the nasm's own tiles
    if (host_nasm->own_lists && !(keep_tiles && atoi(keep_tiles) == 0)) dn->plan.reset(plan_device_tiles(host_nasm, e->precision, e->n_ctas, e->service));
    if (!dn->plan) dn->plan.reset(own_device_tiles(host_nasm));
    const nasm_t *nasm = dn->plan.get();
    if (upload_weights(nasm->dnn, e->device, e->precision, &dn->dd) != 0) return -1;
    // activation arena: one region per layer (no reuse: every layer output stays readable)
    dn->ldata_off.resize(nasm->num_ldata);
    size_t off = 0;
    for (unsigned i = 0; i < nasm->num_ldata; i++) {
        dn->ldata_off[i] = off;
        off += round_up(nasm->ldata[i].out_mat_mem_size + 64, 256);
    }
    dn->arena_bytes = off + 4096;
    CUDA_TRY(cudaMalloc(&dn->arena, dn->arena_bytes));
    CUDA_TRY(cudaMemsetAsync(dn->arena, 0, dn->arena_bytes, e->stream));

    // layers + tensor maps (weights and, where the access pattern allows it, the parents' activations)
    std::vector<LayerDev> layers(nasm->num_ldata);
    std::vector<CUtensorMap> maps;
    // rows of `stride_bytes` with `inner` floats; boxes of 32 floats x box_rows (per = 0), or of `per` consecutive 32-float chunks
    // x box_rows, the chunk being the third dimension (inner % 32 == 0)
    auto add_map = [&](const void *base, cuuint64_t inner, cuuint64_t outer, cuuint64_t stride_bytes, cuuint32_t box_rows, cuuint32_t per) -> int {
        CUtensorMap m;
        cuuint64_t dims[3] = {per ? 32 : inner, outer, inner / 32};
        cuuint64_t strides[2] = {stride_bytes, 128};
        cuuint32_t box[3] = {32, box_rows, per}, estr[3] = {1, 1, 1};
        CUresult r = get_encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, per ? 3 : 2, const_cast<void *>(base), dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { ASPEN_ERR("cuTensorMapEncodeTiled failed (%d)\n", (int)r); return -2; }
        maps.push_back(m);
        return (int)maps.size() - 1;
    };
    // (feature of a head, head, column): boxes of 32 features of one head x box_rows columns; what a box holds past the head's last
    // feature arrives as zeros
    auto add_head_map = [&](const void *base, const LayerDev &L, cuuint64_t columns, unsigned ld, cuuint32_t box_rows) -> int {
        CUtensorMap m;
        cuuint64_t dims[3] = {L.hd, L.heads, columns}, strides[2] = {(cuuint64_t)L.hd * 4, (cuuint64_t)ld * 4};
        cuuint32_t box[3] = {32, 1, box_rows}, estr[3] = {1, 1, 1};
        CUresult r = get_encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(base), dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { ASPEN_ERR("cuTensorMapEncodeTiled failed (%d)\n", (int)r); return -2; }
        maps.push_back(m);
        return (int)maps.size() - 1;
    };
    // The X operand by plain boxes: the chunks of a stage in one where the matrix allows it.
    auto add_x_map = [&](LayerDev &L, const void *base, cuuint64_t inner, cuuint64_t outer, cuuint64_t stride_bytes) {
        L.a_kind = A_TMA;
        L.a_multi = inner % 32 == 0;
        L.amap = add_map(base, inner, outer, stride_bytes, L.a_rows, L.a_multi ? L.per_stage : 0);
    };
    // im2col map: (channel, column, row, sample) with those extents and distances in floats, boxes of 32 channels x a_rows output pixels.
    // The corners bound the first tap of the first and last output pixel; sx, sy: input pixels between two output pixels.
    auto add_im2col_map = [&](const float *base, const unsigned (&extent)[4], const size_t (&ld)[3], int lower, int upper_x, int upper_y, unsigned sx, unsigned sy,
                              unsigned a_rows) -> int {
        CUtensorMap m;
        cuuint64_t dims[4] = {extent[0], extent[1], extent[2], extent[3]}, strides[3] = {ld[0] * 4, ld[1] * 4, ld[2] * 4};
        int low[2] = {lower, lower}, up[2] = {upper_x, upper_y};
        cuuint32_t estr[4] = {1, sx, sy, 1};
        CUresult r = get_encode_im2col_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides, low, up, 32, a_rows, estr,
                                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return -2;
        maps.push_back(m);
        return (int)maps.size() - 1;
    };
    float *probs = nullptr;                                    // see K_ATTENTION below
    size_t probs_bytes = 0;
    unsigned probs_reader = 0;
    std::vector<float *> moved(nasm->num_ldata, nullptr);      // layers that write elsewhere than into the arena
    for (unsigned i = 0; i < nasm->num_ldata; i++) {
        const aspen_layer_t &l = *nasm->ldata[i].layer;
        LayerDev &L = layers[i];
        fill_layer(nasm, dn, i, e->precision, L);
        if (nasm->ldata[i].parent_ldata_idx_arr[PARENT_0] != (unsigned)-1 && moved[nasm->ldata[i].parent_ldata_idx_arr[PARENT_0]])
            L.in0 = moved[nasm->ldata[i].parent_ldata_idx_arr[PARENT_0]];
        if (e->precision != 0 || L.gemv) continue;
        const bool gemm_w = l.type == CONV_LAYER || l.type == FC_LAYER || l.type == MATMUL_LAYER;
        const unsigned p0 = nasm->ldata[i].parent_ldata_idx_arr[PARENT_0], p1 = nasm->ldata[i].parent_ldata_idx_arr[PARENT_1];
        const cuuint64_t W0 = p0 != (unsigned)-1 ? nasm->ldata[p0].out_mat_dims[OUT_W] : 0;
        // Operand ring: a W box holds the tile's rows; a stage holds as many chunks as keep the issuing warps ahead of the MMAs
        // (a wait and a box cost the same whatever the box holds: tiles_tc.cuh)
        // while two or more stages fit.
        const unsigned th = nasm->ldata[i].ninst_tile_dims[OUT_H];
        // the epilogue stores 16-byte pieces: a tile has to start on one (a head of ten features does not)
        const bool aligned_out = th % 4 == 0 || th >= L.H;
        auto cut_ring = [&](unsigned k) {
            L.b_rows = (unsigned)round_up(std::min(th, tc::BLOCK_ROWS), 16);
            L.chunks = std::max(1u, (k + 31) / 32);
            L.per_stage = (unsigned char)std::min(L.chunks, L.b_rows <= 64 ? 4u : L.b_rows <= 128 ? 2u : 1u);
            L.a_rows = std::min(128u, (unsigned)round_up(std::min(nasm->ldata[i].ninst_tile_dims[OUT_W], L.W), 8));
            L.stage_bytes = L.per_stage * (L.a_rows + L.b_rows) * 128;
            L.stages = std::min(tc::MAX_STAGES, tc::RING_BYTES / L.stage_bytes);
        };
        if (gemm_w || l.type == K_ATTENTION_LAYER || l.type == V_ATTENTION_LAYER) cut_ring(l.type == K_ATTENTION_LAYER ? L.hd : l.type == V_ATTENTION_LAYER ? L.seq : L.Kpad);
        const OperandForm form = operand_form(&l, L.seq);
        const float *dense = L.weight;
        const unsigned dense_kpad = L.Kpad;
        if (form.kind == A_IM2COL && L.H0 == l.params[IN_C]) {
            if (dn->dd->weight_boxes[i]) { L.weight = dn->dd->weight_boxes[i]; L.Kpad = form.k(); }
            cut_ring(L.Kpad);
            L.a_kind = A_IM2COL;
            L.tap_c = (unsigned)round_up(form.c, 32);
            L.tap_kw = form.kw;
            L.tap_sy = L.stride;
            if (form.image) {
                // the padded copy as a tensor whose columns are output columns: a row of the window is 4 * KW consecutive values
                const unsigned s_ = L.stride, PW = std::max(L.IW + 2 * L.pad, s_ * (L.OW - 1) + L.KW), PH = std::max(L.IH + 2 * L.pad, s_ * (L.OH - 1) + L.KH);
                const size_t bytes = (size_t)nasm->batch_size * PH * PW * 4 * sizeof(float);
                CUDA_TRY(cudaMalloc(&dn->padded_in, bytes + 256));
                CUDA_TRY(cudaMemsetAsync(dn->padded_in, 0, bytes + 256, e->stream));
                dn->pin_ph = PH; dn->pin_pw = PW; dn->pin_pad = L.pad; dn->pin_ic = l.params[IN_C]; dn->pin_ih = L.IH; dn->pin_iw = L.IW;
                L.tap_sx = 1; L.tap_pad = 0;
                L.amap = add_im2col_map(dn->padded_in, {form.c, L.OW, s_ * (L.OH - 1) + L.KH, nasm->batch_size}, {(size_t)s_ * 4, (size_t)PW * 4, (size_t)PH * PW * 4},
                                        0, 0, 1 - (int)L.KH, 1, s_, L.a_rows);
            } else {
                L.tap_sx = L.stride; L.tap_pad = L.pad;
                L.amap = add_im2col_map(L.in0, {form.c, L.IW, L.IH, nasm->batch_size}, {L.ld0, (size_t)L.IW * L.ld0, (size_t)L.IH * L.IW * L.ld0}, -(int)L.pad,
                                        (int)L.pad - (int)L.KW + 1, (int)L.pad - (int)L.KH + 1, L.stride, L.stride, L.a_rows);
            }
            if (L.amap < 0) L.a_kind = A_NONE;      // a shape that the driver does not take: fp32 blocks
        } else if (form.kind == A_TMA && (l.type == MATMUL_LAYER || l.type == CONV_LAYER)) {
            add_x_map(L, L.in0, L.H0, W0, (cuuint64_t)L.ld0 * sizeof(float));
        } else if (l.type == FC_LAYER && (L.ld0 == L.IC || L.KH * L.KW == 1)) {
            // a sample's NHWC activations are one contiguous row of K values (own tiles may leave more rows between its columns)
            add_x_map(L, L.in0, L.K, nasm->batch_size, (cuuint64_t)L.IH * L.IW * L.ld0 * sizeof(float));
        } else if (l.type == K_ATTENTION_LAYER) {
            const cuuint64_t W1 = nasm->ldata[p1].out_mat_dims[OUT_W];
            if (th < L.seq || L.H0 != L.heads * L.hd || L.H1 != L.H0) {
                // tiles of a part of the keys: the softmax needs them all
            } else if (form.kind == A_TMA) {
                add_x_map(L, L.in0, L.H0, W0, (cuuint64_t)L.ld0 * sizeof(float));
                L.wmap = add_map(L.in1, L.H1, W1, (cuuint64_t)L.ld1 * sizeof(float), L.b_rows, L.per_stage);
            } else if (form.kind == A_HEAD) {
                L.a_kind = A_HEAD;
                L.amap = add_head_map(L.in0, L, W0, L.ld0, L.a_rows);
                L.wmap = add_head_map(L.in1, L, W1, L.ld1, L.b_rows);
            }
        } else if (l.type == V_ATTENTION_LAYER && form.kind == A_TMA && aligned_out && p1 != (unsigned)-1 && p1 < i && nasm->ldata[p1].layer->type != K_ATTENTION_LAYER) {
            // The value operand W(m, k) = V[token k][feature m] is the transpose of how the values' layer stores its output; that
            // layer writes a second, transposed copy into scratch memory: in the epilogue of a tensor-core projection, else by a loop
            // over the stored tile.  Several attention_v layers over the same values share it.
            const size_t seqp = round_up(L.seq, 32), ldt = seqp * nasm->batch_size;
            LayerDev &V = layers[p1];
            if (!V.vt_out) {
                CUDA_TRY(cudaMalloc(&V.vt_out, (size_t)L.H1 * ldt * sizeof(float) + 256));
                dn->scratch.push_back(V.vt_out);
                CUDA_TRY(cudaMemsetAsync(V.vt_out, 0, (size_t)L.H1 * ldt * sizeof(float) + 256, e->stream));
                V.vt_ld = (unsigned)ldt;
                V.vt_seq = (unsigned)seqp;
            }
            L.wmap = add_map(V.vt_out, ldt, L.H1, (cuuint64_t)ldt * sizeof(float), L.b_rows, L.per_stage);
            L.masked = nasm->ldata[p0].layer->type == K_ATTENTION_LAYER && layers[p0].tc && layers[p0].masked;   // its probabilities after the mask are zeros
            L.vt_seq = (unsigned)seqp;
            add_x_map(L, L.in0, L.H0, W0, (cuuint64_t)L.ld0 * sizeof(float));
        }
        if (gemm_w && L.a_kind != A_NONE && L.amap >= 0)
            L.wmap = add_map(L.weight, L.Kpad, layer_weight_rows(&l), (cuuint64_t)L.Kpad * sizeof(float), L.b_rows, L.per_stage);
        L.tc = L.a_kind != A_NONE && L.amap >= 0 && L.wmap >= 0 && aligned_out;
        if (!L.tc) { L.weight = dense; L.Kpad = dense_kpad; }       // fp32 blocks walk the taps as they are
        // ASPEN_B200_ATTN_FUSE=1 with hidden states given up: attention probabilities that only the attention_v layer reads do not
        // stay; every such layer writes the same scratch matrix, which then lives in L2.  The layer's keys have to follow from
        // the attention outputs of the layer before through per-token layers, one of which reads whole columns:
        // all of a sample's probabilities have then been read before the next layer's are written.
        const char *drop_probs = getenv("ASPEN_B200_ATTN_FUSE");
        if (l.type == K_ATTENTION_LAYER && L.tc && drop_probs && atoi(drop_probs) != 0 && !keep_hidden_states() && i != nasm->num_ldata - 1 &&
            (!probs || follows(nasm, p1, probs_reader, false))) {
            unsigned readers = 0, v_readers = 0, reader = 0;
            for (unsigned j = 1; j < nasm->num_ldata; j++)
                for (int k = PARENT_0; k <= PARENT_1; k++)
                    if (nasm->ldata[j].parent_ldata_idx_arr[k] == i) { readers++; if (k == PARENT_0 && nasm->ldata[j].layer->type == V_ATTENTION_LAYER) { v_readers++; reader = j; } }
            const size_t bytes = nasm->ldata[i].out_mat_mem_size + 256;
            if (readers == 1 && v_readers == 1 && (!probs || bytes == probs_bytes)) {
                if (!probs) {
                    CUDA_TRY(cudaMalloc(&probs, bytes));
                    dn->scratch.push_back(probs);
                    CUDA_TRY(cudaMemsetAsync(probs, 0, bytes, e->stream));
                    probs_bytes = bytes;
                }
                L.out = probs;
                probs_reader = reader;
                moved[i] = probs;
            }
        }
    }
    if (e->precision == 0) {
        for (unsigned i = 0; i < nasm->num_ldata; i++) {
            const LAYER_TYPE t = nasm->ldata[i].layer->type;
            if (t == CONV_LAYER || t == FC_LAYER || t == MATMUL_LAYER || t == K_ATTENTION_LAYER || t == V_ATTENTION_LAYER)
                for (int k = PARENT_0; k <= PARENT_1; k++) {
                    unsigned par = nasm->ldata[i].parent_ldata_idx_arr[k];
                    if (par != (unsigned)-1) layers[par].round_out = 1;
                }
        }
    }
    dn->round_input = layers[0].round_out != 0;
    for (LayerDev &L : layers) {
        const bool contraction = L.type == CONV_LAYER || L.type == FC_LAYER || L.type == MATMUL_LAYER || L.type == K_ATTENTION_LAYER || L.type == V_ATTENTION_LAYER;
        L.meets = L.tc ? L.type == K_ATTENTION_LAYER : L.vt_out != nullptr || (contraction && !L.gemv);
    }
    // Residual fusion (tensor-core path): a residual layer whose later parent is a convolution or a matmul
    // is computed in that parent's epilogue, which then needs the earlier parent's tiles of the same region
    // (fused_other[producer] = that layer).  The residual layer's own tiles leave the device
    // graph.  ASPEN_B200_NO_FUSE=1 keeps the layers separate.
    std::vector<unsigned> fused_other(nasm->num_ldata, (unsigned)-1);
    std::vector<unsigned> written_by(nasm->num_ldata, (unsigned)-1);      // residual layer -> the layer whose tiles write it
    const char *no_fuse = getenv("ASPEN_B200_NO_FUSE");
    if (e->precision == 0 && !(no_fuse && atoi(no_fuse) != 0)) {
        for (unsigned i = 1; i < nasm->num_ldata; i++) {
            if (nasm->ldata[i].layer->type != RESIDUAL_LAYER) continue;
            const unsigned a = nasm->ldata[i].parent_ldata_idx_arr[PARENT_0], b = nasm->ldata[i].parent_ldata_idx_arr[PARENT_1];
            if (a == (unsigned)-1 || b == (unsigned)-1 || a == b) continue;
            const unsigned hi = std::max(a, b), lo = std::min(a, b);
            const LAYER_TYPE t = nasm->ldata[hi].layer->type;
            if ((t != CONV_LAYER && t != MATMUL_LAYER) || !layers[hi].tc || layers[hi].res_out || layers[hi].vt_out || layers[i].vt_out) continue;
            const nasm_ldata_t &R = nasm->ldata[i], &P = nasm->ldata[hi], &Q = nasm->ldata[lo];
            if (P.out_mat_dims[OUT_H] != R.out_mat_dims[OUT_H] || P.out_mat_dims[OUT_W] != R.out_mat_dims[OUT_W] ||
                Q.out_mat_dims[OUT_H] != R.out_mat_dims[OUT_H] || Q.out_mat_dims[OUT_W] != R.out_mat_dims[OUT_W])
                continue;
            LayerDev &L = layers[hi];
            L.res_in = layers[lo].out; L.res_ld_in = layers[lo].ldc;
            L.res_out = layers[i].out; L.res_ld_out = layers[i].ldc;
            L.res_act = layers[i].act; L.res_round = layers[i].round_out;
            // The producer's own (pre-add) output: the reference frees it as soon as the residual layer has read it
            // (src/dse.c:84-92).  When nothing else reads it and the caller has not asked for every hidden state,
            // it is not written at all.
            bool only_reader = true;
            for (unsigned j = 1; j < nasm->num_ldata; j++)
                if (j != i && (nasm->ldata[j].parent_ldata_idx_arr[PARENT_0] == hi || nasm->ldata[j].parent_ldata_idx_arr[PARENT_1] == hi)) only_reader = false;
            L.res_elide = (!keep_hidden_states() && only_reader && hi != nasm->num_ldata - 1) ? 1u : 0u;
            fused_other[hi] = lo;
            written_by[i] = hi;
        }
    }
    if (to_device(&dn->layers, layers) != 0) return -1;
    {
        size_t bytes = std::max<size_t>(maps.size(), 1) * sizeof(CUtensorMap);
        CUDA_TRY(cudaMalloc(&dn->wmaps, bytes));
        if (!maps.empty()) CUDA_TRY(cudaMemcpy(dn->wmaps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
    }

    // Tiles, children (CSR).
    const unsigned n = nasm->num_ninst, n_input = nasm->ldata[0].num_ninst;
    std::vector<TileDev> tiles(n);
    size_t parts = 0;                   // sums of layers whose k is split: floats
    std::vector<size_t> cells;          // where those of each set of tiles start
    std::vector<unsigned> cell_of(n);
    std::vector<unsigned> need(n);
    std::vector<std::vector<unsigned>> kids(n);
    bool fused = false;
    for (unsigned i = 0; i < nasm->num_ldata; i++) fused = fused || written_by[i] != (unsigned)-1;
    for (unsigned t = 0; t < n; t++) {
        const ninst_t &ni = nasm->ninst[t];
        TileDev &T = tiles[t];
        T.layer = (unsigned)(ni.ldata - nasm->ldata.data());
        T.pos_h = ni.out_mat_pos[OUT_H]; T.pos_w = ni.out_mat_pos[OUT_W];
        T.tile_h = ni.tile_dims[OUT_H]; T.tile_w = ni.tile_dims[OUT_W];
        const LayerDev &L = layers[T.layer];
        T.slices = ni.ldata->slices;
        T.slice = T.slices > 1 ? (t - ni.ldata->ninst_start) % T.slices : 0;
        // whole steps of the fp32 blocks of the tile's shape (tile_gemm_ffma)
        const unsigned unit = T.tile_w > 32 && T.tile_h > 64 ? 32 : T.tile_w > 32 && T.tile_h > 32 ? 64 : 128, steps = (L.K + unit - 1) / unit;
        T.k0 = (unsigned)((unsigned long long)steps * T.slice / T.slices) * unit;
        T.k1 = T.slice + 1 == T.slices ? 0xffffffffu : (unsigned)((unsigned long long)steps * (T.slice + 1) / T.slices) * unit;
        T.part = nullptr; T.arrived = nullptr;
        if (T.slices > 1) {
            if (T.slice == 0) { cells.push_back(parts); parts += (size_t)T.slices * T.tile_w * round_up(T.tile_h, 4); }
            cell_of[t] = (unsigned)cells.size() - 1;
        }
        for (unsigned par : ni.parent_ninst_idx)
            if (par >= n || par >= t) { ASPEN_ERR("tile %u lists parent %u that does not precede it\n", t, par); return -1; }
        for (unsigned par : ni.extra_parent_idx)
            if (par >= n || par >= t) { ASPEN_ERR("tile %u lists parent %u that does not precede it\n", t, par); return -1; }
        for (unsigned child : ni.child_ninst_idx)
            if (child >= n || child <= t) { ASPEN_ERR("tile %u lists child %u that does not follow it\n", t, child); return -1; }
    }
    unsigned n_bypassed = 0;
    if (!fused) {
        // A tile's count to reach is the length of its parent list plus the true-dependency supplement; the edges walked
        // at completion are the host child lists (as the reference walks child_ninst_arr, src/dse.c:372-375) plus the
        // supplement.  For a generated graph the two agree; a file whose lists disagree yields a tile that
        // never becomes ready, which the scheduler reports as a stall.
        for (unsigned t = 0; t < n; t++) {
            const ninst_t &ni = nasm->ninst[t];
            need[t] = (unsigned)(ni.parent_ninst_idx.size() + ni.extra_parent_idx.size());
            kids[t].insert(kids[t].end(), ni.child_ninst_idx.begin(), ni.child_ninst_idx.end());
            for (unsigned par : ni.extra_parent_idx) kids[par].push_back(t);
        }
    } else {
        // Fused residual layers: their tiles leave the graph (the producer's tiles write their values), so whoever reads them
        // waits for the producer's tiles instead; the producer's tiles also wait for the other operand over their own region.
        std::vector<std::vector<unsigned>> pars(n);
        for (unsigned t = 0; t < n; t++) {
            const ninst_t &ni = nasm->ninst[t];
            const TileDev &T = tiles[t];
            std::vector<unsigned> &list = pars[t];
            const unsigned producer = written_by[T.layer];
            auto reads = [&](unsigned par) {
                if (producer != (unsigned)-1 && tiles[par].layer != producer) return;     // the producer waits for the rest
                if (written_by[tiles[par].layer] != (unsigned)-1) list.insert(list.end(), pars[par].begin(), pars[par].end());
                else list.push_back(par);
            };
            for (unsigned par : ni.parent_ninst_idx) reads(par);
            for (unsigned par : ni.extra_parent_idx) reads(par);
            if (fused_other[T.layer] != (unsigned)-1) {
                // tiles of that layer's grid (rows fastest) that overlap this tile's region
                const nasm_ldata_t &Q = nasm->ldata[fused_other[T.layer]];
                const unsigned qh = Q.ninst_tile_dims[OUT_H], qw = Q.ninst_tile_dims[OUT_W];
                const unsigned per_col = (Q.out_mat_dims[OUT_H] + qh - 1) / qh;
                for (unsigned cw = T.pos_w / qw; cw <= (T.pos_w + T.tile_w - 1) / qw; cw++)
                    for (unsigned ch = T.pos_h / qh; ch <= (T.pos_h + T.tile_h - 1) / qh; ch++) {
                        const unsigned par = Q.ninst_start + cw * per_col + ch;            // residuals are fused where k is not split
                        if (par >= Q.ninst_start + Q.num_ninst || par >= t) { ASPEN_ERR("fused residual: tile %u has no valid producer tile\n", t); return -1; }
                        reads(par);
                    }
            }
            std::sort(list.begin(), list.end());
            list.erase(std::unique(list.begin(), list.end()), list.end());
            if (producer != (unsigned)-1) { n_bypassed++; continue; }
            need[t] = (unsigned)list.size();
            for (unsigned par : list) kids[par].push_back(t);
        }
    }
    for (unsigned t = n_input; t < n; t++)
        if (need[t] == 0 && written_by[tiles[t].layer] == (unsigned)-1) { ASPEN_ERR("tile %u of layer %u has no parents and can never run\n", t, tiles[t].layer); return -1; }
    std::vector<unsigned> children;   // pairs: (child tile, its layer << 16 | count it waits for)
    for (unsigned t = 0; t < n; t++) {
        tiles[t].child_off = (unsigned)(children.size() / 2);
        tiles[t].child_cnt = (unsigned)kids[t].size();
        for (unsigned c : kids[t]) {
            if (need[c] > 0xffffu || tiles[c].layer > 0xffffu) { ASPEN_ERR("tile %u waits for %u tiles: more than the scheduler counts\n", c, need[c]); return -1; }
            children.push_back(c); children.push_back(tiles[c].layer << 16 | need[c]);
        }
    }
    CUDA_TRY(cudaMalloc(&dn->dep, std::max<size_t>(n + cells.size(), 1) * sizeof(unsigned)));
    float *part = nullptr;
    if (parts) {
        CUDA_TRY(cudaMalloc(&part, parts * sizeof(float)));
        dn->scratch.push_back(part);
    }
    for (unsigned t = 0; t < n; t++) {
        tiles[t].need = need[t];
        if (tiles[t].slices > 1) { tiles[t].part = part + cells[cell_of[t]]; tiles[t].arrived = dn->dep + n + cell_of[t]; }
    }
    if (to_device(&dn->tiles, tiles) != 0 || to_device(&dn->children, children) != 0) return -1;
    std::vector<bool> bypassed(n);
    dn->tile_layer.resize(n);
    for (unsigned t = 0; t < n; t++) { dn->tile_layer[t] = tiles[t].layer; bypassed[t] = written_by[tiles[t].layer] != (unsigned)-1; }
    dn->claims = claim_order(nasm, e->precision, e->n_ctas, kids, need, bypassed);
    std::vector<sched::Entry> order;
    for (unsigned t : dn->claims.tile) order.push_back(sched::make_entry(t, 0, tiles[t].layer));
    if (to_device(&dn->order, order) != 0) return -1;
    static std::atomic<unsigned long long> serials{0};
    dn->serial = ++serials;
    CUDA_TRY(cudaHostAlloc(&dn->svc_done_h, sizeof(unsigned), cudaHostAllocMapped));
    *dn->svc_done_h = 0;
    CUDA_TRY(cudaHostGetDevicePointer(&dn->svc_done_d, dn->svc_done_h, 0));
    CUDA_TRY(cudaMalloc(&dn->svc_d, SVC_WORDS * sizeof(unsigned)));
    CUDA_TRY(cudaMemset(dn->svc_d, 0, SVC_WORDS * sizeof(unsigned)));
    const nasm_ldata_t &l0 = nasm->ldata[0];
    if (l0.out_mat_stride != l0.out_mat_dims[OUT_H])
        CUDA_TRY(cudaMalloc(&dn->in_stage, std::max<size_t>((size_t)l0.out_mat_dims[OUT_H] * l0.out_mat_dims[OUT_W], 1) * sizeof(float)));
    const nasm_ldata_t &last = nasm->ldata[nasm->num_ldata - 1];      // the result, which may be read beside a resident kernel
    e->copy->prepare((size_t)last.out_mat_dims[OUT_H] * last.out_mat_dims[OUT_W] * sizeof(float));
    NasmDev &H = dn->host;
    memset(&H, 0, sizeof H);
    H.layers = dn->layers; H.tiles = dn->tiles; H.children = dn->children; H.dep = dn->dep; H.wmaps = dn->wmaps;
    H.completed = dn->svc_done_d; H.svc = dn->svc_d;
    H.n_tiles = n; H.n_counters = n + (unsigned)cells.size(); H.n_exec = n - n_bypassed; H.n_input = n_input;
    return 0;
}

// ---- passes -----------------------------------------------------------------------------------------------------------
// A graph's input is given with rpool_add_nasm* (or kept, rpool_reset_nasm): that asks for one more pass of it (svc_armed).
// A launch serves the passes its graphs owe (svc_armed against the mapped word svc_done_h the device writes).
//   per launch (default)   dse_group_run launches the kernel for the graphs that owe a pass; it leaves when they are complete.
//   service mode           dse_group_run launches it over every graph of the pool and it stays resident: rpool_add_nasm* on a
//                          graph it serves uploads the input on the transfer stream and then writes the graph's pass
//                          number to the device with a 4-byte copy on the same stream; dse_wait_for_nasm_completion polls
//                          the mapped word; dse_group_stop asks the kernel to leave and waits for it.  The kernel also
//                          leaves by itself (idle, or the queue of the launch used up); whoever next runs or waits
//                          launches it again when passes are still owed.
// A pass cut short (stop, relaunch) simply starts over: it only reads its input and writes its own matrices.
// Nothing that allocates or frees device memory, and no kernel, may be issued while a service kernel is resident: those
// paths stop it first.
static bool svc_done(const DeviceNasm *dn) { return *(volatile unsigned *)dn->svc_done_h == dn->svc_armed; }

// Waits for the kernel to end; `halt`: asks it to first (service mode: once nothing is owed, else after the tiles in work).
static int svc_join(Engine *e, bool halt) {
    if (!e->svc_live) return 0;
    bool owed = false;
    // per launch, a kernel whose passes are all complete is about to leave by itself
    for (const nasm_t *n : e->svc_graphs) owed = owed || !svc_done(n->dev);
    if (halt && (owed || e->service) && cudaStreamQuery(e->stream) == cudaErrorNotReady) {
        const unsigned one = 1;
        cudaMemcpyAsync(e->service ? &e->ctrl->svc_stop : &e->ctrl->stop, &one, sizeof(unsigned), cudaMemcpyHostToDevice, e->side);
        // the write must have landed (or been dropped by a kernel that had already left) before the next launch clears the word
        cudaStreamSynchronize(e->side);
    }
    cudaError_t err = cudaStreamSynchronize(e->stream);
    if (e->service) cudaStreamSynchronize(e->io);
    e->svc_live = false;
    e->svc_graphs.clear();
    if (err != cudaSuccess) { ASPEN_ERR("CUDA error after a run: %s\n", cudaGetErrorString(err)); e->status_h->status = ASPEN_B200_ERR_CUDA; return -1; }
    return 0;
}
static int svc_halt(Engine *e) { return svc_join(e, e->service); }

// The graph's entry in a launch (constant while its image lives; token or packed input may change it).
static NasmDev graph_image(const nasm_t *nasm) {
    const DeviceNasm *dn = nasm->dev;
    NasmDev G = dn->host;
    InputDev &I = G.input;
    memset(&I, 0, sizeof I);
    I.round = dn->round_input ? 1u : 0u;
    if (dn->svc_ids) {
        I.ids = dn->ids_stage; I.emb_tok = dn->dd->emb_token; I.emb_pos = dn->dd->emb_position;
        I.emb_vocab = nasm->dnn->emb_vocab; I.emb_seq = nasm->tr_seq_len ? nasm->tr_seq_len : 1u;
    } else I.stage = dn->in_stage;
    I.padded = dn->padded_in; I.IC = dn->pin_ic; I.IH = dn->pin_ih; I.IW = dn->pin_iw; I.PH = dn->pin_ph; I.PW = dn->pin_pw; I.pad = dn->pin_pad;
    return G;
}

// The order of a launch of several graphs.
static sched::Entry *merge_orders(Engine *e, const std::vector<nasm_t *> &graphs, unsigned claims) {
    std::vector<unsigned long long> of;
    for (const nasm_t *n : graphs) of.push_back(n->dev->serial);
    if (MergedOrder *known = e->orders.find(of)) return known->tiles;
    std::vector<const ClaimOrder *> each;
    for (const nasm_t *n : graphs) each.push_back(&n->dev->claims);
    std::vector<sched::Entry> order;
    order.reserve(claims);
    for (const Claim &c : merge_claims(each)) order.push_back(sched::make_entry(c.tile, c.graph, graphs[c.graph]->dev->tile_layer[c.tile]));
    // With more sets than are kept the memory of one that goes is used again: cudaFree would wait for all that runs on the device.  Whatever
    // launch read it is ahead on the stream.
    MergedOrder made;
    e->orders.make_room(made);
    if (claims > made.cap) {
        free_order(made);
        made = MergedOrder();
        if (cudaMalloc(&made.tiles, (size_t)claims * sizeof(sched::Entry)) == cudaSuccess) made.cap = claims;
    }
    // cudaMemcpyAsync from pageable memory returns after the source has been staged
    if (claims > made.cap || cudaMemcpyAsync(made.tiles, order.data(), order.size() * sizeof(sched::Entry), cudaMemcpyHostToDevice, e->stream) != cudaSuccess) {
        ASPEN_ERR("CUDA error for the order of a launch: %s\n", cudaGetErrorString(cudaGetLastError()));
        free_order(made);
        return nullptr;
    }
    e->orders.put(of, made);
    return made.tiles;
}

// `leave`: the kernel ends when the passes owed now are complete.  `chained`: the launch follows others on the stream that
// complete everything asked for before svc_chain (timing loops).
static int svc_launch(Engine *e, const std::vector<nasm_t *> &graphs, bool leave, bool chained = false) {
    unsigned long long total = 0, owed = 0;
    std::vector<NasmDev> images(graphs.size());
    for (size_t i = 0; i < graphs.size(); i++) {
        const DeviceNasm *dn = graphs[i]->dev;
        images[i] = graph_image(graphs[i]);
        total += dn->host.n_tiles;
        owed += (unsigned long long)dn->host.n_tiles * (dn->svc_armed - (chained ? dn->svc_chain : *(volatile unsigned *)dn->svc_done_h));
    }
    if (total >= (1u << 30) || graphs.size() > 0xffffu) { ASPEN_ERR("too many tiles or graphs in one launch\n"); return -1; }
    // Queue of the launch: what is owed now, or room for a number of passes; when it is used up the kernel leaves and is
    // launched again.  (A pass starts only while a whole round of passes still fits.)
    const unsigned long long room = std::max<unsigned long long>(4ull * total, std::min<unsigned long long>(256ull * total, 2u << 20));
    const unsigned cap = (unsigned)(leave ? std::min(room, owed + total) : room);
    if (graphs.size() > e->nasms_cap) {
        cudaFree(e->nasms_d);
        e->nasms_d = nullptr;
        e->nasms_cap = 0;
        e->uploaded.clear();
        CUDA_TRY(cudaMalloc(&e->nasms_d, graphs.size() * sizeof(NasmDev)));
        e->nasms_cap = (unsigned)graphs.size();
    }
    // A launch that leaves hands its tiles out in a fixed order; service mode's queue takes them as they become ready.
    const bool ordered = !e->service;
    sched::Entry *order = nullptr;
    unsigned claims = 0;
    if (ordered) {
        for (const nasm_t *n : graphs) claims += (unsigned)n->dev->claims.tile.size();
        if (graphs.size() == 1) order = graphs[0]->dev->order;
        else if (!(order = merge_orders(e, graphs, claims))) return -1;
    } else if (cap > e->queue_cap) {
        cudaFree(e->queue);
        e->queue = nullptr;
        e->queue_cap = 0;
        CUDA_TRY(cudaMalloc(&e->queue, (size_t)cap * sizeof(sched::Entry)));
        e->queue_cap = cap;
    }
    if (images.size() != e->uploaded.size() || memcmp(images.data(), e->uploaded.data(), images.size() * sizeof(NasmDev)) != 0) {
        // cudaMemcpyAsync from pageable memory returns after the source has been staged
        CUDA_TRY(cudaMemcpyAsync(e->nasms_d, images.data(), images.size() * sizeof(NasmDev), cudaMemcpyHostToDevice, e->stream));
        e->uploaded = images;
    }
    e->status_h->status = 0;
    for (unsigned g0 = 0; g0 < graphs.size(); g0 += sched::ARM_GRAPHS) {
        sched::ArmArgs a;
        a.g0 = g0; a.n = std::min<unsigned>(sched::ARM_GRAPHS, (unsigned)graphs.size() - g0); a.n_nasm = (unsigned)graphs.size();
        a.cap = ordered ? claims : cap; a.total = (unsigned)total; a.svc_stop = leave ? 1u : 0u; a.ahead = ordered ? graphs.size() > 1 : e->svc_ahead; a.ordered = ordered ? 1u : 0u;
        a.stall_ns = e->stall_ns; a.pipe_ns = e->pipe_ns; a.idle_ns = e->idle_ns;
        for (unsigned i = 0; i < a.n; i++) {
            const DeviceNasm *dn = graphs[g0 + i]->dev;
            a.base[i] = chained ? dn->svc_chain : *(volatile unsigned *)dn->svc_done_h;
            a.target[i] = dn->svc_armed;
        }
        sched::arm_kernel<<<std::min<unsigned>((a.cap + 255) / 256, 1024), 256, 0, e->stream>>>(e->nasms_d, e->ctrl, e->queue, a);
        e->launches++;
    }
    if (e->service) {
        // pass numbers written later (transfer stream) must not be overtaken by the ones above
        CUDA_TRY(cudaEventRecord(e->svc_armed_ev, e->stream));
        CUDA_TRY(cudaStreamWaitEvent(e->io, e->svc_armed_ev, 0));
    }
    if (e->precision == 0)
        sched::scheduler_kernel<true><<<e->n_ctas, sched::threads<true>(), e->smem_bytes, e->stream>>>(e->nasms_d, e->ctrl, ordered ? order : e->queue, e->status_d, e->prof);
    else
        fp32_launch(e->n_ctas, e->smem_bytes, e->stream, e->nasms_d, e->ctrl, ordered ? order : e->queue, e->status_d, e->prof);
    e->launches++;
    CUDA_TRY(cudaGetLastError());
    e->svc_graphs = graphs;
    e->svc_live = true;
    e->uploading = false;
    return 0;
}

static void svc_pool_add(Engine *e, const std::vector<nasm_t *> &nasms) {
    for (nasm_t *n : nasms)
        if (n->dev && n->dev->e == e && std::find(e->svc_pool.begin(), e->svc_pool.end(), n) == e->svc_pool.end()) e->svc_pool.push_back(n);
}
static bool svc_serves(Engine *e, const nasm_t *nasm) {
    return e->svc_live && std::find(e->svc_graphs.begin(), e->svc_graphs.end(), nasm) != e->svc_graphs.end();
}

int engine_run(Engine *e, const std::vector<nasm_t *> &nasms) {
    if (!e) return -1;
    CUDA_TRY(cudaSetDevice(e->device));
    svc_pool_add(e, nasms);
    if (e->svc_live) {
        bool served = e->service && cudaStreamQuery(e->stream) == cudaErrorNotReady;
        for (nasm_t *n : e->svc_pool) served = served && svc_serves(e, n);
        if (served) return 0;         // the passes asked for since were signalled to the resident kernel
        if (svc_join(e, e->service) != 0) return -1;   // one kernel at a time per group: the graphs that owe a pass join the next launch
    }
    std::vector<nasm_t *> graphs;
    bool owed = false;
    for (nasm_t *n : e->svc_pool) {
        const bool owes = !svc_done(n->dev);
        owed = owed || owes;
        if (owes || e->service) graphs.push_back(n);
    }
    return owed ? svc_launch(e, graphs, !e->service) : 0;
}

int engine_stop(Engine *e) {
    if (!e || !e->svc_live) return 0;
    CUDA_TRY(cudaSetDevice(e->device));
    return svc_join(e, true);
}

unsigned int engine_poll_nasm(nasm_t *nasm) { return nasm->dev && nasm->dev->svc_armed && svc_done(nasm->dev) ? 1u : 0u; }

int engine_wait_nasm(nasm_t *nasm) {
    DeviceNasm *dn = nasm->dev;
    if (!dn) return -1;
    Engine *e = dn->e;
    unsigned relaunches = 0;
    for (unsigned spin = 0;; spin++) {
        if (svc_done(dn)) return 0;
        if ((spin & 63u) == 0u) {     // the word in host memory is polled; the driver is asked now and then
            if (spin == 0u) cudaSetDevice(e->device);
            if (e->status_h->status != 0) return -1;
            cudaError_t q = svc_serves(e, nasm) ? cudaStreamQuery(e->stream) : cudaSuccess;
            if (q == cudaSuccess) {
                if (svc_done(dn)) return 0;
                if (e->status_h->status != 0) return -1;
                // No kernel serves the graph.  Per launch: it was never run, or the run was stopped.  Service mode: never launched
                // for it, or it left (idle, queue used up, a request that just missed it): launch for everything that is
                // owed.  Every launch completes at least the pass it was launched for unless it reports an
                // error, so many launches in a row without this graph completing are a fault.
                if (!e->service) return -1;
                if (++relaunches > 1000u) { ASPEN_ERR("service mode: the graph's pass does not complete\n"); return -1; }
                if (svc_halt(e) != 0 || svc_launch(e, e->svc_pool, false) != 0) return -1;
            } else if (q != cudaErrorNotReady) {
                ASPEN_ERR("CUDA error while waiting: %s\n", cudaGetErrorString(q));
                e->status_h->status = ASPEN_B200_ERR_CUDA;
                return -1;
            }
            if (spin > 4096u) sched_yield();
        }
    }
}

static int upload_embedding(DeviceDnn *dd, const aspen_dnn_t *dnn) {
    if (dd->emb_token) return 0;
    CUDA_TRY(cudaMalloc(&dd->emb_token, dnn->emb_token.size() * sizeof(float)));
    CUDA_TRY(cudaMemcpy(dd->emb_token, dnn->emb_token.data(), dnn->emb_token.size() * sizeof(float), cudaMemcpyHostToDevice));
    if (!dnn->emb_position.empty()) {
        CUDA_TRY(cudaMalloc(&dd->emb_position, dnn->emb_position.size() * sizeof(float)));
        CUDA_TRY(cudaMemcpy(dd->emb_position, dnn->emb_position.data(), dnn->emb_position.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
    return 0;
}

// Host to device, complete (or staged by the driver) on return: the caller may reuse its buffer.  With no kernel of the group in
// flight a pageable source is copied in stream order ahead of the next launch, without waiting for the DMA; otherwise on
// the transfer stream, beside a running kernel.
static cudaError_t upload(Engine *e, void *dst, const void *src, size_t bytes) {
    cudaPointerAttributes attr;
    const bool pageable = cudaPointerGetAttributes(&attr, src) == cudaSuccess && attr.type == cudaMemoryTypeUnregistered;
    if (pageable && !e->service && !e->svc_live) {
        e->uploading = true;
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, e->stream);
    }
    const cudaError_t err = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, e->io);
    return err != cudaSuccess ? err : cudaStreamSynchronize(e->io);
}

// rpool_add_nasm*: uploads (input_host, or ids_host, or neither: zeros; keep_input: what the graph holds) and asks for a pass.
static int attach(Engine *e, nasm_t *nasm, const void *input_host, const int *ids_host, bool keep_input) {
    CUDA_TRY(cudaSetDevice(e->device));
    if (nasm->dev && nasm->dev->e != e) { if (svc_halt(e) != 0) return -1; engine_detach_nasm(nasm); }
    if (!nasm->dev) {
        if (svc_halt(e) != 0) return -1;
        if (build_device_nasm(e, nasm) != 0) { engine_detach_nasm(nasm); return -1; }
        CUDA_TRY(cudaStreamSynchronize(e->stream));   // the image (zeroed arena, descriptors) is in place before the transfer stream touches it
    }
    DeviceNasm *dn = nasm->dev;
    svc_pool_add(e, std::vector<nasm_t *>{nasm});
    // a pass that is owed or running: in service mode its input must stay until it is complete; per launch only a running one counts
    if (!svc_done(dn)) {
        if (e->service) { if (engine_wait_nasm(nasm) != 0) return -1; }
        else if (svc_serves(e, nasm) && svc_join(e, false) != 0) return -1;
    }
    const nasm_ldata_t &l0 = device_view(nasm)->ldata[0];
    const size_t n = (size_t)l0.out_mat_dims[OUT_H] * l0.out_mat_dims[OUT_W];
    float *dst = dn->in_stage ? dn->in_stage : (float *)((char *)dn->arena + dn->ldata_off[0]);
    if (ids_host) {
        aspen_dnn_t *dnn = nasm->dnn;
        const unsigned M = l0.out_mat_dims[OUT_H];
        if (dnn->emb_token.empty() || dnn->emb_width != M || M % 4 != 0 || l0.out_mat_stride % 4 != 0 || l0.ninst_tile_dims[OUT_H] % 4 != 0) {
            ASPEN_ERR("token input: the dnn has no embedding table of width %u (aspen_b200_dnn_set_embedding), or the width is not a multiple of 4\n", M);
            return -1;
        }
        if (!dnn->emb_position.empty() && nasm->tr_seq_len > dnn->emb_max_pos) {
            ASPEN_ERR("token input: sequence length %u exceeds the position table (%u rows)\n", nasm->tr_seq_len, dnn->emb_max_pos);
            return -1;
        }
        if (!dn->dd->emb_token || !dn->ids_stage || !dn->svc_ids) {
            if (svc_halt(e) != 0) return -1;          // allocations, and the graph's image changes
            if (upload_embedding(dn->dd, dnn) != 0) return -1;
            if (!dn->ids_stage) CUDA_TRY(cudaMalloc(&dn->ids_stage, (size_t)l0.out_mat_dims[OUT_W] * sizeof(int)));
            dn->svc_ids = true;
        }
        CUDA_TRY(upload(e, dn->ids_stage, ids_host, (size_t)l0.out_mat_dims[OUT_W] * sizeof(int)));
    } else if (!keep_input) {
        if (dn->svc_ids) { if (svc_halt(e) != 0) return -1; dn->svc_ids = false; }
        if (!input_host) {
            // no input: cleared on the compute stream, ahead of the graph's next run (a memset may be a kernel: a resident one leaves first)
            if (svc_halt(e) != 0) return -1;
            CUDA_TRY(cudaMemsetAsync(dst, 0, n * sizeof(float), e->stream));
            CUDA_TRY(cudaStreamSynchronize(e->stream));
        } else {
            CUDA_TRY(upload(e, dst, input_host, n * sizeof(float)));
        }
    }
    if (svc_done(dn)) dn->svc_armed++;
    if (e->service && svc_serves(e, nasm))
        CUDA_TRY(cudaMemcpyAsync(&dn->svc_d[SVC_TARGET], &dn->svc_armed, sizeof(unsigned), cudaMemcpyHostToDevice, e->io));
    return 0;
}

int engine_attach_nasm(Engine *e, nasm_t *nasm, const void *input_host) { return e ? attach(e, nasm, input_host, nullptr, false) : -1; }
int engine_attach_tokens(Engine *e, nasm_t *nasm, const int *ids_host) { return e && ids_host ? attach(e, nasm, nullptr, ids_host, false) : -1; }
int engine_rearm(Engine *e, nasm_t *nasm) { return e && nasm->dev ? attach(e, nasm, nullptr, nullptr, true) : -1; }

void engine_detach_nasm(nasm_t *nasm) {
    DeviceNasm *dn = nasm->dev;
    if (!dn) return;
    Engine *e = dn->e;
    cudaSetDevice(e->device);
    svc_halt(e);
    e->svc_pool.erase(std::remove(e->svc_pool.begin(), e->svc_pool.end(), nasm), e->svc_pool.end());
    if (dn->serial) e->orders.drop(dn->serial, free_order);
    free_device_nasm(dn);
    nasm->dev = nullptr;
}

long engine_read_ldata(nasm_t *nasm, unsigned int idx, float *out) {
    DeviceNasm *dn = nasm->dev;
    if (!dn) return -1;
    Engine *e = dn->e;
    if (cudaSetDevice(e->device) != cudaSuccess) return -1;
    const nasm_ldata_t &ld = device_view(nasm)->ldata[idx];
    const size_t n = (size_t)ld.out_mat_dims[OUT_H] * ld.out_mat_dims[OUT_W];
    const float *src = (const float *)((char *)dn->arena + dn->ldata_off[idx]);
    if (!e->service && !svc_done(dn) && svc_serves(e, nasm)) svc_join(e, false);      // the graph is being computed
    if (e->uploading && !e->svc_live) { cudaStreamSynchronize(e->stream); e->uploading = false; }
    // the copy engine packs strided matrices: a kernel could not start next to a resident one
    const size_t row = (size_t)ld.out_mat_dims[OUT_H] * sizeof(float);
    const bool packed = ld.out_mat_stride == ld.out_mat_dims[OUT_H];
    // memory for large results is pinned when one is first read with no resident kernel; beside one, dse_get_nasm_result finds what
    // its graph's image asked for when it was built
    if (!(e->service && e->svc_live)) e->copy->prepare(n * sizeof(float));
    const cudaError_t err = packed ? e->copy->down(out, src, n * sizeof(float), e->io)
        : cudaMemcpy2DAsync(out, row, src, (size_t)ld.out_mat_stride * sizeof(float), row, ld.out_mat_dims[OUT_W], cudaMemcpyDeviceToHost, e->io);
    if (err != cudaSuccess || (!packed && cudaStreamSynchronize(e->io) != cudaSuccess)) {
        ASPEN_ERR("CUDA error reading layer %u: %s\n", idx, cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    return (long)n;
}

int engine_set_service(Engine *e, int on) {
    if (!e) return -1;
    CUDA_TRY(cudaSetDevice(e->device));
    if (e->service == (on != 0)) return 0;
    if (svc_halt(e) != 0) return -1;
    if (e->service) e->svc_pool.clear();
    e->service = on != 0;
    return 0;
}

// Timing loops: passes dealt round robin inside launches that leave when they are done (`passes`), or one launch per pass of
// every graph, back to back on the compute stream.
static double timed(Engine *e, const std::vector<nasm_t *> &graphs, unsigned warmup, unsigned iters, unsigned long long *launches, bool passes) {
    cudaEvent_t t0, t1;
    if (graphs.empty() || cudaEventCreate(&t0) != cudaSuccess || cudaEventCreate(&t1) != cudaSuccess) return -1.0;
    unsigned long long l0 = e->launches;
    bool ok = true;
    if (passes) {
        for (int phase = 0; phase < 2 && ok; phase++) {
            const unsigned count = phase == 0 ? warmup : iters, m = (unsigned)graphs.size();
            for (unsigned i = 0; i < m; i++) graphs[i]->dev->svc_armed += count / m + (i < count % m ? 1u : 0u);
            if (phase == 1) { cudaEventRecord(t0, e->stream); l0 = e->launches; }
            for (unsigned tries = 0; ok && count; tries++) {
                ok = svc_launch(e, graphs, true) == 0;
                if (phase == 1) cudaEventRecord(t1, e->stream);
                ok = ok && svc_join(e, false) == 0 && e->status_h->status == 0 && tries < 100000u;   // each launch completes at least one pass
                bool done = true;
                for (nasm_t *n : graphs) done = done && svc_done(n->dev);
                if (done) break;
            }
        }
    } else {
        for (nasm_t *n : graphs) n->dev->svc_armed = n->dev->svc_chain = *(volatile unsigned *)n->dev->svc_done_h;
        for (unsigned i = 0; i < warmup + iters && ok; i++) {
            if (i == warmup) { cudaEventRecord(t0, e->stream); l0 = e->launches; }
            for (nasm_t *n : graphs) n->dev->svc_armed++;
            ok = svc_launch(e, graphs, true, true) == 0;      // arming waits for the previous run
            for (nasm_t *n : graphs) n->dev->svc_chain++;
        }
        cudaEventRecord(t1, e->stream);
        ok = svc_join(e, false) == 0 && ok;
    }
    cudaError_t err = cudaStreamSynchronize(e->stream);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, t0, t1);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (launches) *launches = e->launches - l0;
    if (!ok || err != cudaSuccess || e->status_h->status != 0) {
        ASPEN_ERR("timed runs failed: cuda=%s engine status=%u (info %u %u)\n", cudaGetErrorString(err), e->status_h->status, e->status_h->info0, e->status_h->info1);
        return -1.0;
    }
    for (nasm_t *n : graphs)
        if (!svc_done(n->dev)) { ASPEN_ERR("timed runs: a graph did not complete\n"); return -1.0; }
    return (double)ms;
}

double engine_time_runs(Engine *e, const std::vector<nasm_t *> &nasms, unsigned int warmup, unsigned int iters, unsigned long long *launches) {
    if (!e || cudaSetDevice(e->device) != cudaSuccess || svc_halt(e) != 0 || svc_join(e, false) != 0) return -1.0;
    std::vector<nasm_t *> run;
    for (nasm_t *n : nasms)
        if (n->dev && n->dev->e == e) run.push_back(n);
    return timed(e, run, warmup, iters, launches, false);
}
double engine_time_passes(Engine *e, const std::vector<nasm_t *> &nasms, unsigned int warmup, unsigned int passes, unsigned long long *launches) {
    if (!e || !e->service || cudaSetDevice(e->device) != cudaSuccess || svc_halt(e) != 0) return -1.0;
    svc_pool_add(e, nasms);
    return timed(e, e->svc_pool, warmup, passes, launches, true);
}

// Sums the per-CTA time accounting (ASPEN_B200_PROFILE=1) into out[PROF_SLOTS] and clears it.
int engine_read_profile(Engine *e, unsigned long long *out, unsigned *n_ctas) {
    if (!e || !e->prof) return -1;
    CUDA_TRY(cudaSetDevice(e->device));
    if (svc_halt(e) != 0) return -1;
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    std::vector<unsigned long long> h((size_t)e->n_ctas * sched::PROF_SLOTS);
    CUDA_TRY(cudaMemcpy(h.data(), e->prof, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemset(e->prof, 0, h.size() * sizeof(unsigned long long)));
    for (unsigned s = 0; s < sched::PROF_SLOTS; s++) out[s] = 0;
    for (unsigned c = 0; c < e->n_ctas; c++)
        for (unsigned s = 0; s < sched::PROF_SLOTS; s++) out[s] += h[(size_t)c * sched::PROF_SLOTS + s];
    if (n_ctas) *n_ctas = e->n_ctas;
    return 0;
}
