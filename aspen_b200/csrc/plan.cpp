// Device tile plan: the grid of tiles the GPU executes a graph with.
//
// A nasm's own tiles (tiler.cpp) follow the reference: their shapes are chosen for its CPU micro-kernels, they are graph node
// ids, and .nasm files name them.  Tile VALUES do not depend on the shapes, so the device image of a graph is free to use its
// own: with the reference's 64-row / 12-column quanta a 128-lane MMA would be mostly padding, and one quantum for a
// whole network leaves SMs idle in the late layers or makes the early ones pay per tile.  Here every layer gets the
// shape with the lowest estimated time on the SMs at hand.  The plan is a nasm of the same layers with that grid and
// with the parents each tile reads (by region, so a graph of ten thousand tiles takes milliseconds).
// Graphs whose lists a file has changed keep their own tiles and lists.  A plan is made for launched or for served passes, whichever
// mode the group is in when the graph's image is built; it stays when the mode changes later (the values are the same).
#include "internal.h"
#include "device_types.h"

#include <algorithm>
#include <functional>
#include <memory>
#include <queue>

namespace {

struct Grid {
    unsigned th = 1, tw = 1;       // tile rows, columns
    unsigned seg = 1;              // tiles do not cross multiples of this many columns (a head's or sample's queries)
    unsigned nh = 1, per_seg = 1;  // row tiles; column tiles of a segment
    unsigned start = 0;
    unsigned ks = 1;               // parts of k, a tile each
};

bool contraction(LAYER_TYPE t) { return t == CONV_LAYER || t == FC_LAYER || t == MATMUL_LAYER || t == K_ATTENTION_LAYER || t == V_ATTENTION_LAYER; }
unsigned ceil_div(unsigned a, unsigned b) { return (a + b - 1) / b; }

// What runs the tiles of a contraction layer.
enum Path { TENSOR, BESIDE_RING, FP32 };      // tensor cores / fp32 blocks in a tensor-core graph (no operand form) / fp32 mode

Path path_of(const aspen_layer_t *l, int precision, unsigned seq) { return precision != 0 ? FP32 : operand_form(l, seq).kind != A_NONE ? TENSOR : BESIDE_RING; }

// Estimated microseconds of one tile of th x tw outputs with a k-deep contraction, `gap` of them between two tiles of an SM.
// Tensor cores: 0.38 us for a 32-deep chunk of a 128-column block with 256 rows, 0.28 with 128 and 0.19 with 64 or less; the epilogue of a
// block takes 0.4 us per 32 rows and runs under the next block's main loop.  Measured in launched networks (layers of the same tiles, k = 768
// and 3072) a chunk takes 0.34, 0.20, 0.17 and, with 32 rows, 0.12 - 0.15 us.  The weights of the narrow ones are larger because a
// tile's time does not count what more and narrower tiles cost the rest of the chip: with 0.11 in place of 0.19 a pass of GPT-2 8 x 512 takes
// 3005 us instead of 2390, BERT 16 x 128 1714 for 1484, ResNet-50 x 32 1477 for 1379; with 0.15 2413, 1662 and 1416; with 0.15 and 0.22 (in
// place of 0.28) 2479, 1473 and 1387.
// Beside the ring (measured): 64 x 32 blocks, 0.8 us and 1.0 per 32 of k (3 x 3 layers of 48 and 24 channels), 1.6 where operands
// come value by value (attention with heads of 10); the softmax of scores 1.4 us per 1024.
// `ks` > 1: one of ks tiles that share k; they wait for each other's counts, some 3 us, each writes its sums and the last one reads all of
// them, 12 KB a us.
double tile_us(Path path, const aspen_layer_t *l, unsigned th, unsigned tw, unsigned k, double gap, unsigned ks = 1) {
    if (ks > 1) return tile_us(path, l, th, tw, ceil_div(k, ks), gap + 3.0 + 4.0 * th * tw * (ks + 1) / 12e3);
    if (path == TENSOR) {
        const unsigned chunks = ceil_div(k, 32), nb = ceil_div(tw, 128) * ceil_div(th, 256), rows = std::min(th, 256u);
        const double loop = chunks * (rows > 128 ? 0.38 : rows > 64 ? 0.28 : 0.19), epi = 0.6 + 0.4 * ceil_div(rows, 32);
        return gap + loop + epi + (nb - 1) * std::max(loop, epi);
    }
    if (path == BESIDE_RING) {
        const bool pieces = l->type == CONV_LAYER ? l->params[IN_C] % 4 == 0 : l->type == K_ATTENTION_LAYER && k % 4 == 0;
        const double softmax = l->type == K_ATTENTION_LAYER ? 1.4 * th * tw / 1024 : 0;
        return gap + ceil_div(th, 64) * ceil_div(tw, 32) * (0.8 + ceil_div(k, 32) * (pieces ? 1.0 : 1.6)) + softmax;
    }
    // fp32 blocks (gemm_ffma.cuh), shapes as tile_gemm_ffma picks them: some 3 us for filling the pipeline, the reduction and the
    // stores, then steps of 32, 64 or 128 of k.  Attention, measured: scores of 200 keys x 64 queries, k = 64, 33 us; values, staged one by one,
    // 64 x 64 with k = 50 and 200 17 and 28 us.
    const int shape = th > 64 && tw > 32 ? 0 : th > 32 && tw > 32 ? 1 : 2;
    const unsigned bm = shape == 0 ? 128 : shape == 1 ? 64 : 32, bn = shape == 2 ? 32 : 64, kt = 32u << shape;
    const bool ka = l->type == K_ATTENTION_LAYER, va = l->type == V_ATTENTION_LAYER;
    const double step = (shape == 2 ? 1.3 : 2.0) + (va ? 1.5 : 0), attention = ka ? 6.0 + 1.4 * th * tw / 1024 : va ? 11.0 : 0;
    return gap + (double)ceil_div(th, bm) * ceil_div(tw, bn) * (3.0 + ceil_div(k, kt) * step) + attention;
}

Grid choose(const nasm_ldata_t &ld, const nasm_t *nasm, int precision, unsigned sms, bool served) {
    const aspen_layer_t *l = ld.layer;
    const unsigned *p = l->params;
    const unsigned H = ld.out_mat_dims[OUT_H], W = ld.out_mat_dims[OUT_W];
    Grid g;
    g.seg = W;
    if (gemv_layer(ld)) {
        // dot products, a warp a row: two tiles per SM, none smaller than its eight warps' rows, so that every SM fetches weights
        g.th = (unsigned)round_up(std::min(64u, std::max(8u, ceil_div(H, 2 * sms))), 8);
        g.tw = W;
    } else if (contraction(l->type)) {
        const Path path = path_of(l, precision, nasm->tr_seq_len);
        const bool ka = l->type == K_ATTENTION_LAYER, va = l->type == V_ATTENTION_LAYER;
        if (ka || va) g.seg = nasm->tr_seq_len;
        unsigned hs[8], nhs = 0;
        if (ka) hs[nhs++] = H;                                      // the softmax reduces over all keys
        else if (va) hs[nhs++] = p[NUM_HEAD] ? p[NUM_HIDDEN] / p[NUM_HEAD] : H;
        else for (unsigned h : {512u, 256u, 128u, 64u, 32u}) if (h < 2 * H && (h <= 256 || path == TENSOR)) hs[nhs++] = h;
        const unsigned k = ka ? p[NUM_HIDDEN] / std::max(1u, p[NUM_HEAD]) : va ? nasm->tr_seq_len : layer_contraction_k(l);
        const unsigned quantum = path == TENSOR ? 128 : 32;
        double best = 0;
        for (unsigned i = 0; i < nhs; i++)
            for (unsigned tw = quantum; tw < g.seg + quantum && tw <= 16 * quantum; tw += quantum) {
                const unsigned tiles = ceil_div(H, hs[i]) * (W / g.seg) * ceil_div(g.seg, tw);
                const double us = tile_us(path, l, std::min(hs[i], H), std::min(tw, g.seg), k, served || path == FP32 ? 4.0 : 2.5);
                const double share = (double)tiles / sms;
                // Launched alone a layer of fewer tiles than SMs takes as long as one tile; of a larger one the last tiles run while
                // half of the chip waits.  (The work and 0.7 tiles whatever the number: ResNet-50 x 3 617 us a pass instead of 570,
                // x 32 1398 and 1373, BERT 1 x 37 799 and 772.)  Served, the passes of other graphs fill those SMs but the graphs in
                // rotation are few: the work, and a share of a tile.  What the best share is depends on their number, which a plan of one graph does
                // not know, and not on their size: up to four graphs prefer 0.5, from six on 0.3.  0.4 is at most 7 % slower than the best of the three
                // over 35 networks, sizes and numbers, 1.5 % on average (0.3: 11 and 2.9; 0.5: 10 and 1.7; 0.3 for passes of less than 100 us of work
                // and 0.5 above: 9.5 and 2.2).  Bursts of three or four requests a graph, us with 0.3 / 0.4 / 0.5 tiles: ResNet-50 x 4 with three
                // graphs 3464 / 3370 / 3164, with four 3776 / 3671 / 3630, six 4463 / 4500 / 4680, eight 6997 / 7129 / 7508; x 16 with four
                // 10647 / 10329 / 10408, eight 14420 / 14611 / 14748; x 32 with three 15399 / 14673 / 14598, six 20418 / 20417 / 20795; BERT 4 x 128 with
                // four 9640 / 10061 / 10044, eight 12249 / 13151 / 13232.
                // (fp32 mode, launched, us a pass with 0.5 and 2.5 us between two tiles as for the tensor cores, and with 0.3 and 4.0: BERT 4 x 200 6173 and
                // 5935, 6 x 128 5332 and 5040, 16 x 128 12858 and 12298, VGG-16 x 8 8379 and 8150, ResNet-50 x 4 1697 and 1655, BERT 1 x 37 1474 and 1476.)
                const double rest = path == FP32 ? 0.3 : 0.5;
                const double cost = us * (served ? share + 0.4 : std::max(1.0, share + rest));
                if (best == 0 || cost < best * 0.999) { best = cost; g.th = hs[i]; g.tw = tw; g.ks = 1; }
                // Launched alone in the fp32 mode, a layer that leaves SMs idle shares its k among them: 512 x 49 outputs with k = 4608 are 32
                // tiles of 48 us, or 128 of 14; ResNet-50 x 1 959 -> 824 us a pass, BERT 1 x 37 1508 -> 1476.  (Not on the tensor cores, where a
                // sample's bits are the same in every batch.)  The tiles of all parts count as a layer's others do: as if they cost one tile
                // however full they leave the chip, 256 x 128 tiles in three parts were chosen for 336 of 64 x 64 (BERT 2 x 200 4817 us a pass,
                // without any sharing 3897, so 3898; 3 x 50 2355, 1953, 1953; ResNet-50 x 3 1578, 1477, 1477).
                if (!served && !ka && !va && path == FP32)
                    for (unsigned ks = 2; ks <= 8 && ks * tiles <= sms && k / ks >= 128; ks++) {
                        const double split = tile_us(path, l, std::min(hs[i], H), std::min(tw, g.seg), k, 2.5, ks) * std::max(1.0, ks * share + 0.5);
                        if (split < best * 0.95) { best = split; g.th = hs[i]; g.tw = tw; g.ks = ks; }
                    }
            }
    } else if (l->type == SOFTMAX_LAYER || l->type == YOLO_LAYER || l->type == APPEND_LAYER) {
        g.th = ld.ninst_tile_dims[OUT_H]; g.tw = ld.ninst_tile_dims[OUT_W];
    } else {
        // memory-bound: whole columns, one tile per SM, more (up to four) where a tile then still writes 96 KB -- a tile costs
        // some 4 us besides its transfers; few columns with many rows (a global pool) split the rows
        g.th = H;
        const unsigned want = (unsigned)std::min(4.0 * sms, std::max(1.0 * sms, (double)H * W * 4.0 / 98304.0));
        g.tw = std::max(1u, ceil_div(W, want));
        if (g.tw > 8) g.tw = (unsigned)round_up(g.tw, 8);
        if (l->type == AVGPOOL_LAYER || l->type == MAXPOOL_LAYER)
            while (g.th > 64 && g.th % 8 == 0 && ceil_div(H, g.th) * W < want / 2) g.th /= 2;
    }
    g.nh = ceil_div(H, g.th);
    g.per_seg = ceil_div(g.seg, g.tw);
    return g;
}

}  // namespace

// Up to 8 columns a weight is worth at most 8 multiplications a load; beyond, the sums of one row no longer fit the registers beside
// the loads in flight, and a 32-column MMA tile or fp32 block takes over.
bool gemv_layer(const nasm_ldata_t &ld) {
    const unsigned *p = ld.layer->params;
    const LAYER_TYPE t = ld.layer->type;
    return ld.out_mat_dims[OUT_W] <= 8 && (t == MATMUL_LAYER || t == FC_LAYER ||
                                           (t == CONV_LAYER && p[WEIGHT_H] == 1 && p[WEIGHT_W] == 1 && p[STRIDE] <= 1 && p[PADDING] == 0));
}

OperandForm operand_form(const aspen_layer_t *l, unsigned seq) {
    const unsigned *p = l->params;
    OperandForm f;
    f.c = p[IN_C];
    switch (l->type) {
        case MATMUL_LAYER: case FC_LAYER: f.kind = A_TMA; break;
        case V_ATTENTION_LAYER:            // a tile is a head's rows and has to start on a 16-byte boundary
            if (p[NUM_HEAD] && p[NUM_HIDDEN] / p[NUM_HEAD] % 4 == 0) f.kind = A_TMA;
            break;
        case K_ATTENTION_LAYER: {
            // all keys of a query have to fit the accumulators, and a head has to start on a 16-byte boundary
            const unsigned hd = p[NUM_HEAD] ? p[NUM_HIDDEN] / p[NUM_HEAD] : 0;
            if (hd == 0 || hd % 4 != 0 || seq > 512) break;
            f.kind = hd % 32 == 0 ? A_TMA : A_HEAD;
            break;
        }
        case CONV_LAYER: {
            const unsigned stride = p[STRIDE] ? p[STRIDE] : 1;
            if (p[WEIGHT_H] == 1 && p[WEIGHT_W] == 1 && stride == 1 && p[PADDING] == 0) { f.kind = A_TMA; break; }
            // limits of an im2col tensor map; a window that lies in the padding alone is left out
            if (stride > 8 || p[WEIGHT_H] > 64 || p[WEIGHT_W] > 64 || p[PADDING] >= p[WEIGHT_H] || p[PADDING] >= p[WEIGHT_W]) break;
            f.kind = A_IM2COL;
            f.kh = p[WEIGHT_H]; f.kw = p[WEIGHT_W];
            // one convolution of a network reads the image that way (there is one padded copy): the first
            const aspen_layer_t *first = l->dnn->layers.data(), *in = l->parent_layers[PARENT_0];
            f.image = in && in->type == INPUT_LAYER && p[IN_C] <= 4;
            for (; first < l; first++)
                if (first->type == CONV_LAYER && first->parent_layers[PARENT_0] == in && operand_form(first, seq).image) f.image = false;
            if (f.image) { f.c = 4 * f.kw; f.kw = 1; }
            break;
        }
        default: break;
    }
    return f;
}

// The run is simulated with the plan's estimates: ready tiles go to the worker that is free first, in the order in which they became
// ready.  (A worker that goes on with the first child its tile made ready, as the ready queue's do: ResNet-50 x 32 1506 us a pass
// instead of 1466, GPT-2 8 x 512 2552 instead of 2461.)  Tiles whose lists cannot be satisfied come last: the scheduler reports them.
ClaimOrder claim_order(const nasm_t *plan, int precision, unsigned workers, const std::vector<std::vector<unsigned>> &children, const std::vector<unsigned> &need,
                       const std::vector<bool> &skip) {
    const unsigned n = plan->num_ninst;
    constexpr float HAND_OVER_US = 2.0f, BYTES_PER_US = 23e3f;      // last store of a tile to first load of its child; memory-bound tiles on one SM
    ClaimOrder order;
    std::vector<unsigned> left(need);
    std::vector<bool> started(n, false);
    std::queue<unsigned> ready;
    typedef std::pair<float, unsigned> Event;                       // end of a tile
    std::priority_queue<Event, std::vector<Event>, std::greater<Event>> running;
    auto us = [&](unsigned t) {
        const ninst_t &ni = plan->ninst[t];
        const aspen_layer_t *l = ni.ldata->layer;
        const unsigned th = ni.tile_dims[OUT_H], tw = ni.tile_dims[OUT_W];
        if (gemv_layer(*ni.ldata)) return 3.0f;
        if (!contraction(l->type)) return 1.0f + 8.0f * th * tw / BYTES_PER_US;
        const unsigned heads = std::max(1u, l->params[NUM_HEAD]);
        const unsigned k = l->type == K_ATTENTION_LAYER ? l->params[NUM_HIDDEN] / heads : l->type == V_ATTENTION_LAYER ? plan->tr_seq_len : layer_contraction_k(l);
        return (float)tile_us(path_of(l, precision, plan->tr_seq_len), l, th, tw, k, 0, ni.ldata->slices);
    };
    float now = 0;
    unsigned idle = workers;
    auto start = [&](unsigned t) {
        started[t] = true;
        order.tile.push_back(t);
        order.at.push_back(now);
        running.push(Event(now + HAND_OVER_US + us(t), t));
    };
    for (unsigned t = 0; t < n; t++) if (need[t] == 0 && !skip[t]) ready.push(t);
    while (true) {
        for (; idle && !ready.empty(); idle--) { start(ready.front()); ready.pop(); }
        if (running.empty()) break;
        now = running.top().first;
        const unsigned t = running.top().second;
        running.pop();
        idle++;
        for (unsigned c : children[t])
            if (!skip[c] && left[c] != 0 && --left[c] == 0) ready.push(c);
    }
    for (float &a : order.at) a = now > 0 ? a / now : 0;
    order.us = now;
    order.runs = (unsigned)order.tile.size();
    for (unsigned t = 0; t < n; t++) if (!started[t] && !skip[t]) { order.tile.push_back(t); order.at.push_back(1.0f); }
    return order;
}

// Graphs of about the same length progress at the same share of their runs, so that each fills the gaps of the others to the end; the shorter
// a graph is, the nearer it comes to its own pace, because whoever waits for a small network should not wait for the large one
// beside it: a graph of r times the longest one's length is through after r (1 + 1.5 r) of the order, from r = 0.55 on after all of it.
// us until the shorter graph of two is complete / until both are, at the same share / each at its own pace / this:
//     CIFAR net + ResNet-50 x 32       1257 / 1417    109 / 1435    125 / 1434
//     CIFAR net + BERT 16 x 128        1211 / 1407     88 / 1410     92 / 1405
//     CIFAR net x 8 + ResNet-50 x 4     494 /  618    116 /  626    119 /  629
//     ResNet-50 + VGG-16 x 16          1342 / 1357    788 / 1419   1009 / 1398
//     BERT 1 x 37 + GPT-2 8 x 512      2528 / 2570   1182 / 2722   1502 / 2614
//     ResNet-50 x 16 + VGG-16 x 16     1762 / 1768   1472 / 1881   1762 / 1769
// Tiles whose lists cannot be satisfied come last.
std::vector<Claim> merge_claims(const std::vector<const ClaimOrder *> &graphs) {
    typedef std::pair<float, unsigned> Next;                   // when a graph's next tile is due; the graph
    std::priority_queue<Next, std::vector<Next>, std::greater<Next>> next;
    std::vector<size_t> place(graphs.size(), 0);
    std::vector<float> length;
    float longest = 0;
    size_t total = 0;
    for (const ClaimOrder *c : graphs) { longest = std::max(longest, c->us); total += c->tile.size(); }
    for (const ClaimOrder *c : graphs) length.push_back(longest > 0 ? std::min(longest, c->us * (1.0f + 1.5f * c->us / longest)) : 0.0f);
    auto push = [&](unsigned g) {
        const ClaimOrder &c = *graphs[g];
        if (place[g] < c.tile.size()) next.push(Next(place[g] < c.runs ? c.at[place[g]] * length[g] : 2 * longest + 1, g));
    };
    std::vector<Claim> order;
    order.reserve(total);
    for (unsigned g = 0; g < graphs.size(); g++) push(g);
    while (!next.empty()) {
        const unsigned g = next.top().second;
        next.pop();
        order.push_back(Claim{g, graphs[g]->tile[place[g]++]});
        push(g);
    }
    return order;
}

nasm_t *own_device_tiles(const nasm_t *nasm) {
    nasm_t *own = new nasm_t();
    own->dnn = nasm->dnn;
    own->batch_size = nasm->batch_size;
    own->tr_seq_len = nasm->tr_seq_len;
    own->num_ldata = nasm->num_ldata;
    own->num_ninst = nasm->num_ninst;
    own->ldata = nasm->ldata;
    own->ninst = nasm->ninst;
    for (nasm_ldata_t &ld : own->ldata) {
        ld.nasm = own;
        ld.out_mat_stride = (unsigned)round_up(ld.out_mat_stride, 4);
        ld.out_mat_mem_size = std::max(ld.out_mat_mem_size, (size_t)ld.out_mat_stride * ld.out_mat_dims[OUT_W] * sizeof(float));
    }
    for (ninst_t &ni : own->ninst) ni.ldata = own->ldata.data() + (ni.ldata - nasm->ldata.data());
    return own;
}

nasm_t *plan_device_tiles(const nasm_t *nasm, int precision, unsigned sms, bool served) {
    std::unique_ptr<nasm_t> plan(new nasm_t());
    plan->dnn = nasm->dnn;
    plan->batch_size = nasm->batch_size;
    plan->tr_seq_len = nasm->tr_seq_len;
    plan->num_ldata = nasm->num_ldata;
    plan->ldata = nasm->ldata;
    std::vector<Grid> grid(plan->num_ldata);
    unsigned total = 0;
    for (unsigned i = 0; i < plan->num_ldata; i++) {
        nasm_ldata_t &ld = plan->ldata[i];
        ld.nasm = plan.get();
        Grid &g = grid[i] = choose(nasm->ldata[i], nasm, precision, sms, served);
        const unsigned H = ld.out_mat_dims[OUT_H], W = ld.out_mat_dims[OUT_W];
        if (H == 0 || W == 0 || W % g.seg != 0) return nullptr;
        g.start = total;
        ld.ninst_tile_dims[OUT_H] = g.th;
        ld.ninst_tile_dims[OUT_W] = g.tw;
        ld.out_mat_stride = (unsigned)round_up(H, 4);
        ld.out_mat_mem_size = (size_t)ld.out_mat_stride * W * sizeof(float);
        ld.ninst_start = total;
        ld.slices = g.ks;
        ld.num_ninst = g.nh * (W / g.seg) * g.per_seg * g.ks;
        total += ld.num_ninst;
    }
    plan->num_ninst = total;
    plan->ninst.resize(total);
    for (unsigned i = 0; i < plan->num_ldata; i++) {
        nasm_ldata_t &ld = plan->ldata[i];
        const aspen_layer_t *l = ld.layer;
        const unsigned *p = l->params;
        const Grid &g = grid[i];
        const unsigned H = ld.out_mat_dims[OUT_H], seq = plan->tr_seq_len;
        const unsigned i0 = ld.parent_ldata_idx_arr[PARENT_0], i1 = ld.parent_ldata_idx_arr[PARENT_1];
        for (unsigned t = 0; t < ld.num_ninst; t++) {
            ninst_t &ni = plan->ninst[g.start + t];
            const unsigned cell = t / g.ks, ch = cell % g.nh, cw = cell / g.nh, seg = cw / g.per_seg, in_seg = (cw % g.per_seg) * g.tw;
            const unsigned h0 = ch * g.th, h1 = std::min(H, h0 + g.th), w0 = seg * g.seg + in_seg, w1 = seg * g.seg + std::min(g.seg, in_seg + g.tw);
            ni.ldata = &ld;
            ni.ninst_idx = g.start + t;
            ni.out_mat_pos[OUT_H] = h0; ni.out_mat_pos[OUT_W] = w0;
            ni.tile_dims[OUT_H] = h1 - h0; ni.tile_dims[OUT_W] = w1 - w0;
            // the tiles of parent layer `par` that overlap rows [r0, r1) x columns [c0, c1)
            auto reads = [&](unsigned par, unsigned r0, unsigned r1, unsigned c0, unsigned c1) {
                const Grid &q = grid[par];
                const nasm_ldata_t &pl = plan->ldata[par];
                r1 = std::min(r1, pl.out_mat_dims[OUT_H]); c1 = std::min(c1, pl.out_mat_dims[OUT_W]);
                for (unsigned c = c0; c < c1;) {
                    const unsigned s = c / q.seg, k = (c % q.seg) / q.tw, col = s * q.per_seg + k;
                    for (unsigned r = r0 / q.th; r * q.th < r1; r++)
                        for (unsigned s = 0; s < q.ks; s++) ni.parent_ninst_idx.push_back(q.start + (col * q.nh + r) * q.ks + s);
                    c = s * q.seg + std::min(q.seg, (k + 1) * q.tw);
                }
            };
            const unsigned all = 0xffffffffu;
            if (l->type == INPUT_LAYER || i0 == (unsigned)-1) continue;
            const bool like0 = plan->ldata[i0].out_mat_dims[OUT_W] == ld.out_mat_dims[OUT_W];
            switch (l->type) {
                case CONV_LAYER: case MAXPOOL_LAYER: case AVGPOOL_LAYER: {
                    const unsigned OW = p[OUT_W], hw = p[OUT_H] * OW, IW = p[IN_W], IH = p[IN_H], s = p[STRIDE] ? p[STRIDE] : 1;
                    const unsigned r0 = l->type == CONV_LAYER ? 0 : h0, r1 = l->type == CONV_LAYER ? all : h1;
                    if (p[WEIGHT_H] == 1 && p[WEIGHT_W] == 1 && s == 1 && p[PADDING] == 0 && like0) { reads(i0, r0, r1, w0, w1); break; }
                    // whole input rows; a tile that spans samples reads every row in between
                    const unsigned b0 = w0 / hw, b1 = (w1 - 1) / hw, y0 = (w0 % hw) / OW * s, y1 = ((w1 - 1) % hw) / OW * s + p[WEIGHT_H] - 1;
                    const unsigned first = y0 > p[PADDING] ? y0 - p[PADDING] : 0, last = std::min(IH - 1, y1 > p[PADDING] ? y1 - p[PADDING] : 0);
                    reads(i0, r0, r1, (b0 * IH + std::min(first, IH - 1)) * IW, (b1 * IH + last + 1) * IW);
                    break;
                }
                case FC_LAYER: { const unsigned px = p[IN_H] * p[IN_W]; reads(i0, 0, all, w0 * px, w1 * px); break; }
                case MATMUL_LAYER: case LAYERNORM_LAYER: reads(i0, 0, all, w0, w1); break;
                case RESIDUAL_LAYER:
                    reads(i0, h0, h1, w0, w1);
                    if (i1 != (unsigned)-1) reads(i1, h0, h1, w0, w1);
                    break;
                case K_ATTENTION_LAYER: {
                    const unsigned heads = p[NUM_HEAD], hd = p[NUM_HIDDEN] / heads, b = w0 / (seq * heads), head = w0 / seq % heads, q0 = w0 % seq;
                    reads(i0, head * hd, (head + 1) * hd, b * seq + q0, b * seq + q0 + (w1 - w0));
                    if (i1 != (unsigned)-1) reads(i1, head * hd, (head + 1) * hd, b * seq + h0, b * seq + h1);
                    break;
                }
                case V_ATTENTION_LAYER: {
                    const unsigned heads = p[NUM_HEAD], hd = p[NUM_HIDDEN] / heads, b = w0 / seq, head = h0 / hd, c = (b * heads + head) * seq + w0 % seq;
                    reads(i0, 0, all, c, c + (w1 - w0));
                    if (i1 != (unsigned)-1) reads(i1, h0, h1, b * seq, (b + 1) * seq);
                    break;
                }
                default:
                    reads(i0, 0, all, 0, all);
                    if (i1 != (unsigned)-1) reads(i1, 0, all, 0, all);
                    break;
            }
            if (ni.parent_ninst_idx.empty()) return nullptr;
        }
    }
    graph_set_children(plan.get());
    return plan.release();
}
