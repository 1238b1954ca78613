// Order in which a launch hands out the tiles of a cfg's device plan: every tile once, parents before children, and tiles whose lists
// cannot be satisfied last.  claim_order cfg batch seq workers precision; prints how many layers share their k among tiles
#include "../../aspen_b200/csrc/internal.h"

static int check(const nasm_t *plan, int precision, unsigned workers, const std::vector<std::vector<unsigned>> &children, const std::vector<unsigned> &need, unsigned stuck) {
    const unsigned n = plan->num_ninst;
    std::vector<bool> skip(n, false);
    const unsigned left_out = plan->ldata.back().ninst_start;        // as if another layer's tiles wrote this one's values
    skip[left_out] = true;
    const ClaimOrder o = claim_order(plan, precision, workers, children, need, skip);
    std::vector<unsigned> place(n, n);
    if (o.tile.size() != n - 1 || o.at.size() != n - 1) return 1;
    for (unsigned i = 0; i < n - 1; i++) {
        if (o.tile[i] >= n || o.tile[i] == left_out || place[o.tile[i]] != n) return 2;
        place[o.tile[i]] = i;
        if (o.at[i] < 0 || o.at[i] > 1 || (i && o.at[i] < o.at[i - 1])) return 3;
    }
    for (unsigned t = 0; t < n; t++)
        for (unsigned c : children[t])
            if (t != left_out && c != left_out && place[c] < place[t]) return 4;
    if (stuck < n)
        for (unsigned t = 0; t < stuck; t++) if (t != left_out && place[t] > place[stuck]) return 5;
    return 0;
}

int main(int, char **argv) {
    aspen_dnn_t *dnn = apu_create_dnn(argv[1], nullptr);
    nasm_t *nasm = dnn ? apu_create_transformer_nasm(dnn, 100, (unsigned)atoi(argv[2]), (unsigned)atoi(argv[3])) : nullptr;
    nasm_t *plan = nasm ? plan_device_tiles(nasm, atoi(argv[5]), 148, false) : nullptr;
    if (!plan) return 9;
    std::vector<std::vector<unsigned>> children;
    std::vector<unsigned> need;
    for (const ninst_t &ni : plan->ninst) {
        children.push_back(ni.child_ninst_idx);
        need.push_back((unsigned)ni.parent_ninst_idx.size());
    }
    int rc = check(plan, atoi(argv[5]), (unsigned)atoi(argv[4]), children, need, plan->num_ninst);
    const unsigned stuck = plan->ldata[plan->num_ldata / 2].ninst_start;
    need[stuck]++;
    if (rc == 0) rc = check(plan, atoi(argv[5]), (unsigned)atoi(argv[4]), children, need, stuck);
    // a tile that reads an output whose k is shared waits for each of the tiles that share it
    unsigned shared = 0;
    for (const nasm_ldata_t &ld : plan->ldata) {
        shared += ld.slices > 1;
        for (unsigned t = 0; t < ld.num_ninst && rc == 0; t++)
            if (children[ld.ninst_start + t] != children[ld.ninst_start + t / ld.slices * ld.slices]) rc = 6;
    }
    printf("%u", shared);
    delete plan;
    apu_destroy_nasm(nasm);
    apu_destroy_dnn(dnn);
    return rc;
}
