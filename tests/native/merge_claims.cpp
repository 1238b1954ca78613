// Launches of several graphs: every tile once, each graph's in its own order, a short graph complete long before a long one, graphs of about the
// same length together, tiles that never run behind all others.
#include "../../aspen_b200/csrc/internal.h"

static ClaimOrder graph(unsigned tiles, float us, unsigned stuck = 0) {
    ClaimOrder c;
    for (unsigned i = 0; i < tiles; i++) {
        c.tile.push_back((i * 7u) % tiles);                                     // tiles: no multiple of 7
        c.at.push_back(i < tiles - stuck ? (float)i / (tiles - stuck) : 1.0f);
    }
    c.us = us;
    c.runs = tiles - stuck;
    return c;
}
struct Seen { std::vector<size_t> first, last; };
static int check(const std::vector<const ClaimOrder *> &graphs, Seen &seen) {
    const std::vector<Claim> order = merge_claims(graphs);
    std::vector<size_t> place(graphs.size(), 0);
    seen.first.assign(graphs.size(), 0);
    seen.last.assign(graphs.size(), 0);
    for (size_t i = 0; i < order.size(); i++) {
        const Claim c = order[i];
        if (c.graph >= graphs.size() || place[c.graph] >= graphs[c.graph]->tile.size() || graphs[c.graph]->tile[place[c.graph]] != c.tile) return 1;
        if (place[c.graph]++ == 0) seen.first[c.graph] = i;
        if (place[c.graph] == graphs[c.graph]->runs) seen.last[c.graph] = i;
    }
    for (size_t g = 0; g < graphs.size(); g++) if (place[g] != graphs[g]->tile.size()) return 2;
    return 0;
}

int main() {
    Seen s;
    const ClaimOrder small = graph(100, 50), large = graph(5000, 1400), other = graph(4000, 1100), stuck = graph(100, 50, 90);
    int rc = check({&small, &large}, s);
    if (rc) return rc;
    if (s.first[0] > 10 || s.last[0] > 350 || s.last[1] != 5099) return 10;     // 1.05 x 50 / 1400 of 5000 tiles, and its own 100
    rc = check({&other, &large, &small}, s);
    if (rc) return rc;
    if (s.last[0] < 9000 || s.last[1] < 9000 || s.last[2] > 850) return 11;
    rc = check({&stuck, &large}, s);
    if (rc) return rc;
    if (s.last[0] > 450 || s.last[1] != 5009) return 12;                        // ten tiles run, the other 90 lie behind all of the large graph
    return check({}, s) || check({&small}, s) ? 13 : 0;
}
