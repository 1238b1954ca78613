// Eight threads walk worker_loop over random tiles as the worker warps do; from some moment on each of their bounded waits may give up
// or be met, for every warp by chance.  All of them have to leave, and a tile with barriers is walked by all or by none.
//   worker_loop SEED
#include "../../aspen_b200/csrc/worker_loop.h"

#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

constexpr unsigned WARPS = 8, TILES = 40;

struct Barrier {      // of all warps, with a vote
    std::mutex m;
    std::condition_variable cv;
    unsigned here = 0, round = 0;
    bool yes = true, result = true;
    bool meet(bool vote) {
        std::unique_lock<std::mutex> l(m);
        yes = yes && vote;
        const unsigned mine = round;
        if (++here == WARPS) { result = yes; yes = true; here = 0; round++; cv.notify_all(); }
        else cv.wait(l, [&] { return round != mine; });
        return result;
    }
};

struct Run {
    Barrier barrier;
    std::vector<unsigned> barriers;             // of each tile; 0: none
    std::vector<unsigned> fails_from;           // waits of a warp may give up from this tile on
    std::atomic<unsigned> walked[TILES];
};

struct Warp {
    Run &r;
    unsigned id;
    std::mt19937 rng;
    bool wait(unsigned seq) { return seq < r.fails_from[id] || rng() % 3 != 0; }
    bool posted(unsigned seq) { return wait(seq); }
    bool live(unsigned seq) { return seq < TILES; }
    bool meets(unsigned seq) { return r.barriers[seq] != 0; }
    bool agree(bool yes) { return r.barrier.meet(yes); }
    bool run(unsigned seq) {
        bool ok = true;
        for (unsigned b = 0; b < r.barriers[seq]; b++) { ok = ok && wait(seq); r.barrier.meet(true); }
        if (r.barriers[seq]) r.walked[seq]++;
        else ok = wait(seq);
        return ok;
    }
    void finished(unsigned) {}
};

int main(int, char **argv) {
    std::mt19937 rng((unsigned)atoi(argv[1]));
    for (unsigned trial = 0; trial < 300; trial++) {
        Run r;
        for (unsigned i = 0; i < TILES; i++) { r.barriers.push_back(rng() % 3 ? 0 : 1 + rng() % 3); r.walked[i] = 0; }
        for (unsigned i = 0; i < WARPS; i++) r.fails_from.push_back(trial % 4 ? rng() % (2 * TILES) : 2 * TILES);
        std::vector<std::thread> team;
        for (unsigned i = 0; i < WARPS; i++) team.emplace_back([&r, i, seed = rng()] { Warp w{r, i, std::mt19937(seed)}; worker_loop(w); });
        for (std::thread &t : team) t.join();
        for (unsigned i = 0; i < TILES; i++)
            if (r.walked[i] != 0 && r.walked[i] != WARPS) { printf("tile %u was walked by %u warps\n", i, r.walked[i].load()); return 1; }
        if (trial % 4 == 0 && r.barriers[TILES - 1] && r.walked[TILES - 1] != WARPS) { printf("the last tile was not reached\n"); return 1; }
    }
    return 0;
}
