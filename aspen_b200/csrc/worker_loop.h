// How a worker warp walks over the posted tiles.
//
// Some tiles make the worker warps meet at barriers, and a barrier waits without a bound: it must never happen that a warp has
// given up a (bounded) wait and left while another, whose wait was met at that very moment, goes on to a barrier.  So the
// warps agree before every tile that has barriers, a warp leaves only through such an agreement, and a tile with barriers is
// walked to its end by all of them or by none.  An agreement completes when all warps are there: each is, after a
// bounded time, since between two agreements there are only bounded waits.
#pragma once

#ifdef __CUDACC__
#define WORKER_LOOP_FN __device__ __forceinline__
#else
#define WORKER_LOOP_FN inline
#endif

// Warp:  bool posted(seq): the seq-th tile is there (false: gave up waiting);  bool live(seq): it is a tile, not the end;
//        bool meets(seq): the tile has barriers;  bool run(seq): false: gave up a wait (a tile with barriers has gone through them all);
//        void finished(seq);  bool agree(bool): barrier of all worker warps, true if all of them say so.
template <typename Warp>
WORKER_LOOP_FN void worker_loop(Warp &w) {
    for (unsigned seq = 0;; seq++) {
        if (!w.posted(seq) || !w.live(seq)) break;
        if (w.meets(seq) && !w.agree(true)) return;      // another warp is leaving
        const bool ok = w.run(seq);
        w.finished(seq);
        if (!ok) break;
    }
    w.agree(false);
}
