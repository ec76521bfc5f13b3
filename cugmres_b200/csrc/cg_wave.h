// Runs the buckets of a wave to their ends from one host thread (cg_batch.cu).
#pragma once

#include <stddef.h>

#include <thread>

namespace cg {

// Until every bucket is done: for each that is ready, its next step and, after the
// last, its results.  ready(b, last, &go) says whether b can go on (it may wait for
// `last`, the only one left), step(b) sets b.done at its end, finish(b) delivers; all
// return 0 or a status.  A bucket that fails is done without results; the others
// run on and deliver theirs.  Returns the first failure's status.
template <typename Wave, typename Ready, typename Step, typename Finish>
int run_side_by_side(Wave &wave, Ready ready, Step step, Finish finish) {
    int first = 0;
    size_t left = wave.size();
    while (left > 0) {
        for (auto &b : wave) {
            if (b->done) continue;
            bool go = true;
            int st = ready(*b, left == 1, &go);
            if (st == 0 && !go) continue;
            if (st == 0) st = step(*b);
            if (st == 0 && b->done) st = finish(*b);
            if (st != 0) {
                if (first == 0) first = st;
                b->done = true;
            }
            if (b->done) left--;
        }
        if (left > 1) std::this_thread::yield();
    }
    return first;
}

}  // namespace cg
