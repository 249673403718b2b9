// When a repeated piece of device work is issued and when it is replayed from a captured
// graph.  Host code without CUDA types.
#pragma once

#include <cstdint>

namespace nkr {

// The first call issues its launches, the second captures them and replays from then on, so
// a program that calls once does not pay for a capture.  A capture and its graph take memory
// that issuing does not: where either fails, this call and all later ones issue.
struct ReplayPolicy {
    uint64_t calls = 0;   // completed
    bool refused = false; // a capture or a launch failed

    // captured(): is there a graph; capture(), launch() and issue() return a status, 0 for
    // success
    template <class Captured, class Capture, class Launch, class Issue>
    int run(Captured &&captured, Capture &&capture, Launch &&launch, Issue &&issue)
    {
        if (calls > 0 && !refused) {
            if ((captured() || capture() == 0) && launch() == 0) {
                ++calls;
                return 0;
            }
            refused = true;
        }
        const int s = issue();
        if (s == 0) ++calls;
        return s;
    }
};

} // namespace nkr
