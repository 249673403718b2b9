// The choice of the MSM window autotuner among its measured widths.  Host code without CUDA
// types.
#pragma once

#include <utility>
#include <vector>

namespace nkr {

// Of the widths within 3% of the fastest the one of the least work, and its own time: they
// differ in the work that they leave for others (a batch of 8 proofs of 2^15 constraints took
// 7.0 to 7.7 ms with whichever happened to be the fastest).
template <class Work>
std::pair<int, float> choose_width(const std::vector<std::pair<int, float>> &times, Work &&work)
{
    float best = 1e30f;
    for (const auto &t : times) best = t.second < best ? t.second : best;
    std::pair<int, float> choice{0, 0.f};
    double least = 1e300;
    for (const auto &t : times) {
        const double w = work(t.first);
        if (t.second <= 1.03f * best && w < least) {
            least = w;
            choice = t;
        }
    }
    return choice;
}

} // namespace nkr
