// Host-side check of opened_by_staying (csrc/common.cuh): every outcome of the first attempt of an epoch
// that starts in a bin not visited before, counted as the attempt loop counts it, against the number of
// visited bins itself.  Prints "ok <cases>" or the first mismatch.
#include <cstdio>
#include <vector>

#include "../../replica_exchange_wang_landau_b200/csrc/common.cuh"

int main() {
    const int bins = 5;
    int cases = 0;
    for (int mask = 0; mask < (1 << bins); ++mask)
        for (int from = 0; from < bins; ++from) {
            if ((mask >> from) & 1) continue;  // visited already
            for (int to = 0; to < bins; ++to)
                for (int accepted = 0; accepted < 2; ++accepted) {
                    const uint32_t before = static_cast<uint32_t>(__builtin_popcount(static_cast<unsigned>(mask)));
                    const int cur = accepted ? to : from;
                    const int after = mask | (1 << cur);
                    uint32_t active = before + (accepted && !((mask >> to) & 1) ? 1u : 0u);
                    if (wlg::opened_by_staying(cur, from, active, before)) ++active;
                    if (active != static_cast<uint32_t>(__builtin_popcount(static_cast<unsigned>(after)))) {
                        std::printf("mask %d from %d to %d accepted %d: %u\n", mask, from, to, accepted, active);
                        return 1;
                    }
                    ++cases;
                }
        }
    std::printf("ok %d\n", cases);
    return 0;
}
