// Host-side check of most_shared_epochs (csrc/engine.hpp): a launch makes at least one epoch and at most 2^32 - 1
// attempts of a walker, all of which may visit one bin.  Prints "ok" or the first mismatch.
#include <cstdio>

#include "../../replica_exchange_wang_landau_b200/csrc/engine.hpp"

int main() {
    for (uint64_t interval = 1; interval <= (uint64_t{1} << 17); ++interval) {
        const uint64_t epochs = wlg::most_shared_epochs(interval);
        if (epochs < 1 || epochs * interval > 0xffffffffULL || (epochs + 1) * interval <= 0xffffffffULL) {
            std::printf("%llu attempts: %llu epochs\n", static_cast<unsigned long long>(interval),
                        static_cast<unsigned long long>(epochs));
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
