// Host-side check of the two routines that stand in for a division on the device (csrc/common.cuh):
//  * quotient_rn(a, b, y) must equal a / b rounded to nearest, whatever approximation y of 1 / b with
//    a relative error below 2^-18 it starts from;
//  * floor_near_integer(d, w, rint(q)) must equal floor(d / w) wherever q = d * (1 / w) lies within the
//    margin of an integer in which the attempt loop asks for it, and outside the margin floor(q) must
//    be floor(d / w) already (the loop's own test, restated here).
// Prints "ok <cases>" or the first mismatch.
#include <cinttypes>
#include <cmath>
#include <cstdio>

#include "../../replica_exchange_wang_landau_b200/csrc/common.cuh"

int main() {
    wlg::Rng rng;
    rng.seed(77, 3);
    uint64_t cases = 0;
    auto unit = [&] { return static_cast<double>(rng.next() >> 11) * 0x1.0p-53; };
    // counts over counts, as the 1/t factor divides them; small numbers, neighbours of powers of two,
    // quotients next to a rounding boundary
    for (int k = 0; k < 4000000; ++k) {
        uint64_t ai = 1 + rng.next() % (k % 4 == 0 ? 64 : (k % 4 == 1 ? 100000 : 0x7fffffffULL));
        uint64_t bi = 1 + (rng.next() >> (1 + rng.next() % 63));
        if (k % 7 == 0) bi = (uint64_t{1} << (rng.next() % 63)) + rng.next() % 5;
        if (k % 11 == 0) ai = bi % 1000 + 1;
        if (k % 13 == 0) bi = ai + rng.next() % 3;
        if (bi == 0) bi = 1;
        const double a = static_cast<double>(ai), b = static_cast<double>(bi);
        const double y = static_cast<double>(static_cast<float>(1.0 / b)) * (1.0 + (unit() - 0.5) * 0x1.0p-18);
        const double got = wlg::quotient_rn(a, b, y), want = a / b;
        if (got != want) {
            std::printf("quotient_rn(%.17g, %.17g) = %.17g, not %.17g\n", a, b, got, want);
            return 1;
        }
        ++cases;
    }
    uint64_t asked = 0;
    for (int k = 0; k < 6000000; ++k) {
        const double w = k % 3 == 0 ? 0.001 * static_cast<double>(1 + rng.next() % 5000)
                                    : (k % 3 == 1 ? unit() * 3.0 + 1e-3 : 1.0 / (1.0 + static_cast<double>(rng.next() % 999)));
        const double count = static_cast<double>(2 + rng.next() % (k % 2 ? 3000 : 2000000000));
        const double n = std::floor(unit() * (count + 3.0)) - 1.0;
        double d = n * w;  // next to a bin's edge: the nearest doubles on both sides of it
        const int steps = static_cast<int>(rng.next() % 9) - 4;
        for (int s = 0; s < std::abs(steps); ++s) d = std::nextafter(d, steps < 0 ? -HUGE_VAL : HUGE_VAL);
        if (k % 5 == 0) d = (n + unit()) * w;
        // EnergyGrid::index rejects an energy below the grid before it divides (src/wang_landau.cpp:27-38)
        const double want = d < 0.0 ? -1.0 : std::floor(d / w);
        const double q = d * (1.0 / w), fl = std::floor(q);
        const double half_clear = 0.5 - (count + 2.0) * 0x1p-49;
        const bool ask = !(std::fabs(q - fl - 0.5) < half_clear);
        const double got = ask ? wlg::floor_near_integer(d, w, std::rint(q)) : fl;
        asked += ask ? 1 : 0;
        if (got != want && !(got < 0.0 && want < 0.0)) {
            std::printf("floor(%.17g / %.17g) = %.17g, not %.17g (asked %d)\n", d, w, got, want, ask ? 1 : 0);
            return 1;
        }
        ++cases;
    }
    if (asked < 1000000) {
        std::printf("the exact floor was asked for only %" PRIu64 " times\n", asked);
        return 1;
    }
    std::printf("ok %" PRIu64 "\n", cases);
    return 0;
}
