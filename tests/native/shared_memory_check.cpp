// Host-side check of SharedMemoryOptIn (csrc/shared_memory.hpp) against a fake runtime of three devices:
// every kernel gets its attribute on every device it is used on, once, also from several host threads
// and after a call that failed.  Prints "ok" or the first mismatch.
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "../../replica_exchange_wang_landau_b200/csrc/shared_memory.hpp"

namespace {
thread_local int current = 0;
std::mutex mu;
int calls[64] = {};
bool refuse = false;
}  // namespace

extern "C" cudaError_t cudaGetDevice(int* device) {
    *device = current;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int) {
    std::lock_guard<std::mutex> lock(mu);
    if (refuse) return cudaErrorInvalidValue;
    ++calls[current];
    return cudaSuccess;
}

int main() {
    int kernel = 0;
    {
        wlg::SharedMemoryOptIn opt_in;
        refuse = true;
        if (opt_in(&kernel) != cudaErrorInvalidValue) return std::printf("a refusal was not reported\n"), 1;
        refuse = false;
        for (int round = 0; round < 2; ++round)
            for (current = 0; current < 3; ++current)
                if (opt_in(&kernel) != cudaSuccess || calls[current] != 1)
                    return std::printf("device %d: %d calls\n", current, calls[current]), 1;
    }
    wlg::SharedMemoryOptIn opt_in;
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            current = 3 + t % 4;
            for (int k = 0; k < 1000; ++k) {
                opt_in(&kernel);
                std::lock_guard<std::mutex> lock(mu);
                if (calls[current] == 0) std::printf("device %d used without its attribute\n", current);
            }
        });
    for (auto& t : threads) t.join();
    for (int d = 3; d < 7; ++d)
        if (calls[d] < 1 || calls[d] > 2) return std::printf("device %d: %d calls\n", d, calls[d]), 1;
    std::printf("ok\n");
    return 0;
}
