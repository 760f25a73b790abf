// check_smem_limit.cpp — physecs_gb300/csrc/smem_limit.cuh with threads that ask for different
// sizes at once (test infrastructure).  The attribute is a variable whose setter takes its
// time, so that a thread that looks and sets in two steps would lower it again.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.cuh"

int main() {
    for (int round = 0; round < 40; ++round) {
        psx::SmemLimit limit;
        std::atomic<int> attribute{0}, waiting{0}, low{0}, sets{0};
        std::vector<std::thread> threads;
        for (int i = 0; i < 8; ++i)
            threads.emplace_back([&, i] {
                const int bytes = 1024 * (1 + (i * 5 + round) % 8);
                ++waiting;
                while (waiting < 8) {}
                limit.raise(round % 2 ? 0 : 70, bytes, [&](int b) {
                    std::this_thread::sleep_for(std::chrono::microseconds(50 * ((b / 1024 * 3) % 7)));
                    attribute = b;
                    ++sets;
                });
                if (round % 2 && attribute < bytes) ++low;   // the launch that follows would be refused
            });
        for (auto& t : threads) t.join();
        if (low) { std::printf("round %d: %d threads found the limit below their size\n", round, low.load()); return 1; }
        if (round % 2 && attribute != 8 * 1024) { std::printf("round %d: the limit ends at %d\n", round, attribute.load()); return 1; }
        if (!(round % 2) && sets != 8) { std::printf("round %d: a device past the table was not set\n", round); return 1; }
    }
    return 0;
}
