/* launch_unit.cpp — the host-side choices of b2g_launch.h, without a GPU. */
#include <cstdio>
#include <thread>
#include <vector>

#include "b2g_launch.h"

using namespace b2g;

static int failures = 0;
static void check(bool ok, const char* what) {
    if (!ok) {
        std::printf("wrong: %s\n", what);
        ++failures;
    }
}

int main() {
    /* found once for each device, not once for the process, from any thread */
    PerDevice<int> value;
    int found[4] = {0, 0, 0, 0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 16; ++t)
        threads.emplace_back([&, t] {
            for (int k = 0; k < 100; ++k) {
                const int dev = (t + k) % 4;
                const int got = value.at(dev, [&] {
                    ++found[dev];
                    return 100 + dev;
                });
                if (got != 100 + dev) ++found[dev];
            }
        });
    for (auto& t : threads) t.join();
    for (int dev = 0; dev < 4; ++dev) check(found[dev] == 1, "a value is found once for each device");

    for (int limit : {0, 1, 2, 3, 4, 8, 15, 16, 64}) {
        int asked = 0;
        const int c = largest_cluster([&](int blocks) {
            ++asked;
            return blocks <= limit;
        });
        int best = 0;
        for (int q = 1; q <= kClusterMaxBlocks; q <<= 1) best = q <= limit ? q : best;
        check(c == best && asked <= 5, "the largest cluster that fits");
    }
    std::printf("%d wrong\n", failures);
    return failures != 0;
}
