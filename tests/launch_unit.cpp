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

    /* the backward pass: never a cluster larger than fits, and as before where it does */
    for (int largest : {0, 1, 2, 4, 8, 16})
        for (int parts : {0, 1, 2, 5, 8, 9, 16, 17, 152})
            for (int slots : {0, 1, 512, 513, 1000, 4096, 4097, 8192, 8193, 200000}) {
                const AdjointBlocks on = adjoint_blocks(slots, parts, 152, largest);
                const bool small = slots <= 8192 && parts <= 16;
                if (on.cluster) {
                    check(on.blocks <= largest && small, "a cluster that fits");
                    check(on.blocks >= parts && 512 * on.blocks >= slots, "a block for each part and 512 slots");
                } else {
                    check(on.blocks >= 1 && on.blocks <= 152, "a grid of at most one block for each SM");
                    check(!small || largest < 16, "a cluster wherever the largest fits");
                }
            }
    check(adjoint_blocks(5000, 1, 152, 16).cluster && adjoint_blocks(5000, 1, 152, 16).blocks == 16, "5000 slots on 16 blocks");
    check(!adjoint_blocks(5000, 1, 152, 8).cluster && adjoint_blocks(5000, 1, 152, 8).blocks == 20, "5000 slots where 16 do not fit");
    check(adjoint_blocks(4000, 1, 152, 8).cluster && adjoint_blocks(4000, 1, 152, 8).blocks == 8, "4000 slots on 8 blocks");
    std::printf("%d wrong\n", failures);
    return failures != 0;
}
