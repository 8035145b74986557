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
    /* replay buffers: what is wanted where there is room, never past the limits, one at the least */
    const size_t mb = (size_t)1 << 20, gb = (size_t)1 << 30;
    check(replay_groups(15, 136 * mb, 200 * gb) == 15, "all segments of 512 worlds over 240 steps");
    check(replay_groups(15, 136 * mb, 0) == 1 && replay_groups(1, 100 * gb, 0) == 1, "one segment whatever is free");
    check(replay_groups(15, 136 * mb, 4 * gb) == 1 + 1024 / 136, "a quarter of the free memory");
    check(replay_groups(1 << 20, 1 * gb, 280 * gb) == 1 + 8, "8 GiB");
    check(replay_groups(1 << 20, 0, 280 * gb) == 1 << 20 && replay_groups(0, mb, gb) == 1, "sizes of nothing");
    /* an allocator with a small limit: halved until it fits, not even one, and what was wanted is not asked again */
    for (int limit : {0, 1, 2, 3, 7, 15, 100}) {
        int calls = 0, last = 0;
        const int got = allocate_groups(15, [&](int n) {
            ++calls;
            last = n;
            return n <= limit;
        });
        check(got <= limit && got == (limit >= 15 ? 15 : limit >= 8 ? 8 : limit >= 4 ? 4 : limit >= 2 ? 2 : limit), "groups that fit");
        check(got == 0 ? last == 1 && calls == 5 : last == got, "the last attempt is the one kept");
    }
    WorkSizes held;
    check(!held.serve(1, 1, 1, 1), "nothing held serves nothing");
    held.slots = 100, held.vi = 8, held.pi = 3, held.wanted = 15;
    check(held.serve(100, 8, 3, 15) && held.serve(1, 1, 1, 1), "buffers of fewer groups than wanted serve the same call");
    check(!held.serve(101, 8, 3, 15) && !held.serve(100, 9, 3, 15) && !held.serve(100, 8, 4, 15) && !held.serve(100, 8, 3, 16), "larger calls");
    std::printf("%d wrong\n", failures);
    return failures != 0;
}
