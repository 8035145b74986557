/*
 * b2g_launch.h — host-side choices about launches that need no CUDA call, so that they can be tested without a
 * GPU: values found once for each device, the largest cluster that fits, the backward pass's blocks.
 */
#ifndef B2G_LAUNCH_H
#define B2G_LAUNCH_H

#include <algorithm>
#include <map>
#include <mutex>

namespace b2g {

constexpr int kClusterMaxBlocks = 16; /* above 8 a kernel has to allow it, and the device to have room for it */

/* A value found once for each device. A function's attributes and what fits a device belong to the device that
 * is current when they are set or asked for, and worlds of one process may live on several. */
template <class T>
class PerDevice {
  public:
    template <class Find>
    T at(int device, Find&& find) {
        std::lock_guard<std::mutex> lock(mutex_);
        auto it = found_.find(device);
        if (it == found_.end()) it = found_.emplace(device, find()).first;
        return it->second;
    }

  private:
    std::mutex mutex_;
    std::map<int, T> found_;
};

/* the largest power of two up to kClusterMaxBlocks for which fits(blocks) holds, 0 if none */
template <class Fits>
int largest_cluster(Fits&& fits) {
    for (int c = kClusterMaxBlocks; c >= 1; c >>= 1)
        if (fits(c)) return c;
    return 0;
}

/* How a backward pass is launched, from the slots of its largest step, the parts of its solves and the largest
 * cluster its kernels fit: on clusters of up to 16 blocks (one block for a small world) where a step fits 512
 * slots a block, else on a cooperative grid of a block for each part or 256 slots. (One block for up to 4096
 * slots took 110 ms for 128 steps of 10 throw-and-stack worlds, whose 1000 slots in two parts it swept one
 * after the other; the cluster of two takes 31. 128 steps of one world: 34.7 -> 18.5 ms, 64 steps of 512
 * worlds: 42.7 -> 28 ms, replays side by side and local memory gone.) */
struct AdjointBlocks {
    int blocks;
    bool cluster;
};
inline AdjointBlocks adjoint_blocks(int max_slots, int parts, int num_sms, int largest) {
    if (max_slots <= 512 * kClusterMaxBlocks && parts <= kClusterMaxBlocks) {
        int c = 1;
        while (c < kClusterMaxBlocks && (c < parts || 512 * c < max_slots)) c <<= 1;
        if (c <= largest) return {c, true};
    }
    return {std::max(1, std::min(num_sms, std::max(parts, (max_slots + 255) / 256))), false};
}

}  // namespace b2g

#endif
