/*
 * b2g_launch.h — host-side choices about launches that need no CUDA call, so that they can be tested without a
 * GPU: values found once for each device, the largest cluster that fits, the backward pass's blocks and buffers.
 */
#ifndef B2G_LAUNCH_H
#define B2G_LAUNCH_H

#include <algorithm>
#include <cstddef>
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

/* Segments of a backward pass whose replays get buffers side by side, `each` bytes a segment: as many as are
 * wanted, but beyond the one it cannot do without no more than kReplayBytes and a quarter of the free memory
 * take. 512 worlds over 240 steps hold 15 segments in 1.9 GB more than one segment's. */
constexpr size_t kReplayBytes = (size_t)8 << 30;
inline int replay_groups(int wanted, size_t each, size_t free_bytes) {
    const size_t room = std::min(kReplayBytes, free_bytes / 4) / std::max<size_t>(each, 1);
    return 1 + (int)std::min<size_t>((size_t)std::max(wanted - 1, 0), room);
}

/* fewer, down to one, while allocate(groups) fails; 0: not even one */
template <class Allocate>
int allocate_groups(int groups, Allocate&& allocate) {
    for (;; groups = (groups + 1) / 2) {
        if (allocate(groups)) return groups;
        if (groups <= 1) return 0;
    }
}

/* What a backward pass's buffers were allocated for. They serve every call that asks for no more, also where
 * they hold fewer groups than were wanted: the memory was not there, and asking for it again on every call
 * would free and allocate all of them on every call. */
struct WorkSizes {
    int slots = 0, vi = 0, pi = 0, wanted = 0;
    bool serve(int s, int v, int p, int w) const { return wanted > 0 && s <= slots && v <= vi && p <= pi && w <= wanted; }
};

}  // namespace b2g

#endif
