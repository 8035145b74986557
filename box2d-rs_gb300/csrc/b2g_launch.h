/*
 * b2g_launch.h — host-side choices about launches that need no CUDA call, so that they can be tested without a
 * GPU: values found once for each device, the largest cluster that fits.
 */
#ifndef B2G_LAUNCH_H
#define B2G_LAUNCH_H

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

}  // namespace b2g

#endif
