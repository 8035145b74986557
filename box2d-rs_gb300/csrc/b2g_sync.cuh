/*
 * b2g_sync.cuh — grid-wide barrier for the cooperative (persistent) kernels.
 *
 * Counting barrier over the co-resident blocks of a cooperative launch. The counter is one of two words
 * (CNT_BARRIER, CNT_BARRIER2), zero when the kernel starts: zeroed by a kernel that ran before it and after
 * the word's last user, or by the launcher (a memset), so the k-th barrier of the
 * launch completes when the counter reaches (k + 1) x gridDim.x. Thread 0 of each block keeps k in
 * shared memory, arrives with one fire-and-forget release add and polls the counter with acquire
 * loads; nobody resets anything, so the last block to arrive waits for no extra round trip, and a
 * barrier costs one arrival and the polls (the launch's settings are read once, at its first
 * barrier). Each wait is bounded: a clock64 limit checked every 256 polls, cnt[CNT_BARRIER_LIMIT] x
 * 1024 cycles (b2g_set_barrier_limit; 0 means 2e9 cycles, ~1 s at 2 GHz). cnt[CNT_BARRIER_HOLD] (0
 * unless a test sets it) is added to every wait's target: arrivals that never come, so the wait runs
 * out its limit; it exists to test the timeout path without a fault. On timeout the block sets
 * ST_BARRIER_TIMEOUT in the status word and leaves the kernel; a block waiting at any barrier sees
 * the status at its next check (every 256 polls) and leaves too, so all blocks leave within one
 * limit and the host reports B2G_ERR_TIMEOUT (kernels launched later return at once). Thread 0
 * decides for its block and broadcasts through shared memory, so all threads of a block see the
 * same result. Every cooperative kernel calls grid_barrier_start() first.
 *
 * A grid that was launched as one thread-block cluster (worlds of a few thousand bodies: launch_front,
 * launch_back) takes the hardware's cluster barrier instead, whose release and acquire order global
 * memory between the cluster's blocks in the same way: about 0.3 us where the counting barrier of 152
 * blocks takes 1.4 us. It needs no counter and no limit (the blocks of a cluster run at the same time);
 * a kernel launched so calls barriers_held() at its start instead, which stands for the first barrier's
 * wait when a test holds the barriers.
 */
#ifndef B2G_SYNC_CUH
#define B2G_SYNC_CUH

#include "b2g_internal.h"

namespace b2g {

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add_gpu(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

/* blocks of this block's cluster; the whole grid when it was launched as one cluster */
__device__ __forceinline__ unsigned cluster_blocks() {
    unsigned n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

/* barriers this block has passed in the current launch, and the launch's wait limit and held
 * arrivals (used by thread 0) */
static __shared__ unsigned b2g_barrier_epoch;
static __shared__ long long b2g_barrier_limit;
static __shared__ unsigned b2g_barrier_hold;
static __shared__ int b2g_barrier_word;

/* word: the launch's counter, CNT_BARRIER or CNT_BARRIER2 */
__device__ __forceinline__ void grid_barrier_start(int word = CNT_BARRIER) {
    if (threadIdx.x == 0) {  /* ordered by the barrier's first __syncthreads */
        b2g_barrier_epoch = 0u;
        b2g_barrier_word = word;
    }
}

/* Thread 0's wait until the launch's counter (in the block cnt, which also holds CNT_STATUS) has reached
 * `target` arrivals; false when it ran out or another block's did. */
__device__ __forceinline__ bool grid_wait(int* cnt, unsigned target) {
    const unsigned* count = (const unsigned*)&cnt[b2g_barrier_word];
    target += b2g_barrier_hold;
    const long long t0 = clock64();
    unsigned polls = 0;
    while ((int)(ld_acquire_gpu(count) - target) < 0) {
        if ((++polls & 255u) == 0u) {
            if (((volatile int*)cnt)[CNT_STATUS] & ST_BARRIER_TIMEOUT) return false;
            if (clock64() - t0 > b2g_barrier_limit) {
                atomicOr((unsigned*)&cnt[CNT_STATUS], ST_BARRIER_TIMEOUT);
                return false;
            }
        }
    }
    return true;
}
/* thread 0's arrival at the next barrier of the launch, for `blocks` blocks; returns the barrier's number */
__device__ __forceinline__ unsigned grid_arrive(int* cnt, unsigned blocks) {
    if (b2g_barrier_epoch == 0u) {
        int2 lim_hold;
        asm volatile("ld.volatile.global.v2.s32 {%0, %1}, [%2];"
                     : "=r"(lim_hold.x), "=r"(lim_hold.y) : "l"(&cnt[CNT_BARRIER_LIMIT]) : "memory");
        b2g_barrier_limit = lim_hold.x > 0 ? (long long)lim_hold.x << 10 : 2000000000LL;
        b2g_barrier_hold = (unsigned)max(lim_hold.y, 0);
    }
    ++b2g_barrier_epoch;
    if (blocks) red_release_add_gpu((unsigned*)&cnt[b2g_barrier_word], blocks);
    return b2g_barrier_epoch;
}
/* the grid is one cluster: its barrier */
__device__ __forceinline__ bool grid_is_cluster() { return cluster_blocks() == gridDim.x; }
__device__ __forceinline__ void cluster_grid_barrier() {
    if (gridDim.x == 1) __syncthreads();
    else cluster_barrier();
}

/* cnt: the counter block */
__device__ __forceinline__ bool grid_barrier(int* cnt) {
    __shared__ int s_ok;
    if (grid_is_cluster()) {
        cluster_grid_barrier();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_ok = grid_wait(cnt, grid_arrive(cnt, 1u) * gridDim.x) ? 1 : 0;
    __syncthreads();
    return s_ok != 0;
}

/* A barrier in two halves around work of one block, `one`: grid_gather returns to that block when every
 * block has arrived (to the others at once), grid_release to the others when that block has come to it.
 * Work that would take several grid barriers when it is spread over the blocks takes __syncthreads there. */
__device__ __forceinline__ bool grid_gather(int* cnt, int one) {
    __shared__ int s_ok;
    if (grid_is_cluster()) {
        cluster_grid_barrier();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned k = grid_arrive(cnt, 1u);
        s_ok = (int)blockIdx.x != one || grid_wait(cnt, k * gridDim.x) ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}
__device__ __forceinline__ bool grid_release(int* cnt, int one) {
    __shared__ int s_ok;
    if (grid_is_cluster()) {
        cluster_grid_barrier();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool mine = (int)blockIdx.x == one;
        const unsigned k = grid_arrive(cnt, mine ? gridDim.x : 0u);
        s_ok = mine || grid_wait(cnt, k * gridDim.x) ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ bool grid_barrier(const DevWorld& w) { return grid_barrier(w.cnt); }

/* Barriers held by a test (CNT_BARRIER_HOLD), in a kernel launched as one cluster: each block waits out
 * the limit, as at its first barrier, and sets the status. Every thread of the grid calls it and all get
 * the same answer: true, leave the kernel. */
__device__ __forceinline__ bool barriers_held(const DevWorld& w) {
    int2 lim_hold;
    asm volatile("ld.volatile.global.v2.s32 {%0, %1}, [%2];"
                 : "=r"(lim_hold.x), "=r"(lim_hold.y) : "l"(&w.cnt[CNT_BARRIER_LIMIT]) : "memory");
    if (lim_hold.y <= 0) return false;
    if (threadIdx.x == 0) {
        const long long limit = lim_hold.x > 0 ? (long long)lim_hold.x << 10 : 2000000000LL;
        const long long t0 = clock64();
        while (clock64() - t0 <= limit && !(((volatile int*)w.cnt)[CNT_STATUS] & ST_BARRIER_TIMEOUT)) __nanosleep(500);
        atomicOr((unsigned*)&w.cnt[CNT_STATUS], ST_BARRIER_TIMEOUT);
    }
    return true;
}

/* whether a kernel launched as one cluster leaves at its start: the world was aborted, or its barriers
 * are held (then every block leaves, whichever of the two it sees) */
__device__ __forceinline__ bool cluster_leaves(const DevWorld& w) {
    const bool aborted = world_aborted(w.cnt);
    return barriers_held(w) || aborted;
}

}  // namespace b2g
#endif
