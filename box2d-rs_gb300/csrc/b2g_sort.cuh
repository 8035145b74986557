/*
 * b2g_sort.cuh — block scan and the stable 8-bit-digit radix sort of (64-bit key, 32-bit value) pairs by
 * a whole grid, shared by the device-wide sort (k_prims.cu) and the broadphase's one-cluster kernel
 * (k_broadphase.cu).
 */
#ifndef B2G_SORT_CUH
#define B2G_SORT_CUH

#include "b2g_internal.h"
#include "b2g_sync.cuh"

namespace b2g {
namespace {

constexpr int kSortBlock = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortBlock * kSortItems;

/* block-wide exclusive scan of one value per thread; returns the block total in *total */
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t warp_sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < nwarps ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;  /* inclusive */
    }
    __syncthreads();
    uint32_t warp_prefix = warp > 0 ? warp_sums[warp - 1] : 0u;
    *total = warp_sums[nwarps - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

/* Stable scatter of one 2048-item tile given its per-digit output bases in s_base. */
__device__ void scatter_tile(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                             unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, int n, int shift,
                             int tile_base, const uint32_t* s_base, uint32_t* s_run, uint32_t (*s_warp)[256]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s_run[threadIdx.x] = 0;
    for (int w = 0; w < 8; ++w) s_warp[w][threadIdx.x] = 0;
    __syncthreads();
    const unsigned lt_mask = (1u << lane) - 1u;
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = tile_base + r * kSortBlock + threadIdx.x;
        const bool valid = idx < n;
        unsigned long long k = 0;
        uint32_t v = 0;
        uint32_t d = 256u + (uint32_t)lane;
        if (valid) {
            k = kin[idx];
            v = vin[idx];
            d = (uint32_t)(k >> shift) & 255u;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rank = (uint32_t)__popc(peers & lt_mask);
        if (valid && (peers & lt_mask) == 0u) s_warp[warp][d] = (uint32_t)__popc(peers);
        __syncthreads();
        {
            const int dd = threadIdx.x;
            uint32_t run = s_run[dd];
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                uint32_t c = s_warp[w][dd];
                s_warp[w][dd] = run;
                run += c;
            }
            s_run[dd] = run;
        }
        __syncthreads();
        if (valid) {
            const uint32_t dst = s_base[d] + s_warp[warp][d] + rank;
            if (dst < (uint32_t)n) {
                kout[dst] = k;
                vout[dst] = v;
            }
        }
        __syncthreads();
        for (int w = 0; w < 8; ++w) s_warp[w][threadIdx.x] = 0;
        __syncthreads();
    }
}

/* 256-bin histogram of one tile into s_cnt (block-wide) */
__device__ void tile_histogram(const unsigned long long* __restrict__ keys, int n, int shift, int tile_base, uint32_t* s_cnt) {
    s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < kSortTile; i += kSortBlock) {
        const int idx = tile_base + i;
        if (idx < n) atomicAdd(&s_cnt[(unsigned)(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
}

/* Stable LSD radix sort of n (key, value) pairs by key bits [0, bits) by a whole grid of kSortBlock
 * threads a block (cooperative, or one cluster), two grid barriers per 8-bit pass; the result is in
 * (ka, va). At most one tile is sorted by block 0 alone (no grid barrier). Returns false when a barrier
 * timed out. */
__device__ __forceinline__ bool radix_sort_grid(unsigned long long* ka, uint32_t* va, unsigned long long* kb, uint32_t* vb,
                                                int n, int bits, uint32_t* hist, int* cnt) {
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_run[256];
    __shared__ uint32_t s_warp[8][256];
    __shared__ uint32_t s_cnt[256];
    const int passes = (bits + 7) / 8;
    if (n <= 0 || passes <= 0) return true;
    if (n <= kSortTile) {
        /* one tile: block 0 sorts alone, synchronising with __syncthreads only */
        if (blockIdx.x != 0) return true;
        unsigned long long *kin = ka, *kout = kb;
        uint32_t *vin = va, *vout = vb;
        for (int p = 0; p < passes; ++p) {
            tile_histogram(kin, n, 8 * p, 0, s_cnt);
            uint32_t total;
            const uint32_t ex = block_exclusive_scan(s_cnt[threadIdx.x], &total);
            s_base[threadIdx.x] = ex;
            __syncthreads();
            scatter_tile(kin, vin, kout, vout, n, 8 * p, 0, s_base, s_run, s_warp);
            __syncthreads();
            unsigned long long* tk = kin; kin = kout; kout = tk;
            uint32_t* tv = vin; vin = vout; vout = tv;
        }
        if (kin != ka)
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                ka[i] = kin[i];
                va[i] = vin[i];
            }
        return true;
    }
    const int tiles = (n + kSortTile - 1) / kSortTile;
    unsigned long long *kin = ka, *kout = kb;
    uint32_t *vin = va, *vout = vb;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        /* H: per-tile digit counts, tile-major */
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            tile_histogram(kin, n, shift, t * kSortTile, s_cnt);
            hist[(size_t)t * 256 + threadIdx.x] = s_cnt[threadIdx.x];
            __syncthreads();
        }
        if (!grid_barrier(cnt)) return false;
        /* X: a block with tiles derives its digit bases itself (thread d sums digit d over the
         * tiles: the digit's total and the counts of the tiles before each of its own), then
         * scatters its tiles stably; no separate scan phase and barrier */
        if ((int)blockIdx.x < tiles) {
            const int d = threadIdx.x;
            uint32_t tot = 0;
#pragma unroll 8
            for (int t = 0; t < tiles; ++t) tot += hist[(size_t)t * 256 + d];
            uint32_t total;
            const uint32_t digit_base = block_exclusive_scan(tot, &total);
            uint32_t before = 0;
            int next = 0;
            for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
                for (; next < t; ++next) before += hist[(size_t)next * 256 + d];
                s_base[d] = digit_base + before;
                __syncthreads();
                scatter_tile(kin, vin, kout, vout, n, shift, t * kSortTile, s_base, s_run, s_warp);
                __syncthreads();
            }
        }
        if (!grid_barrier(cnt)) return false;
        unsigned long long* tk = kin; kin = kout; kout = tk;
        uint32_t* tv = vin; vin = vout; vout = tv;
    }
    if (kin != ka) {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            ka[i] = kin[i];
            va[i] = vin[i];
        }
    }
    return true;
}

}  // namespace
}  // namespace b2g
#endif
