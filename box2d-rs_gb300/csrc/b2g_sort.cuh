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

/* Stable scatter of one tile of 256 x items pairs given its per-digit output bases in s_base. A warp takes
 * 32 x items neighbours, groups equal digits row by row and counts them in its own row of s_warp; one prefix
 * over the warps then places every item, so a tile takes two block barriers whatever its rows. */
__device__ void scatter_tile(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                             unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, int n, int shift,
                             int tile_base, int items, const uint32_t* s_base, uint32_t (*s_warp)[256]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = tile_base + warp * 32 * items;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned long long k[kSortItems];
    uint32_t v[kSortItems], at[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = first + r * 32 + lane;
        const bool valid = r < items && idx < n;
        k[r] = valid ? kin[idx] : 0ull;
        v[r] = valid ? vin[idx] : 0u;
    }
    for (int q = lane; q < 256; q += 32) s_warp[warp][q] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        if (r >= items) break;
        const bool valid = first + r * 32 + lane < n;
        const uint32_t d = valid ? (uint32_t)(k[r] >> shift) & 255u : 256u + (uint32_t)lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        at[r] = (valid ? s_warp[warp][d] : 0u) + (uint32_t)__popc(peers & lt_mask);
        __syncwarp();
        if (valid && (peers & lt_mask) == 0u) s_warp[warp][d] += (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t run = s_base[threadIdx.x];
#pragma unroll
        for (int q = 0; q < kSortBlock / 32; ++q) {
            const uint32_t c = s_warp[q][threadIdx.x];
            s_warp[q][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        if (r >= items || first + r * 32 + lane >= n) break;
        const uint32_t dst = s_warp[warp][(uint32_t)(k[r] >> shift) & 255u] + at[r];
        if (dst < (uint32_t)n) {
            kout[dst] = k[r];
            vout[dst] = v[r];
        }
    }
}

/* 256-bin histogram of one tile of 256 x items into s_cnt (block-wide) */
__device__ void tile_histogram(const unsigned long long* __restrict__ keys, int n, int shift, int tile_base, int items,
                               uint32_t* s_cnt) {
    s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < items * kSortBlock; i += kSortBlock) {
        const int idx = tile_base + i;
        if (idx < n) atomicAdd(&s_cnt[(unsigned)(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
}

/* tiles of the largest input for which radix_sort_hist_size(max_n) was allocated, and twice as many smaller */
__device__ __forceinline__ int sort_hist_tiles(int max_n) { return 2 * ((max_n + kSortTile - 1) / kSortTile); }

/* Stable LSD radix sort of n (key, value) pairs by key bits [0, bits) by a whole grid of kSortBlock
 * threads a block (cooperative, or one cluster), two grid barriers per 8-bit pass; the result is in
 * (ka, va). At most one tile is sorted by block 0 alone (no grid barrier). A tile has as few rows of 256 as
 * the blocks and the histograms (max_tiles of them) allow: the rows of a tile follow each other, the tiles do
 * not. 100k keys of 23 bits and their making 41 us, 56 with tiles of 2048 (49 of 152 blocks at work) and
 * four barriers for each row; 4000 on a cluster of 16 blocks 18 and 41; nine keys of 30 bits, alone in their
 * tile, with the merge 39 and 55. Returns false when a barrier timed out. */
__device__ __forceinline__ bool radix_sort_grid(unsigned long long* ka, uint32_t* va, unsigned long long* kb, uint32_t* vb,
                                                int n, int bits, uint32_t* hist, int* cnt, int max_tiles) {
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_warp[kSortBlock / 32][256];
    __shared__ uint32_t s_cnt[256];
    const int passes = (bits + 7) / 8;
    if (n <= 0 || passes <= 0) return true;
    if (n <= kSortTile) {
        /* one tile: block 0 sorts alone, synchronising with __syncthreads only */
        if (blockIdx.x != 0) return true;
        const int items = (n + kSortBlock - 1) / kSortBlock;
        unsigned long long *kin = ka, *kout = kb;
        uint32_t *vin = va, *vout = vb;
        for (int p = 0; p < passes; ++p) {
            tile_histogram(kin, n, 8 * p, 0, items, s_cnt);
            uint32_t total;
            const uint32_t ex = block_exclusive_scan(s_cnt[threadIdx.x], &total);
            s_base[threadIdx.x] = ex;
            __syncthreads();
            scatter_tile(kin, vin, kout, vout, n, 8 * p, 0, items, s_base, s_warp);
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
    const int spread = max(1, min((int)gridDim.x, max_tiles));
    const int items = min(kSortItems, (n + spread * kSortBlock - 1) / (spread * kSortBlock));
    const int tile = items * kSortBlock;
    const int tiles = (n + tile - 1) / tile;
    unsigned long long *kin = ka, *kout = kb;
    uint32_t *vin = va, *vout = vb;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        /* H: per-tile digit counts, tile-major */
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            tile_histogram(kin, n, shift, t * tile, items, s_cnt);
            hist[(size_t)t * 256 + threadIdx.x] = s_cnt[threadIdx.x];
            __syncthreads();
        }
        if (!grid_barrier(cnt)) return false;
        /* X: a block with tiles derives its digit bases itself (thread d sums digit d over the
         * tiles: the digit's total and the counts of the tiles before each of its own), then
         * scatters its tiles stably; no separate scan phase and barrier */
        if ((int)blockIdx.x < tiles) {
            const int d = threadIdx.x;
            uint32_t tot = 0, before = 0;
#pragma unroll 16
            for (int t = 0; t < tiles; ++t) {
                const uint32_t c = hist[(size_t)t * 256 + d];
                tot += c;
                before += t < (int)blockIdx.x ? c : 0u;
            }
            uint32_t total;
            const uint32_t digit_base = block_exclusive_scan(tot, &total);
            int next = blockIdx.x;
            for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
                for (; next < t; ++next) before += hist[(size_t)next * 256 + d];
                s_base[d] = digit_base + before;
                __syncthreads();
                scatter_tile(kin, vin, kout, vout, n, shift, t * tile, items, s_base, s_warp);
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
