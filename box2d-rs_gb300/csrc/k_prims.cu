/*
 * k_prims.cu — device-wide stable sort of (64-bit key, 32-bit value) pairs.
 *
 * The count comes from device memory (d_n), so a step can chain the sort after kernels that produce a variable
 * number of items without a host round trip; grids are sized for the capacity. Between one tile and kRankSort
 * pairs a rank count in three kernels, else the radix sort of b2g_sort.cuh as one cooperative launch.
 */
#include <algorithm>
#include <mutex>
#include <vector>

#include "b2g_sort.cuh"

namespace b2g {

unsigned long long g_kernel_launches = 0;

int current_sm_count() {
    static std::mutex m;
    static std::vector<int> counts;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 1;
    std::lock_guard<std::mutex> lock(m);
    if ((int)counts.size() <= dev) counts.resize((size_t)dev + 1, 0);
    if (counts[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 1;
        counts[dev] = n;
    }
    return counts[dev];
}

namespace {

__device__ __forceinline__ int load_n(const int* d_n, int max_n) {
    if (!d_n) return max_n;
    int n = *d_n;
    return n < max_n ? n : max_n;
}

/* Between one tile and kRankSort pairs, the sort is a rank count instead of the multi-block radix
 * sort (whose two grid barriers per 8-bit pass dominate a few thousand keys): a block takes one
 * tile x of keys and a slice of the tiles y; each thread counts, for its key of tile x, the keys of
 * those tiles that precede it in (key, input position) order and adds the count to the key's rank
 * (one atomic per key and slice); the keys then go to their ranks. The order is the radix sort's
 * (stable: equal keys keep their input order). A fixed grid of kRankBlocks is mapped onto the
 * tiles and slices of the actual count. */
constexpr int kRankSort = 8192;  /* the count is quadratic: beyond this the radix sort is faster */
constexpr int kRankTile = 256;
constexpr int kRankBlocks = 1024;

__global__ void __launch_bounds__(kRankTile) k_rank_count(const unsigned long long* __restrict__ keys, const int* d_n,
                                                          int max_n, uint32_t* rank, int* cnt) {
    pdl_entry();
    if (world_aborted(cnt)) return;
    const int n = load_n(d_n, max_n);
    if (n <= kSortTile || n > kRankSort) return;
    __shared__ unsigned long long s_k[kRankTile];
    const int tiles = (n + kRankTile - 1) / kRankTile;
    const int slices = max(1, min(tiles, (int)gridDim.x / tiles));
    if ((int)blockIdx.x >= tiles * slices) return;
    const int tx = blockIdx.x % tiles, sl = blockIdx.x / tiles;
    const int per = (tiles + slices - 1) / slices;
    const int y0 = sl * per, y1 = min(tiles, y0 + per);
    const int j = tx * kRankTile + threadIdx.x;
    const unsigned long long kj = j < n ? keys[j] : 0ull;
    uint32_t r = 0;
    for (int ty = y0; ty < y1; ++ty) {
        const int i0 = ty * kRankTile;
        const int m = min(kRankTile, n - i0);
        __syncthreads();  /* the previous tile's keys are no longer read */
        if (threadIdx.x < m) s_k[threadIdx.x] = keys[i0 + threadIdx.x];
        __syncthreads();
        for (int i = 0; i < m; ++i) {
            const unsigned long long ki = s_k[i];
            r += (ki < kj || (ki == kj && i0 + i < j)) ? 1u : 0u;
        }
    }
    if (j < n && r) atomicAdd(&rank[j], r);
}

__global__ void k_rank_scatter(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                               unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, const int* d_n,
                               int max_n, const uint32_t* rank, int* cnt) {
    pdl_entry();
    if (world_aborted(cnt)) return;
    const int n = load_n(d_n, max_n);
    if (n <= kSortTile || n > kRankSort) return;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t r = rank[j];
        if (r < (uint32_t)n) {
            kout[r] = kin[j];
            vout[r] = vin[j];
        }
    }
}

__global__ void k_rank_copy(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                            unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, const int* d_n, int max_n,
                            int* cnt) {
    pdl_entry();
    if (world_aborted(cnt)) return;
    const int n = load_n(d_n, max_n);
    if (n <= kSortTile || n > kRankSort) return;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        kout[j] = kin[j];
        vout[j] = vin[j];
    }
}

__global__ void __launch_bounds__(kSortBlock) k_radix_coop(unsigned long long* ka, uint32_t* va, unsigned long long* kb,
                                                           uint32_t* vb, const int* d_n, int max_n, int bits,
                                                           uint32_t* hist, int* cnt, int barrier_word) {
    if (world_aborted(cnt)) return;
    grid_barrier_start(barrier_word);
    const int n = load_n(d_n, max_n);
    if (n > kSortTile && n <= kRankSort && max_n > kSortTile) return;  /* the rank count sorted it */
    radix_sort_grid(ka, va, kb, vb, n, bits, hist, cnt, sort_hist_tiles(max_n));
}

}  // namespace

/* words past the ranks in scan_tmp and past the histograms in sort_hist: part of the layout of saved states */
size_t scan_tmp_size(int max_n) { return (size_t)((max_n + 1023) / 1024 + 1); }

void radix_sort_pairs_coop(unsigned long long* key_a, uint32_t* val_a, unsigned long long* key_b, uint32_t* val_b,
                           const int* d_n, int max_n, int bits, uint32_t* hist, int* cnt, cudaStream_t s, int num_sms,
                           int barrier_word, bool zero_or_max) {
    /* one block per SM keeps the grid barrier short */
    const int blocks = num_sms;
    if (max_n > kSortTile && (!zero_or_max || max_n <= kRankSort)) {
        /* the rank count for inputs between one tile and kRankSort keys (each kernel checks n) */
        const int m = std::min(max_n, kRankSort);
        const int tiles = (m + kRankTile - 1) / kRankTile;
        launch_pdl(k_rank_count, kRankBlocks, kRankTile, 0, s, (const unsigned long long*)key_a, d_n, max_n, hist, cnt);
        launch_pdl(k_rank_scatter, tiles, kRankTile, 0, s, (const unsigned long long*)key_a, (const uint32_t*)val_a,
                   key_b, val_b, d_n, max_n, (const uint32_t*)hist, cnt);
        launch_pdl(k_rank_copy, tiles, kRankTile, 0, s, (const unsigned long long*)key_b, (const uint32_t*)val_b, key_a,
                   val_a, d_n, max_n, cnt);
        B2G_LAUNCHED(3);
    }
    void* args[] = {&key_a, &val_a, &key_b, &val_b, (void*)&d_n, &max_n, &bits, &hist, &cnt, &barrier_word};
    cudaLaunchCooperativeKernel((const void*)k_radix_coop, dim3(blocks), dim3(kSortBlock), args, 0, s);
    B2G_LAUNCHED(1);
}

size_t radix_sort_hist_size(int max_n) {
    const int tiles = (max_n + kSortTile - 1) / kSortTile;
    /* the rank count uses the first kRankSort entries */
    static_assert(kRankSort == kSortRankWords, "the callers zero that many");
    return std::max((size_t)tiles * 256 * 2 + scan_tmp_size(tiles * 256) + 16, (size_t)kRankSort);
}

}  // namespace b2g
