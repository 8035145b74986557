/*
 * k_toi.cu — time of impact of two moving shapes, many pairs per launch.
 *
 * Reference: b2_time_of_impact (private/collision/b2_time_of_impact.rs:191-463) with its
 * separation function (:10-189), the GJK distance b2_distance_fn
 * (private/collision/b2_distance.rs:331-440) with the simplex (:58-329) and the distance proxy
 * (:8-47, src/b2_distance.rs:12-130), and the sweep (src/b2_math.rs:764-787).
 *
 * One thread per pair runs the routines of b2g_toi.cuh (a long serial chain with little memory
 * traffic, so a pair stays in one thread's registers); results equal the host restatement bit for
 * bit.
 *
 * The caller's arrays (144-byte definitions, 40-byte sweeps) are read as they are, and the shapes
 * (gift-wrapped hulls among them) are built by the pair's thread: 100k pairs take 0.45 ms with the call's
 * overheads, where a host loop over the shapes, copies and allocations took 10.7 ms. A block reads its definitions (up to 128) in one contiguous piece into shared memory
 * (8 bytes a thread, coalesced: the array may lie in host memory, across C2C) and every thread takes
 * its own from there, rows an odd number of words apart so that lanes meet different banks.
 */
#include "b2g_shape.cuh"
#include "b2g_toi.cuh"

namespace b2g {
namespace {

constexpr int kBlock = 128;
constexpr int kDefWords = sizeof(b2g_fixture_def) / 4, kDefRow = kDefWords + 1;
constexpr int kSweepWords = sizeof(b2g_sweep) / 4, kSweepRow = kSweepWords + 1;
static_assert(sizeof(b2g_fixture_def) % 8 == 0 && alignof(b2g_fixture_def) == 8, "definitions are read 8 bytes at a time");

/* the definitions' types: any but the three shapes sets *bad */
__global__ void __launch_bounds__(kBlock) k_toi_check(const b2g_fixture_def* da, const b2g_fixture_def* db, int n, int* bad) {
    bool ok = true;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int ta = da[i].shape_type, tb = db[i].shape_type;
        ok = ok && (unsigned)ta <= (unsigned)B2G_SHAPE_POLYGON && (unsigned)tb <= (unsigned)B2G_SHAPE_POLYGON;
    }
    if (!ok) *(volatile int*)bad = 1;
}

/* items [base, base + m) of an array of `words`-word items into rows of `row` words */
template <typename T>
__device__ __forceinline__ void stage(uint32_t* rows, const T* items, int m, int words, int row) {
    constexpr int per = sizeof(T) / 4;  /* words of one load */
    const int loads = words / per;
    for (int k = threadIdx.x; k < m * loads; k += blockDim.x) {
        const int item = k / loads, at = (k % loads) * per;
        const T v = items[k];
        const uint32_t* w = (const uint32_t*)&v;
#pragma unroll
        for (int q = 0; q < per; ++q) rows[item * row + at + q] = w[q];
    }
}

__device__ __forceinline__ void proxy_of(const uint32_t* row, DistProxy& p) {
    b2g_fixture_def d;
    uint32_t* w = (uint32_t*)&d;
#pragma unroll
    for (int k = 0; k < kDefWords; ++k) w[k] = row[k];
    ShapeRec s;
    build_shape(d, s);
    make_proxy(s, p);
}

__device__ __forceinline__ Sweep sweep_of(const uint32_t* row) {
    auto f = [row](int k) { return __uint_as_float(row[k]); };
    Sweep s;
    s.lc = mk(f(0), f(1));
    s.c0 = mk(f(2), f(3));
    s.c = mk(f(4), f(5));
    s.a0 = f(6);
    s.a = f(7);
    s.alpha0 = f(8);
    return s;
}

__global__ void __launch_bounds__(kBlock) k_time_of_impact(const b2g_fixture_def* da, const b2g_sweep* swa,
                                                           const b2g_fixture_def* db, const b2g_sweep* swb,
                                                           const float* t_max, int n, int per, b2g_toi_output* out,
                                                           const int* bad) {
    __shared__ uint32_t s_rows[kBlock * kDefRow];
    static_assert(kDefRow >= 2 * kSweepRow, "two sweeps fit a definition's row");
    if (__syncthreads_or(threadIdx.x == 0 && *(const volatile int*)bad != 0)) return;
    /* `per` pairs to a warp (lanes_for); a lane without one only helps to fetch */
    const int items = kBlock / 32 * per;
    const int t = (int)(threadIdx.x & 31) < per ? (int)(threadIdx.x >> 5) * per + (int)(threadIdx.x & 31) : kBlock;
    for (int base = blockIdx.x * items; base < n; base += gridDim.x * items) {
        const int m = min(items, n - base);
        DistProxy pa, pb;
        Sweep a, b;
        __syncthreads();
        stage(s_rows, (const uint2*)(da + base), m, kDefWords, kDefRow);
        __syncthreads();
        if (t < m) proxy_of(s_rows + t * kDefRow, pa);
        __syncthreads();
        stage(s_rows, (const uint2*)(db + base), m, kDefWords, kDefRow);
        __syncthreads();
        if (t < m) proxy_of(s_rows + t * kDefRow, pb);
        __syncthreads();
        stage(s_rows, (const uint32_t*)(swa + base), m, kSweepWords, kSweepRow);
        stage(s_rows + kBlock * kSweepRow, (const uint32_t*)(swb + base), m, kSweepWords, kSweepRow);
        __syncthreads();
        if (t >= m) continue;
        a = sweep_of(s_rows + t * kSweepRow);
        b = sweep_of(s_rows + (kBlock + t) * kSweepRow);
        int state;
        float at;
        time_of_impact(pa, a, pb, b, t_max ? t_max[base + t] : 1.0f, state, at);
        b2g_toi_output o;
        o.state = state;
        o.t = at;
        out[base + t] = o;
    }
}

}  // namespace

void launch_time_of_impact(const b2g_fixture_def* da, const b2g_sweep* swa, const b2g_fixture_def* db,
                           const b2g_sweep* swb, const float* t_max, int n, b2g_toi_output* out, int* bad, cudaStream_t s) {
    const int sms = current_sm_count();
    k_toi_check<<<grid_for(n, kBlock, sms * 8), kBlock, 0, s>>>(da, db, n, bad);
    const int per = lanes_for(n, sms);
    k_time_of_impact<<<grid_for(n, kBlock / 32 * per, sms * 16), kBlock, 0, s>>>(da, swa, db, swb, t_max, n, per, out, bad);
    B2G_LAUNCHED(2);
}

}  // namespace b2g
