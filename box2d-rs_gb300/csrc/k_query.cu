/*
 * k_query.cu — world queries on the step's LBVH: many AABB queries or ray casts in one launch.
 *
 * Reference: B2world::query_aabb and B2world::ray_cast (private/dynamics/b2_world.rs:969-1056)
 * over B2dynamicTree::query / ray_cast (src/b2_dynamic_tree.rs:239-347), with the fixtures' ray
 * casts B2circleShape (private/collision/b2_circle_shape.rs:26-59), B2polygonShape
 * (private/collision/b2_polygon_shape.rs:226-287) and B2edgeShape
 * (private/collision/b2_edge_shape.rs:39-102).
 *
 * The hierarchy walked is the one of the last step's broadphase (fat AABBs as of that step): a thread
 * for each ray, a warp for each box. The queries and their results are the caller's arrays where the
 * device reaches them (Grace's coherent access), so a call is its kernels and a wait: 16k rays and 2k
 * boxes against 20k bodies take 134 + 50 us, and took 373 + 887 us with an allocation for every array,
 * host loops over the results and a host sort of the boxes' pairs. A ray keeps the reference's clipping: every hit clips the segment to its fraction,
 * so the result is the closest hit; only the order in which equally distant fixtures are met can
 * differ from the reference's tree (the GPU keeps the first it meets).
 */
#include <climits>

#include "b2g_internal.h"
#include "b2g_lists.h"
#include "b2g_walk.cuh"

namespace b2g {
namespace {

constexpr int kBlock = 128;
constexpr int kStack = 64;

/* the separating-axis test of the tree ray cast: |dot(v, p1 - c)| - dot(|v|, h) > 0 separates */
__device__ __forceinline__ bool ray_box(const float4 box, const float4 seg, V2 p1, V2 v, V2 abs_v) {
    if (!aabb_overlap(box, seg)) return false;
    const V2 c = scale(0.5f, add(mk(box.x, box.y), mk(box.z, box.w)));
    const V2 h = scale(0.5f, sub(mk(box.z, box.w), mk(box.x, box.y)));
    const float separation = fabsf(dot(v, sub(p1, c))) - dot(abs_v, h);
    return !(separation > 0.0f);
}

__device__ bool shape_ray_cast(const ShapeRec& sh, const Xf& xf, V2 ip1, V2 ip2, float max_fraction, float* fraction,
                               V2* normal) {
    const int type = shape_type(sh);
    if (type == SHAPE_CIRCLE) {
        const V2 position = add(xf.p, mul(xf.q, sh.v[0]));
        const V2 s = sub(ip1, position);
        const float b = dot(s, s) - sh.radius * sh.radius;
        const V2 r = sub(ip2, ip1);
        const float c = dot(s, r);
        const float rr = dot(r, r);
        const float sigma = c * c - rr * b;
        if (sigma < 0.0f || rr < kEpsilon) return false;
        float a = -(c + fsqrt(sigma));
        if (0.0f <= a && a <= max_fraction * rr) {
            a = fdiv(a, rr);
            *fraction = a;
            V2 n = add(s, scale(a, r));
            normalize(n);
            *normal = n;
            return true;
        }
        return false;
    }
    const V2 p1 = mul_t(xf.q, sub(ip1, xf.p));
    const V2 p2 = mul_t(xf.q, sub(ip2, xf.p));
    const V2 d = sub(p2, p1);
    if (type == SHAPE_POLYGON) {
        /* the reference starts the entering bound at 0.032 (b2_polygon_shape.rs:239) */
        float lower = 0.032f, upper = max_fraction;
        int index = -1;
        const int count = shape_count(sh);
        for (int i = 0; i < count; ++i) {
            const float numerator = dot(sh.n[i], sub(sh.v[i], p1));
            const float denominator = dot(sh.n[i], d);
            if (denominator == 0.0f) {
                if (numerator < 0.0f) return false;
            } else if (denominator < 0.0f && numerator < lower * denominator) {
                lower = fdiv(numerator, denominator);
                index = i;
            } else if (denominator > 0.0f && numerator < upper * denominator) {
                upper = fdiv(numerator, denominator);
            }
            if (upper < lower) return false;
        }
        if (index >= 0) {
            *fraction = lower;
            *normal = mul(xf.q, sh.n[index]);
            return true;
        }
        return false;
    }
    /* edge: vertex1 = v[1], vertex2 = v[2] */
    const V2 v1 = sh.v[1], v2 = sh.v[2];
    const V2 e = sub(v2, v1);
    V2 nrm = mk(e.y, -e.x);
    normalize(nrm);
    const float numerator = dot(nrm, sub(v1, p1));
    if (shape_one_sided(sh) && numerator > 0.0f) return false;
    const float denominator = dot(nrm, d);
    if (denominator == 0.0f) return false;
    const float t = fdiv(numerator, denominator);
    if (t < 0.0f || max_fraction < t) return false;
    const V2 q = add(p1, scale(t, d));
    const V2 r = sub(v2, v1);
    const float rr = dot(r, r);
    if (rr == 0.0f) return false;
    const float sf = fdiv(dot(sub(q, v1), r), rr);
    if (sf < 0.0f || 1.0f < sf) return false;
    *fraction = t;
    *normal = numerator > 0.0f ? neg(mul(xf.q, nrm)) : mul(xf.q, nrm);
    return true;
}

__device__ __forceinline__ Xf body_xf(const DevWorld& w, int b) {
    const float4 x = w.b_xf[b];
    Xf xf;
    xf.p = mk(x.x, x.y);
    xf.q.s = x.z;
    xf.q.c = x.w;
    return xf;
}

/* one thread per ray, `per` rays to a warp (lanes_for). A world whose status holds an error answers
 * nothing: the caller reports it */
__global__ void __launch_bounds__(kBlock) k_ray_cast(DevWorld w, const float* rays, const uint32_t* ray_world, int n,
                                                     int per, b2g_ray_hit* out) {
    if (((volatile int*)w.cnt)[CNT_STATUS] & ~ST_STACK_OVERFLOW) return;
    const int lane = threadIdx.x & 31, warps = (int)blockDim.x >> 5;
    if (lane >= per) return;
    for (int i = (blockIdx.x * warps + ((int)threadIdx.x >> 5)) * per + lane; i < n; i += gridDim.x * warps * per) {
        const float4 ray = make_float4(rays[4 * (size_t)i], rays[4 * (size_t)i + 1], rays[4 * (size_t)i + 2],
                                       rays[4 * (size_t)i + 3]);
        const V2 p1 = mk(ray.x, ray.y), p2 = mk(ray.z, ray.w);
        int hit = -1;
        V2 hit_point = mk(0.0f, 0.0f), hit_normal = mk(0.0f, 0.0f);
        float hit_fraction = 1.0f;
        const uint32_t wd = ray_world ? ray_world[i] : 0u;
        if (wd < (uint32_t)w.num_worlds) {
            V2 r = sub(p2, p1);
            normalize(r);
            const V2 v = mk(-1.0f * r.y, 1.0f * r.x);
            const V2 abs_v = mk(fabsf(v.x), fabsf(v.y));
            float max_fraction = 1.0f;
            auto seg_box = [&]() {
                const V2 t = add(p1, scale(max_fraction, sub(p2, p1)));
                const V2 lo = vmin(p1, t), hi = vmax(p1, t);
                return make_float4(lo.x, lo.y, hi.x, hi.y);
            };
            float4 seg = seg_box();
            auto leaf = [&](int p) {
                const int f = (int)w.bp_val[p];
                float fraction;
                V2 normal;
                if (shape_ray_cast(w.f_shape[f], body_xf(w, w.f_body[f]), p1, p2, max_fraction, &fraction, &normal)) {
                    hit = f;
                    hit_point = add(scale(1.0f - fraction, p1), scale(fraction, p2));
                    hit_normal = normal;
                    hit_fraction = fraction;
                    max_fraction = fraction;
                    seg = seg_box();
                }
            };
            /* the world's hierarchy, then the one of its large static proxies */
            for (int h = 0; h < 2; ++h) {
                const int root = w.bp_world_root[wd + (h ? (uint32_t)w.num_worlds : 0u)];
                if (root == INT_MIN) continue;
                if (root < 0) {  /* a hierarchy of one proxy */
                    if (ray_box(w.bp_leaf[~root], seg, p1, v, abs_v)) leaf(~root);
                    continue;
                }
                int stack[kStack];
                int top = 0;
                stack[top++] = root;
                while (top > 0) {
                    const int node = stack[--top];
                    const int2 ch = w.bp_node_child[node];
                    const float4 boxes[2] = {w.bp_node_b0[node], w.bp_node_b1[node]};
                    const int kids[2] = {ch.x, ch.y};
                    for (int c = 0; c < 2; ++c) {
                        if (!ray_box(boxes[c], seg, p1, v, abs_v)) continue;
                        if (kids[c] < 0) leaf(~kids[c]);
                        else if (top < kStack) stack[top++] = kids[c];
                        else atomicOr((unsigned*)&w.cnt[CNT_STATUS], ST_STACK_OVERFLOW);
                    }
                }
            }
        }
        b2g_ray_hit h;
        h.fixture = hit;
        h.point = b2g_vec2{hit_point.x, hit_point.y};
        h.normal = b2g_vec2{hit_normal.x, hit_normal.y};
        h.fraction = hit_fraction;
        out[i] = h;
    }
}

/* The fixtures whose fat AABBs overlap each box, in two kernels. k_query_find: a warp walks the hierarchy
 * for its box (up to 32 pending nodes a round, from a stack in shared memory) and keeps what it finds in shared
 * memory; the box's list then goes to a piece of `found` that it reserves with one atomic (a longer list
 * than fits is written by a second walk). lists[i] = (first entry, entries); *total counts all of them,
 * written or not, in 64 bits: boxes over a whole world of 250k fixtures pass 31 bits at 8600 of them. k_query_write: the lists in the order of the boxes, each by fixture. */
constexpr int kBoxWarps = 4;
constexpr int kFoundMax = 256;   /* a box's fixtures kept in shared memory */
constexpr int kRankMax = 1024;   /* longer lists are left to the host to sort */

__global__ void __launch_bounds__(32 * kBoxWarps) k_query_find(DevWorld w, const float* boxes, const uint32_t* box_world,
                                                               int n, uint32_t* found, int cap, int2* lists,
                                                               unsigned long long* total) {
    if (((volatile int*)w.cnt)[CNT_STATUS] & ~ST_STACK_OVERFLOW) return;
    __shared__ int s_pend[kBoxWarps][kPendMax];
    __shared__ uint32_t s_found[kBoxWarps][kFoundMax];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    for (int i = blockIdx.x * kBoxWarps + wid; i < n; i += gridDim.x * kBoxWarps) {
        const float v = lane < 4 ? boxes[4 * (size_t)i + lane] : 0.0f;
        const float4 q = make_float4(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1),
                                     __shfl_sync(0xffffffffu, v, 2), __shfl_sync(0xffffffffu, v, 3));
        const uint32_t wd = box_world ? box_world[i] : 0u;
        int count = 0;
        if (wd < (uint32_t)w.num_worlds)
            walk_box(w, q, wd, s_pend[wid], [&](bool ok, int p) {
                const unsigned who = __ballot_sync(0xffffffffu, ok);
                const int at = count + __popc(who & below);
                if (ok && at < kFoundMax) s_found[wid][at] = w.bp_val[p];
                count += __popc(who);
            });
        __syncwarp();
        unsigned long long place = 0;
        if (lane == 0 && count > 0) place = atomicAdd(total, (unsigned long long)count);
        place = __shfl_sync(0xffffffffu, place, 0);
        if (!list_fits(place, count, cap)) continue;  /* the caller learns the total and asks again with room for it */
        const int first = (int)place;
        if (lane == 0) lists[i] = make_int2(first, count);
        if (count <= kFoundMax) {
            for (int k = lane; k < count; k += 32) found[first + k] = s_found[wid][k];
        } else {
            int done = 0;
            walk_box(w, q, wd, s_pend[wid], [&](bool ok, int p) {
                const unsigned who = __ballot_sync(0xffffffffu, ok);
                if (ok) found[first + done + __popc(who & below)] = w.bp_val[p];
                done += __popc(who);
            });
        }
        __syncwarp();
    }
}

/* A block of 8 warps takes 8 boxes at a time; their lists start after all those of the boxes before,
 * whose entries the block adds up itself. *unsorted: a list longer than kRankMax was written as found */
__global__ void __launch_bounds__(256) k_query_write(int n, const uint32_t* found, const int2* lists, uint32_t* out,
                                                     int* unsorted) {
    __shared__ int s_sum[8];
    __shared__ int s_count[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int before = 0, next = 0;  /* entries of the boxes before `next` */
    for (int base = blockIdx.x * 8; base < n; base += gridDim.x * 8) {
        int sum = 0;
        for (int i = next + threadIdx.x; i < base; i += 256) sum += lists[i].y;
        next = base;
        sum = __reduce_add_sync(0xffffffffu, sum);
        __syncthreads();
        const int i = base + wid;
        const int2 list = i < n ? lists[i] : make_int2(0, 0);
        if (lane == 0) {
            s_sum[wid] = sum;
            s_count[wid] = list.y;
        }
        __syncthreads();
        for (int k = 0; k < 8; ++k) before += s_sum[k];
        int at = before;
        for (int k = 0; k < wid; ++k) at += s_count[k];
        const uint32_t* f = found + list.x;
        for (int k = lane; k < list.y; k += 32) {
            const uint32_t mine = f[k];
            int rank = k;
            if (list.y <= kRankMax) {
                rank = 0;
                for (int j = 0; j < list.y; ++j) rank += f[j] < mine ? 1 : 0;
            }
            out[2 * (size_t)(at + rank)] = (uint32_t)i;
            out[2 * (size_t)(at + rank) + 1] = mine;
        }
        if (lane == 0 && list.y > kRankMax) *(volatile int*)unsorted = 1;
    }
}

/* the status word, and a count if there is one, where the host reads them */
__global__ void k_query_end(DevWorld w, const unsigned long long* total, int* status, unsigned long long* total_out) {
    *status = ((volatile int*)w.cnt)[CNT_STATUS];
    if (total) *total_out = *total;
}

}  // namespace

void launch_ray_cast(const DevWorld& w, const float* rays, const uint32_t* ray_world, int n, b2g_ray_hit* out, int* status,
                     cudaStream_t s) {
    const int per = lanes_for(n, w.num_sms);
    k_ray_cast<<<grid_for(n, kBlock / 32 * per, w.num_sms * 16), kBlock, 0, s>>>(w, rays, ray_world, n, per, out);
    k_query_end<<<1, 1, 0, s>>>(w, nullptr, status, nullptr);
    B2G_LAUNCHED(2);
}

void launch_query_find(const DevWorld& w, const float* boxes, const uint32_t* box_world, int n, uint32_t* found, int cap,
                       int2* lists, unsigned long long* total, int* status, unsigned long long* total_out, cudaStream_t s) {
    k_query_find<<<grid_for(n, kBoxWarps, w.num_sms * 16), 32 * kBoxWarps, 0, s>>>(w, boxes, box_world, n, found, cap,
                                                                                  lists, total);
    k_query_end<<<1, 1, 0, s>>>(w, total, status, total_out);
    B2G_LAUNCHED(2);
}

void launch_query_write(const DevWorld& w, int n, const uint32_t* found, const int2* lists, uint32_t* out, int* unsorted,
                        cudaStream_t s) {
    k_query_write<<<grid_for(n, 8, w.num_sms * 8), 256, 0, s>>>(n, found, lists, out, unsorted);
    B2G_LAUNCHED(1);
}

}  // namespace b2g
