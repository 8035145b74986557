/*
 * b2g_tape_record.cuh — the passes that record a taped step around its solver, as kernels of their own
 * (k_adjoint.cu) or, in worlds that step on one cluster, inside k_front (k_solver.cu).
 */
#ifndef B2G_TAPE_RECORD_CUH
#define B2G_TAPE_RECORD_CUH

#include "b2g_sync.cuh"
#include "b2g_tape.h"

namespace b2g {
namespace {

__device__ __forceinline__ bool tape_ok(const TapeDev& t, long long step, long long base, int ncons) {
    return t.cnt[TAPE_CNT_STATUS] == 0 && step < t.step_cap && base + ncons <= t.slot_cap;
}

/* After the colouring: the step's parameters, colour offsets and part rows, a checkpoint every ckpt_every
 * steps, and its solver slots in solve order with where each point's carried impulse came from. */
__device__ __forceinline__ void tape_record(const DevWorld& w, const TapeDev& t, const StepParams& sp) {
    const long long step = t.cnt[TAPE_CNT_STEPS];
    const long long base = t.cnt[TAPE_CNT_SLOTS];
    const int ncons = w.cnt[CNT_CONS];
    const int ncol = w.cnt[CNT_COLOURS];
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsize = gridDim.x * blockDim.x;
    if (!tape_ok(t, step, base, ncons)) {
        if (gtid == 0) t.cnt[TAPE_CNT_STATUS] |= (long long)TAPE_ST_OVERFLOW;
        return;
    }
    if (gtid == 0) {
        TapeStep s;
        s.dt = sp.dt;
        s.dt_ratio = sp.dt_ratio;
        s.gx = sp.gx;
        s.gy = sp.gy;
        s.vi = sp.vi;
        s.pi = sp.pi;
        s.warm = sp.warm;
        s.nslots = ncons;
        s.slot_off = base;
        s.ncol = ncol;
        s.ncontacts = w.cnt[CNT_CONTACTS];
        t.steps[step] = s;
    }
    for (int c = gtid; c <= ncol; c += gsize) t.col_off[(size_t)step * (kMaxColours + 1) + c] = w.col_off[c];
    if (blockIdx.x == 0) {
        /* the part-local layout: one row [n, offsets 0..n] per part, packed into the pool */
        __shared__ int s_row[kMaxParts + 2];
        const int np = w.cnt[CNT_INTERIOR] > 0 ? min(w.cnt[CNT_PARTS], t.max_parts) : 0;
        for (int q = threadIdx.x; q < np; q += blockDim.x) s_row[q] = w.part_ncol[q] + 2;
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int q = 0; q < np; ++q) {
                const int len = s_row[q];
                s_row[q] = acc;
                acc += len;
            }
            const long long at = t.cnt[TAPE_CNT_POOL];
            if (w.cnt[CNT_INTERIOR] > 0 && w.cnt[CNT_PARTS] > t.max_parts) t.cnt[TAPE_CNT_STATUS] |= (long long)TAPE_ST_OVERFLOW;
            if (at + acc > t.pool_cap) {
                t.cnt[TAPE_CNT_STATUS] |= (long long)TAPE_ST_OVERFLOW;
                s_row[kMaxParts + 1] = -1;
            } else {
                t.cnt[TAPE_CNT_POOL] = at + acc;
                s_row[kMaxParts + 1] = (int)at;
                t.part_np[step] = np;
            }
        }
        __syncthreads();
        const int at = s_row[kMaxParts + 1];
        if (at >= 0) {
            for (int q = threadIdx.x; q < np; q += blockDim.x) {
                const int nc = w.part_ncol[q];
                int* row = t.part_pool + at + s_row[q];
                t.part_row[(size_t)step * t.max_parts + q] = at + s_row[q];
                row[0] = nc;
                for (int c = 0; c <= nc; ++c) row[1 + c] = w.part_off[(size_t)q * (kMaxColours + 1) + c];
            }
        }
    }
    if (step % t.ckpt_every == 0) {
        const size_t o = (size_t)(step / t.ckpt_every) * t.n_bodies;
        for (int b = gtid; b < t.n_bodies; b += gsize) {
            const float4 p = w.b_pos[b], v = w.b_vel[b];
            t.ckpt_pos[o + b] = make_float4(p.x, p.y, p.z, 0.0f);
            t.ckpt_vel[o + b] = make_float4(v.x, v.y, v.z, 0.0f);
        }
    }
    int nprev = 0;
    long long prev_off = 0;
    if (step > 0) {
        nprev = t.steps[step - 1].ncontacts;
        prev_off = t.steps[step - 1].slot_off;
    }
    unsigned long long* cur = t.cmap[step & 1];
    const unsigned long long* prev = t.cmap[(step + 1) & 1];
    for (int k = gtid; k < ncons; k += gsize) {
        const int ci = w.s_contact[k];
        const int2 bd = w.c.body[ci];
        const int2 fx = w.c.fix[ci];
        const uint4 ids = w.c.mids[ci];
        const int mtype = (int)(ids.z & 0xffu);
        const int count = (int)((ids.z >> 8) & 0xffu);
        const float4 massA = w.b_mass[bd.x], massB = w.b_mass[bd.y];
        const float2 lcA = w.b_lc[bd.x], lcB = w.b_lc[bd.y];
        const int dyn = ((w.b_flags[bd.x] & BF_TYPE_MASK) == BODY_DYNAMIC ? 1 : 0) |
                        ((w.b_flags[bd.y] & BF_TYPE_MASK) == BODY_DYNAMIC ? 2 : 0);
        int lo = 0, hi = ncol - 1;
        while (lo < hi) { /* last colour whose offset is <= k */
            const int mid = (lo + hi + 1) >> 1;
            if (w.col_off[mid] <= k) lo = mid;
            else hi = mid - 1;
        }
        TapeSlot s;
        s.idx = make_int4(bd.x, bd.y, count | (mtype << 8) | (dyn << 16), lo);
        s.geo = w.c.mgeo[ci];
        s.lp = w.c.mpts[ci];
        s.inv = make_float4(massA.y, massB.y, massA.w, massB.w);
        s.lc = make_float4(lcA.x, lcA.y, lcB.x, lcB.y);
        s.mat = w.c.mat[ci];
        s.rad = make_float4(w.f_shape[fx.x].radius, w.f_shape[fx.y].radius, __int_as_float(w.cons_island[w.s_cons[k]]),
                            __int_as_float(sp.pi));
        s.imp = w.c.mimp[ci];
        int carry[2] = {-1, -1};
        if (step > 0 && count > 0 && nprev > 0) {
            const unsigned long long key = w.c.key[ci];
            int a = 0, b = nprev - 1, found = -1;
            while (a <= b) {
                const int mid = (a + b) >> 1;
                const unsigned long long kk = w.c_alt.key[mid];
                if (kk == key) {
                    found = mid;
                    break;
                }
                if (kk < key) a = mid + 1;
                else b = mid - 1;
            }
            if (found >= 0) {
                const unsigned long long m = prev[found];
                if ((m >> 32) == (unsigned long long)step) {
                    const int pk = (int)(m & 0xffffffffull);
                    const int4 pc = t.slots[prev_off + pk].carry;
                    const int pcount = t.slots[prev_off + pk].idx.z & 0xff;
                    /* the narrowphase's impulse match (b2_contact.rs:277-298) */
                    for (int p = 0; p < count; ++p) {
                        const uint32_t id = p == 0 ? ids.x : ids.y;
                        if (pcount > 0 && (uint32_t)pc.z == id) carry[p] = pk * 2;
                        else if (pcount > 1 && (uint32_t)pc.w == id) carry[p] = pk * 2 + 1;
                    }
                }
            }
        }
        s.carry = make_int4(carry[0], carry[1], (int)ids.x, (int)ids.y);
        t.slots[base + k] = s;
        cur[ci] = ((unsigned long long)(step + 1) << 32) | (unsigned long long)(unsigned)k;
    }
}

/* After the solver: the position iterations each slot's island ran. */
__device__ __forceinline__ void tape_post(const DevWorld& w, const TapeDev& t, const StepParams& sp) {
    const long long step = t.cnt[TAPE_CNT_STEPS];
    const long long base = t.cnt[TAPE_CNT_SLOTS];
    const int ncons = w.cnt[CNT_CONS];
    if (!tape_ok(t, step, base, ncons)) return;
    const float tol = 3.0f * kLinearSlop;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ncons; k += gridDim.x * blockDim.x) {
        const int isl = w.vc_island[k];
        int n = sp.pi;
        for (int j = 0; j < sp.pi; ++j) {
            if (__uint_as_float(w.isl_minsep[(size_t)j * w.body_cap + isl]) <= tol) {
                n = j + 1;
                break;
            }
        }
        t.slots[base + k].rad.w = __int_as_float(n);
    }
}

/* After every thread's tape_post, one thread: the step and its slots are counted. */
__device__ __forceinline__ void tape_advance(const DevWorld& w, const TapeDev& t) {
    const long long step = t.cnt[TAPE_CNT_STEPS];
    const long long base = t.cnt[TAPE_CNT_SLOTS];
    const int ncons = w.cnt[CNT_CONS];
    if (!tape_ok(t, step, base, ncons)) return;
    t.cnt[TAPE_CNT_STEPS] = step + 1;
    t.cnt[TAPE_CNT_SLOTS] = base + ncons;
}

}  // namespace
}  // namespace b2g
#endif
