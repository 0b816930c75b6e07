// Megakernel over block-local path pools (templates; mega_l0.cu and mega_l2.cu instantiate the SAH
// pairs and the eight-wide tree): the persistent megakernel of large renders.
//
// One thread per path (mega.cuh's k_mega) holds a warp for the longest of its 32 rays at every
// vertex: 5.4 of 32 lanes active on the 1.3M-triangle frame. Here a block owns a pool of path slots
// in device memory and alternates between two phases: every slot whose rays are back is shaded
// (vertices, emission, light sample, BSDF sample, a new path for a free slot), then the block's
// warps trace the extension and shadow rays of all slots from a queue in shared memory, a lane
// taking the next ray as soon as its own is done. Rays still on their way when the queue is empty
// stay in their lanes over the next shading phase, so no block waits for its longest ray. No phase
// leaves the kernel: no launches, no host synchronisation. Renders that fill the slots only once or twice
// gain nothing and stay with k_mega (mega_pool_takes).
//
// Measured on one GB300, device time of the integrator, k_mega -> pools: the 1080p, 16-spp MIS frame of that
// scene 26.3 -> 16.9 ms on the pairs and 30.8 -> 16.2 on the eight-wide tree, its one-sample frame 1.90 -> 1.71 and
// 2.15 -> 1.47, 1.07M paths of the Cornell room 0.72 -> 0.61 and 0.84 -> 0.54, a one-sample 1080p frame of a
// 50,000-triangle soup 4.55 -> 2.81 and 5.40 -> 2.70. What bounds it now (pairs, 8 spp): issue slots (0.48 per cycle and
// scheduler, 15.1 of 32 lanes) and the latency of fetches (6.3 of the stall cycles per issue) at 28 warps per
// SM; three quarters of the time is tracing.
#pragma once

#include "mega.cuh"
#include "wavefront.h"

#include <algorithm>

namespace e8g {

namespace {

// Blocks per SM (72 registers): 6 / 7 / 8 blocks took 21.5 / 19.6 / 20.0 ms per 16-spp frame (before paths were
// numbered tile by tile).
constexpr int kPoolBlocks = 7;
// Slots per block at most (pool_slots).
constexpr uint32_t kPoolSlots = 1024;
// Idle lanes of a warp that wait for each other before they take new rays (4 / 8 / 16: within 2%).
constexpr uint32_t kPoolRefill = 8;

// State of a slot's ray. Extension: no path, on its way (or queued), back with its hit; kRayEnd: the path
// has none and ends once its shadow ray is back. Shadow: none or occluded, on its way, unoccluded.
enum : uint8_t { kRayNone = 0, kRayOut = 1, kRayHit = 2, kRayEnd = 3 };

// A block's slots: arrays of float4, `slots` each. kPoolRad: the radiance the path has gathered, without
// the shadow ray on its way; kPoolShAdd: with it (in the backward, the light sample's term alone).
enum { kPoolIds = 0, kPoolBeta, kPoolDir, kPoolHit, kPoolPos, kPoolShDir, kPoolShAdd, kPoolRad, kPoolArrays };

struct PoolVertex {
    float3 beta, p, n, o;
    int32_t mesh;
    uint32_t depth;
};

struct PoolRays {
    float3 add;        // contribution that needs no shadow ray
    float3 sd, vis;    // shadow ray direction, contribution when unoccluded
    float st;          // shadow ray length
    uint32_t occ_nan;  // channels that an occluded sample turns into NaN (reference estimators)
    float3 i;          // extension direction
    float pdf;
    bool shadow, extend;
};

// One vertex up to its rays (mega_step's draws and arithmetic): v.beta becomes the throughput
// after the extension.
template <int MODE, class R>
__device__ __forceinline__ void pool_shade(DevScene const &S, RenderArgs const &A, PoolVertex &v, R &rng, PoolRays &q) {
    q.add = q.vis = f3(0, 0, 0);
    q.sd = q.i = f3(0, 0, 1);
    q.st = q.pdf = 0.0f;
    q.occ_nan = 0;
    q.shadow = q.extend = false;
    const DevMaterial &m = vert_mat(S, v.mesh);
    float3 bl = v.beta;
    if (MODE != E8G_MODE_REF_DIRECT) {
        if ((A.max_depth && v.depth >= A.max_depth) || v.depth >= kHardDepth)
            return;
        float surv = A.rr_prob;
        if (v.depth >= A.rr_start) {
            if (rng.next() >= surv)
                return;
        }
        if (MODE == E8G_MODE_MIS) {
            if (v.depth >= A.rr_start)
                v.beta = divs(v.beta, surv);
            bl = v.beta;
        } else {
            bl = divs(v.beta, v.depth >= A.rr_start ? surv : 1.0f);
        }
    }
    if (MODE == E8G_MODE_REF_LT1) { // transport_direct_illum with one light sample (pathtracer.cpp:152-242)
        float pmf;
        int light = sample_light(S, rng, pmf);
        Surf ls = mesh_sample(S, __ldg(&S.light_mesh[light]), rng, false);
        ls.area_dens *= pmf;
        float3 l = sub(v.p, ls.p);
        float3 illum = light_eval(S, light, l, ls.n, v.n);
        float3 occ = mul(bl, divs(divs(f3(0, 0, 0), ls.area_dens), 1.0f)); // zero, or NaN
        if (!vequals0(illum)) {
            float dist = norm(l);
            q.sd = divs(neg(l), dist);
            q.st = dist - 1e-3f;
            q.vis = mul(bl, divs(divs(mul(illum, bsdf_eval(S, m, v.n, v.o, q.sd)), ls.area_dens), 1.0f));
            q.occ_nan = (occ.x == 0.0f ? 0u : 1u) | (occ.y == 0.0f ? 0u : 2u) | (occ.z == 0.0f ? 0u : 4u);
            q.shadow = true;
        } else {
            q.add = occ;
        }
    } else if (MODE == E8G_MODE_MIS) {
        float pmf;
        int light = sample_light(S, rng, pmf);
        Surf ls = mesh_sample(S, __ldg(&S.light_mesh[light]), rng, true);
        float3 l = sub(v.p, ls.p);
        float r2 = dot(l, l);
        float dist = sqrtf(r2);
        float3 ln = divs(l, dist);
        float cos_l = dot(ls.n, ln);
        float3 wi = neg(ln);
        float cos_x = dot(v.n, wi);
        if (cos_l > 0.0f && cos_x > 0.0f) {
            float3 f = bsdf_eval(S, m, v.n, v.o, wi);
            if (!vequals0(f)) {
                float p_l = pmf * ls.area_dens * r2 / cos_l;
                float p_b = bsdf_pdf(S, m, v.n, v.o, wi);
                float w = power_heuristic(p_l, p_b);
                q.vis = scale(mul(mul(v.beta, f), light_rad(S, light)), cos_x * w / p_l);
                q.sd = wi;
                q.st = dist - 1e-3f;
                q.shadow = true;
            }
        }
    } else if (MODE == E8G_MODE_REF_UNI) { // emission at every vertex (pathtracer.cpp:543-547)
        int32_t light = __ldg(&S.mesh_light[v.mesh]);
        if (light >= 0)
            q.add = mul(bl, light_radiance(S, light, v.o, v.n));
    }
    if (MODE == E8G_MODE_MIS) {
        q.i = bsdf_sample_mis(S, m, rng, q.pdf, v.n, v.o);
        if (q.pdf > 0.0f) {
            float cw = dot(v.n, q.i);
            if (cw > 0.0f) {
                float3 f = bsdf_eval(S, m, v.n, v.o, q.i);
                v.beta = mul(v.beta, scale(f, cw / q.pdf));
                q.extend = true;
            }
        }
    } else {
        q.i = bsdf_sample_ref(S, m, rng, q.pdf, v.n, v.o);
        if (q.pdf != 0.0f) {
            float3 f = bsdf_eval(S, m, v.n, v.o, q.i);
            v.beta = divs(scale(mul(bl, f), dot(v.n, q.i)), q.pdf);
            q.extend = true;
        }
    }
}

// A block's ray queue and slot states (shared memory): extension rays from the front, shadow rays
// from the back.
struct PoolQueue {
    uint16_t slot[2 * kPoolSlots];
    uint8_t ext_st[kPoolSlots], sh_st[kPoolSlots];
    uint32_t n_ext, n_sh, head;
    uint32_t over; // no path is left
};

// Appends a warp's rays of slot s.
__device__ __forceinline__ void pool_push(PoolQueue &Q, uint32_t s, bool extend, bool shadow) {
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
    const uint32_t me = __ballot_sync(~0u, extend), ms = __ballot_sync(~0u, shadow);
    uint32_t be = 0, bs = 0;
    if (lane == 0 && me)
        be = atomicAdd(&Q.n_ext, static_cast<uint32_t>(__popc(me)));
    if (lane == 0 && ms)
        bs = atomicAdd(&Q.n_sh, static_cast<uint32_t>(__popc(ms)));
    be = __shfl_sync(~0u, be, 0);
    bs = __shfl_sync(~0u, bs, 0);
    if (extend)
        Q.slot[be + __popc(me & below)] = static_cast<uint16_t>(s);
    if (shadow)
        Q.slot[2 * kPoolSlots - 1 - (bs + __popc(ms & below))] = static_cast<uint16_t>(s);
}

// A lane's ray: kept over a shading phase when it is still on its way.
constexpr uint32_t kPoolNone = 0xFFFFFFFFu;
struct PoolLane {
    uint32_t cur; // its slot, or kPoolNone
    bool any;
    SahWalk T;
    WideTrav TW;
    SahOverflow ov;
};

// Traces the block's queue: ne extension rays, then shadow rays, n in all. A warp leaves when the
// queue is empty and at most `keep` of its rays are on their way, after 16 steps at least.
template <int LAYOUT>
__device__ __forceinline__ void pool_trace(DevScene const &S, PoolLane &L, float4 *P, uint32_t slots, PoolQueue &Q,
                                           uint32_t ne, uint32_t n, uint32_t *stk, uint32_t keep) {
    const uint32_t lane = lane_id();
    const WideView WV{S.wnodes, S.tri, S.nnodes, S.ntris, S.check};
    // the ray's state in locals for the loop (as members of L they stay in local memory)
    uint32_t cur = L.cur;
    bool any = L.any;
    SahWalk T = L.T;
    WideTrav TW = L.TW;
    bool drained = n == 0;
    for (uint32_t steps = 0;; steps++) {
        uint32_t busy = __ballot_sync(~0u, cur != kPoolNone);
        uint32_t idle = drained ? 0u : ~busy;
        if (idle && (static_cast<uint32_t>(__popc(idle)) >= kPoolRefill || busy == 0)) {
            const uint32_t k = static_cast<uint32_t>(__popc(idle));
            uint32_t b = 0;
            if (lane == 0)
                b = atomicAdd(&Q.head, k);
            b = __shfl_sync(~0u, b, 0);
            drained = b + k >= n;
            const uint32_t idx = b + __popc(idle & ((1u << lane) - 1u));
            if (cur == kPoolNone && idx < n) {
                any = idx >= ne;
                cur = Q.slot[any ? 2 * kPoolSlots - 1 - (idx - ne) : idx];
                float4 o = P[kPoolPos * slots + cur];
                float4 d = P[(any ? kPoolShDir : kPoolDir) * slots + cur];
                float tmax = any ? d.w : 1000.0f;
                if (LAYOUT == 2)
                    wide_begin(TW, xyz(o), xyz(d), 1e-4f, tmax, any);
                else
                    sah_begin(S, T, xyz(o), xyz(d), 1e-4f, tmax);
            }
            busy = __ballot_sync(~0u, cur != kPoolNone);
        }
        if (drained && (busy == 0 || (static_cast<uint32_t>(__popc(busy)) <= keep && steps >= 16)))
            break;
        bool done = false;
        if (LAYOUT == 2) {
            if (cur != kPoolNone)
                done = wide_step<true>(WV, TW, stk, kBlock, nullptr, nullptr);
        } else {
            if (cur != kPoolNone && !T.leaf())
                done = sah_interior(S, T, stk, L.ov);
            const bool leaf = cur != kPoolNone && !done && T.leaf();
            const uint32_t lf = __ballot_sync(~0u, leaf);
            if (lf && (static_cast<uint32_t>(__popc(lf)) >= kLeafMin || lf == busy)) {
                if (leaf)
                    done = sah_leaf(S, T, any, stk, L.ov);
            }
        }
        if (done) {
            const Hit h = LAYOUT == 2 ? TW.h : T.h;
            if (!any) {
                P[kPoolHit * slots + cur] = make_float4(h.t, __uint_as_float(h.tri), h.b1, h.b2);
                Q.ext_st[cur] = kRayHit;
            } else {
                Q.sh_st[cur] = h.tri == 0xFFFFFFFFu ? kRayHit : kRayNone;
            }
            cur = kPoolNone;
        }
    }
    L.cur = cur;
    L.any = any;
    if (LAYOUT == 2)
        L.TW = TW;
    else
        L.T = T;
}

// Finishes a slot's extension ray: its vertex and the emission there with the MIS weight (add).
// False when the path ends (miss or back face).
template <int MODE>
__device__ __forceinline__ bool pool_complete(DevScene const &S, float4 hv, float4 dd, float4 bp, PoolVertex &v,
                                              float3 &add) {
    Hit h;
    h.t = hv.x;
    h.tri = __float_as_uint(hv.y);
    h.b1 = hv.z;
    h.b2 = hv.w;
    Vert nv = make_vert(S, h);
    v.o = neg(xyz(dd));
    if (dot(nv.n, v.o) <= 0.0f)
        return false;
    v.beta = xyz(bp);
    if (MODE == E8G_MODE_MIS) {
        int32_t hl = __ldg(&S.mesh_light[nv.mesh]);
        if (hl >= 0) {
            float cos_l2 = dot(nv.n, v.o);
            float pl = __ldg(&S.light_pnorm[hl]) / S.total_power;
            float inv_area = 1.0f / __ldg(&S.mesh_area[__ldg(&S.light_mesh[hl])]);
            float p_l = pl * inv_area * (nv.t * nv.t) / cos_l2;
            float w = power_heuristic(bp.w, p_l);
            add = scale(mul(v.beta, light_rad(S, hl)), w);
        }
    }
    v.p = nv.p;
    v.n = nv.n;
    v.mesh = nv.mesh;
    v.depth = __float_as_uint(dd.w) + 1u;
    return true;
}

__device__ __forceinline__ bool pool_nonzero(float3 a) { return a.x != 0.0f || a.y != 0.0f || a.z != 0.0f; }

// A path's radiance (kPoolRad) to its pixel, or to its entry of the per-path output (which the host zeroed):
// once a path, so that a pixel's sum is rounded once a sample, and lt1's first-hit emission last, as the
// reference adds it (w: whether there is one). Against an atomic for every term, which rounded a pixel's sum two
// to six times a sample: 1080p, 16-spp frame of the 1.3M-triangle icosphere, pairs, MIS / lt1 / uni 16.9 / 14.1 /
// 8.0 -> 16.9 / 14.2 / 8.5 ms, eight-wide 17.0 / 14.2 / 7.8 -> 16.2 / 13.4 / 7.9.
template <int MODE>
__device__ __forceinline__ void pool_finish(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum,
                                            float *path_rgb, uint32_t pixel, uint32_t out, float4 rad) {
    float3 L = xyz(rad);
    if (MODE == E8G_MODE_REF_LT1 && rad.w != 0.0f) {
        const FirstHit f = fh[pixel];
        L = add(L, light_radiance(S, __float_as_int(f.n.w), neg(xyz(f.d)), xyz(f.n)));
    }
    if (pool_nonzero(L))
        emit(A, accum, path_rgb, out, L);
}

// Starts a path at its cached first hit. False when the camera ray has none.
__device__ __forceinline__ bool pool_start(FirstHit const &f, PoolVertex &v) {
    if (__float_as_int(f.p.w) < 0)
        return false;
    v.p = xyz(f.p);
    v.n = xyz(f.n);
    v.o = neg(xyz(f.d));
    v.mesh = __float_as_int(f.p.w);
    v.depth = 0;
    v.beta = f3(1.0f, 1.0f, 1.0f);
    return true;
}

// The next path index of every lane that wants one, one atomic per warp.
__device__ __forceinline__ uint64_t pool_next_path(unsigned long long *work, uint32_t mask) {
    const uint32_t lane = lane_id();
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (static_cast<int>(lane) == leader)
        base = atomicAdd(work, static_cast<unsigned long long>(__popc(mask)));
    base = __shfl_sync(~0u, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

template <class R, int LAYOUT, int MODE>
__global__ void __launch_bounds__(kBlock, kPoolBlocks)
    k_mega_pool(const __grid_constant__ DevScene S, const __grid_constant__ RenderArgs A,
                FirstHit const *__restrict__ fh, float4 *accum, float *path_rgb, unsigned long long *work, float4 *pool,
                uint32_t slots, uint32_t keep) {
    __shared__ uint32_t stk_all[kStackOf<LAYOUT> * kBlock];
    __shared__ PoolQueue Q;
    uint32_t *stk = stk_all + threadIdx.x;
    const uint64_t mix = splitmix64(A.seed);
    float4 *P = pool + static_cast<size_t>(blockIdx.x) * kPoolArrays * slots;
    for (uint32_t s = threadIdx.x; s < slots; s += kBlock)
        Q.ext_st[s] = Q.sh_st[s] = kRayNone;
    if (threadIdx.x == 0)
        Q.n_ext = Q.n_sh = Q.head = Q.over = 0;
    __syncthreads();
    PoolLane L;
    L.cur = kPoolNone;
    L.any = false;
    while (true) {
        // ---- shade every slot ----
        // The barriers keep the block's warps in the same part of a code that does not fit the
        // instruction cache of a partition: 18.6 -> 18.1 ms per 16-spp frame on the pairs, 19.7 -> 18.7 on
        // the wide tree.
        for (uint32_t s0 = 0; s0 < slots; s0 += kBlock) {
            __syncthreads();
            const uint32_t s = s0 + threadIdx.x;
            bool at_vertex = false;
            PoolVertex v;
            R rng;
            uint32_t pixel = 0, sample = 0, out = 0;
            const uint32_t es = Q.ext_st[s], sh = Q.sh_st[s];
            const bool open = es != kRayOut && sh != kRayOut;
            if (open && es != kRayNone) { // a path whose rays are back
                const float4 ids = P[kPoolIds * slots + s];
                float3 hit = f3(0, 0, 0); // emission at the vertex
                if (es == kRayHit) {
                    const float4 hv = P[kPoolHit * slots + s];
                    at_vertex = __float_as_uint(hv.y) != 0xFFFFFFFFu &&
                                pool_complete<MODE>(S, hv, P[kPoolDir * slots + s], P[kPoolBeta * slots + s], v, hit);
                    if (at_vertex)
                        rng = RngSlot<R>::load(A, __float_as_uint(ids.x), __float_as_uint(ids.y), __float_as_uint(ids.w));
                }
                const bool grew = sh == kRayHit || (MODE == E8G_MODE_MIS && pool_nonzero(hit));
                if (!at_vertex || grew) {
                    float4 rad = P[(sh == kRayHit ? kPoolShAdd : kPoolRad) * slots + s];
                    if (MODE == E8G_MODE_MIS) {
                        const float3 r = add(xyz(rad), hit);
                        rad = make_float4(r.x, r.y, r.z, 0.0f);
                    }
                    if (at_vertex)
                        P[kPoolRad * slots + s] = rad;
                    else
                        pool_finish<MODE>(S, A, fh, accum, path_rgb, __float_as_uint(ids.x), __float_as_uint(ids.z), rad);
                }
            }
            // a path for every free slot; paths without a first hit end at once
            bool want = open && !at_vertex && Q.over == 0;
            while (const uint32_t mask = __ballot_sync(~0u, want)) {
                const uint64_t idx = pool_next_path(work, mask);
                if (want) {
                    if (idx >= A.total_paths) {
                        want = false;
                        Q.over = 1;
                    } else if (path_coords(A, idx, pixel, sample, out)) {
                        FirstHit f = fh[pixel];
                        if (pool_start(f, v)) {
                            rng = RngSlot<R>::fresh(A, mix, pixel, sample);
                            int32_t light = __float_as_int(f.n.w);
                            const float3 rad =
                                MODE == E8G_MODE_MIS && light >= 0 ? light_radiance(S, light, v.o, v.n) : f3(0, 0, 0);
                            P[kPoolIds * slots + s] =
                                make_float4(__uint_as_float(pixel), __uint_as_float(sample), __uint_as_float(out), 0.0f);
                            P[kPoolRad * slots + s] = make_float4(rad.x, rad.y, rad.z, light >= 0 ? 1.0f : 0.0f);
                            at_vertex = true;
                            want = false;
                        }
                    }
                }
            }
            __syncthreads();
            bool shadow = false, extend = false;
            if (at_vertex) {
                PoolRays q;
                pool_shade<MODE>(S, A, v, rng, q);
                shadow = q.shadow;
                extend = q.extend;
                if (extend) {
                    P[kPoolBeta * slots + s] = make_float4(v.beta.x, v.beta.y, v.beta.z, q.pdf);
                    P[kPoolDir * slots + s] = make_float4(q.i.x, q.i.y, q.i.z, __uint_as_float(v.depth));
                }
                const bool plus = MODE != E8G_MODE_MIS && pool_nonzero(q.add), ends = !shadow && !extend;
                if (shadow || plus || ends) {
                    // read again: held over the shading it would be spilled
                    float4 rad = P[kPoolRad * slots + s];
                    if (plus) {
                        const float3 r = add(xyz(rad), q.add);
                        P[kPoolRad * slots + s] = rad = make_float4(r.x, r.y, r.z, rad.w);
                    }
                    if (shadow) {
                        const float3 r = add(xyz(rad), q.vis);
                        P[kPoolShAdd * slots + s] = make_float4(r.x, r.y, r.z, rad.w);
                        if (MODE == E8G_MODE_REF_LT1 && q.occ_nan) {
                            const float nan = __uint_as_float(0x7FFFFFFFu);
                            P[kPoolRad * slots + s] = make_float4(q.occ_nan & 1u ? nan : rad.x, q.occ_nan & 2u ? nan : rad.y,
                                                                  q.occ_nan & 4u ? nan : rad.z, rad.w);
                        }
                    }
                    if (ends) {
                        const float4 ids = P[kPoolIds * slots + s];
                        pool_finish<MODE>(S, A, fh, accum, path_rgb, __float_as_uint(ids.x), __float_as_uint(ids.z), rad);
                    }
                }
                if (shadow)
                    P[kPoolShDir * slots + s] = make_float4(q.sd.x, q.sd.y, q.sd.z, q.st);
                if (!ends) {
                    P[kPoolPos * slots + s] = make_float4(v.p.x, v.p.y, v.p.z, 0.0f);
                    if (extend)
                        reinterpret_cast<float *>(&P[kPoolIds * slots + s])[3] = __uint_as_float(RngSlot<R>::store(rng));
                }
            }
            if (open) {
                Q.ext_st[s] = extend ? kRayOut : shadow ? kRayEnd : kRayNone;
                Q.sh_st[s] = shadow ? kRayOut : kRayNone;
            }
            pool_push(Q, s, extend, shadow);
        }
        const int out_rays = __syncthreads_or(L.cur != kPoolNone);
        const uint32_t ne = Q.n_ext, n = ne + Q.n_sh;
        if (n == 0 && Q.over && !out_rays)
            break;
        pool_trace<LAYOUT>(S, L, P, slots, Q, ne, n, stk, keep);
        __syncthreads();
        if (threadIdx.x == 0)
            Q.n_ext = Q.n_sh = Q.head = 0;
        __syncthreads();
    }
}

} // namespace

// Slots per block: about sixteen paths each, since a pool that the render fills only a few times
// spends its time in the end, when slots run empty (2 M paths: 256 / 512 / 1024 slots 0.89 / 0.92 /
// 1.05 ms; 33 M: 19.9 / 19.4 / 18.8). At least 256, and 128 below 2^20 paths. With 128 / 256 slots, pairs,
// 541,000 paths of a one-sample frame: 0.81 / 0.86 ms (1.3M-triangle icosphere), 1.21 / 1.26 (50,000-triangle
// soup), backward 0.71 / 0.82 (327,690 triangles) and 1.24 / 1.24; 1.07M paths: 1.09 / 1.11 and 1.85 / 1.79;
// 2.07M: 1.77 / 1.70 and 3.01 / 2.81. The eight-wide tree alike.
inline uint32_t pool_slots(RenderArgs const &A, int num_sms) {
    const uint64_t per_block = A.total_paths / (static_cast<uint64_t>(num_sms) * kPoolBlocks);
    const uint64_t want = (per_block / 16 + kBlock - 1) / kBlock * kBlock;
    const uint64_t least = A.total_paths < (1u << 20) ? 128 : 256;
    return static_cast<uint32_t>(std::min<uint64_t>(std::max<uint64_t>(want, least), kPoolSlots));
}

// Rays a warp may leave the trace phase with: 0 / 8 / 16 / 24 take 1.99 / 1.70 / 1.74 / 1.79 ms in a one-sample
// 1080p frame of 1.3M triangles, 3.19 / 2.81 / 2.83 / 2.91 in one of a 50,000-triangle soup and 1.18 / 1.15 / 1.20 / 1.25
// with 20,000 triangles. In a tiny tree rays are short and of one length, and leaving slots out of the next
// shading costs more than their wait (Cornell: 0.91 ms with 0, 0.96 with 8).
inline uint32_t pool_keep(DevScene const &S) { return S.nnodes >= 1024 ? 8u : 0u; }

template <int LAYOUT>
inline void launch_pool(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                        unsigned long long *work, float4 *pool, int num_sms, cudaStream_t st) {
    const int grid = num_sms * kPoolBlocks;
    const uint32_t slots = pool_slots(A, num_sms);
    const uint32_t keep = pool_keep(S);
    auto go = [&](auto *kern) { kern<<<grid, kBlock, 0, st>>>(S, A, fh, accum, path_rgb, work, pool, slots, keep); };
    if (A.mode == E8G_MODE_MIS)
        go(k_mega_pool<RngPhilox, LAYOUT, E8G_MODE_MIS>);
    else if (A.mode == E8G_MODE_REF_LT1)
        go(k_mega_pool<RngMinstd, LAYOUT, E8G_MODE_REF_LT1>);
    else
        go(k_mega_pool<RngMinstd, LAYOUT, E8G_MODE_REF_UNI>);
}

} // namespace e8g
