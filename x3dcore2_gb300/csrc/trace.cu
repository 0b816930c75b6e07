// Primary-hit, ray-batch traversal and resolve kernels.
#include "launch.h"

#include <algorithm>

namespace e8g {

// compute_first_hit (pathtracer.cpp:456-472): camera ray, closest hit, back-facing hits become
// misses, emitter lookup.
template <int LAYOUT>
__global__ void __launch_bounds__(kBlock) k_first_hits(const __grid_constant__ DevScene S, uint32_t w, uint32_t h,
                                                       FirstHit *out) {
    __shared__ uint32_t stk[kStackOf<LAYOUT> * kBlock];
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h)
        return;
    float3 o, d;
    camera_ray(S.cam, i % w, i / w, w, h, o, d);
    Hit hit = trace_l<LAYOUT, false>(S, o, d, 1e-4f, 1000.0f, false, stk + threadIdx.x, nullptr);
    FirstHit f;
    f.d = make_float4(d.x, d.y, d.z, 0.0f);
    int32_t mesh = -1, light = -1;
    float3 p = f3(0, 0, 0), n = f3(0, 0, 0);
    if (hit.tri != 0xFFFFFFFFu) {
        Vert v = make_vert(S, hit);
        if (dot(v.n, neg(d)) > 0) {
            mesh = v.mesh;
            p = v.p;
            n = v.n;
            light = __ldg(&S.mesh_light[mesh]);
        }
    }
    f.p = make_float4(p.x, p.y, p.z, __int_as_float(mesh));
    f.n = make_float4(n.x, n.y, n.z, __int_as_float(light));
    out[i] = f;
}

// compute_first_hit for explicit rays: ray i's first hit into out[i].
template <int LAYOUT>
__global__ void __launch_bounds__(kBlock) k_first_hits_rays(const __grid_constant__ DevScene S, float const *rays6,
                                                             uint32_t n, FirstHit *out) {
    __shared__ uint32_t stk[kStackOf<LAYOUT> * kBlock];
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float3 o = f3(rays6[6 * i], rays6[6 * i + 1], rays6[6 * i + 2]);
    float3 d = f3(rays6[6 * i + 3], rays6[6 * i + 4], rays6[6 * i + 5]);
    Hit hit = trace_l<LAYOUT, false>(S, o, d, 1e-4f, 1000.0f, false, stk + threadIdx.x, nullptr);
    FirstHit f;
    f.d = make_float4(d.x, d.y, d.z, 0.0f);
    int32_t mesh = -1, light = -1;
    float3 p = f3(0, 0, 0), nn = f3(0, 0, 0);
    if (hit.tri != 0xFFFFFFFFu) {
        Vert v = make_vert(S, hit);
        if (dot(v.n, neg(d)) > 0) {
            mesh = v.mesh;
            p = v.p;
            nn = v.n;
            light = __ldg(&S.mesh_light[mesh]);
        }
    }
    f.p = make_float4(p.x, p.y, p.z, __int_as_float(mesh));
    f.n = make_float4(nn.x, nn.y, nn.z, __int_as_float(light));
    out[i] = f;
}

// Identity pixel list and a constant sample list for explicit rays.
__global__ void k_ray_lists(uint32_t n, uint32_t sample, uint32_t *pixel, uint32_t *samples) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        pixel[i] = i;
        samples[i] = sample;
    }
}

__global__ void k_camera_rays(DevScene S, uint32_t w, uint32_t h, float *rays6) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h)
        return;
    float3 o, d;
    camera_ray(S.cam, i % w, i / w, w, h, o, d);
    float *r = rays6 + 6 * static_cast<size_t>(i);
    r[0] = o.x;
    r[1] = o.y;
    r[2] = o.z;
    r[3] = d.x;
    r[4] = d.y;
    r[5] = d.z;
}

__device__ __forceinline__ void store_hit(DevScene const &S, Hit const &h, HitOut const &out, uint32_t i) {
    float t = 0.0f, b1 = 0.0f, b2 = 0.0f;
    int mesh = -1, tri = -1;
    if (h.tri != 0xFFFFFFFFu) {
        uint4 ti = __ldg(&S.tidx[h.tri]);
        t = h.t;
        mesh = static_cast<int>(ti.w);
        tri = static_cast<int>(h.tri - __ldg(&S.mesh_toff[ti.w]));
        b1 = h.b1;
        b2 = h.b2;
    }
    const size_t k = static_cast<size_t>(i) * out.stride;
    out.t[k] = t;
    out.mesh[k] = __int_as_float(mesh);
    out.tri[k] = __int_as_float(tri);
    float *b = out.b + static_cast<size_t>(i) * out.b_stride;
    b[0] = b1;
    b[1] = b2;
}

// Ray batches on the SAH pairs and the eight-wide tree. Each warp owns `chunk` consecutive rays and
// gives an idle lane the next of them once kRayRefill lanes are idle: a batch's rays have no order,
// and with one ray per lane the warp waits for its longest (3.3 of 32 lanes active on 300,000 random
// rays against the 1.3M-triangle icosphere). The chunks are fixed, so calls on several streams
// share nothing. ANY: any-hit on [tmin[i], tmax[i]] into occ, else the closest hit into hits.
constexpr uint32_t kRayRefill = 8;
constexpr int kRayBlocks = 8; // blocks of 128 threads per SM (64 registers), as the wavefront's trace kernel

template <int LAYOUT, bool ANY>
__global__ void __launch_bounds__(kBlock, kRayBlocks)
    k_trace_rays(const __grid_constant__ DevScene S, float const *__restrict__ rays6, float const *__restrict__ tmin,
                 float const *__restrict__ tmax, uint32_t n, uint32_t chunk, HitOut hits, uint8_t *occ) {
    __shared__ uint32_t stk_all[kStackOf<LAYOUT> * kBlock];
    uint32_t *stk = stk_all + threadIdx.x;
    const uint32_t lane = lane_id();
    const uint64_t first = static_cast<uint64_t>(blockIdx.x * (kBlock / 32) + threadIdx.x / 32) * chunk;
    if (first >= n)
        return;
    uint32_t next = static_cast<uint32_t>(first); // the warp's next ray, up to `end` (the same in every lane)
    const uint32_t end = static_cast<uint32_t>(first + chunk < n ? first + chunk : n);
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t cur = kNone;
    const WideView WV{S.wnodes, S.tri, S.nnodes, S.ntris, S.check};
    SahWalk T;
    SahOverflow ov;
    WideTrav TW;
    while (true) {
        uint32_t busy = __ballot_sync(~0u, cur != kNone);
        const uint32_t idle = ~busy;
        if (next < end && (busy == 0 || static_cast<uint32_t>(__popc(idle)) >= kRayRefill)) {
            const uint32_t r = __popc(idle & ((1u << lane) - 1u));
            if (cur == kNone && r < end - next) {
                cur = next + r;
                float const *q = rays6 + 6 * static_cast<size_t>(cur);
                float3 o = f3(q[0], q[1], q[2]), d = f3(q[3], q[4], q[5]);
                float t0 = ANY ? tmin[cur] : 1e-4f, t1 = ANY ? tmax[cur] : 1000.0f;
                if (LAYOUT == 2)
                    wide_begin(TW, o, d, t0, t1, ANY);
                else
                    sah_begin(S, T, o, d, t0, t1);
            }
            const uint32_t k = static_cast<uint32_t>(__popc(idle));
            next = k < end - next ? next + k : end;
            busy = __ballot_sync(~0u, cur != kNone);
        }
        if (busy == 0)
            break;
        bool done = false;
        if (S.nnodes == 0) {
            done = cur != kNone;
        } else if (LAYOUT == 2) {
            if (cur != kNone)
                done = wide_step<true>(WV, TW, stk, kBlock, nullptr, nullptr);
        } else {
            if (cur != kNone && !T.leaf())
                done = sah_interior(S, T, stk, ov);
            const bool leaf = cur != kNone && !done && T.leaf();
            const uint32_t lf = __ballot_sync(~0u, leaf);
            if (lf && 4 * __popc(lf) >= __popc(busy)) {
                if (leaf)
                    done = sah_leaf(S, T, ANY, stk, ov);
            }
        }
        if (done) {
            const Hit h = LAYOUT == 2 ? TW.h : T.h;
            if (ANY)
                occ[cur] = h.tri != 0xFFFFFFFFu ? 1 : 0;
            else
                store_hit(S, h, hits, cur);
            cur = kNone;
        }
    }
}

// Small batches: a warp per ray. One lane's walk is a chain of dependent loads (a ray against a soup of
// 1,000 triangles took 40 us with the GPU idle around it); here the warp takes up to 32 pending nodes
// of its ray at once and tests leaves four lanes each, so the chain is about as long as the tree is
// deep. The visiting order differs from the one-lane walk's, the hit does not: the nearest triangle is
// the nearest in any order, and a ray that meets two triangles at exactly the same distance (a shared
// edge), or whose pending nodes outgrow the lists, is walked again by one lane. Bound by the latency of
// its rounds (a node or leaf fetch from L2 each), then, from about a ray per resident warp on, by issue
// slots. A closest-hit and an any-hit query together: 1,500 rays against that soup 149 -> 77 us on the
// pairs, 115 -> 72 on the eight-wide tree; against 100,000 triangles 276 -> 99 and 211 -> 101.
constexpr uint32_t kWarpList = 256;            // pending nodes, and pending leaves, of a ray
constexpr uint32_t kWarpRayTris = 1u << 27;    // eight-wide leaves are listed as count << 27 | first record
// Rays per resident warp up to which a warp takes one ray at a time. Both forms at 10,000 / 14,000 / 19,000
// rays (2 to 4 per warp): pairs, 1,000-triangle soup 142 / 181 / 223 us against 220 / 225 / 246;
// eight-wide, same soup 157 / 204 / 255 against 200 / 229 / 255.
constexpr uint32_t kWarpRays = 4;

template <int LAYOUT, bool ANY>
__global__ void __launch_bounds__(kBlock, kRayBlocks)
    k_trace_warp(const __grid_constant__ DevScene S, float const *__restrict__ rays6, float const *__restrict__ tmin,
                 float const *__restrict__ tmax, uint32_t n, HitOut hits, uint8_t *occ) {
    __shared__ uint32_t stk_all[kStackOf<LAYOUT> * kBlock];
    __shared__ uint32_t node_all[kBlock / 32][kWarpList], leaf_all[kBlock / 32][kWarpList];
    uint32_t *nodes = node_all[threadIdx.x / 32], *leaves = leaf_all[threadIdx.x / 32];
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u, group = lane / 4, sub = lane & 3u;
    constexpr uint32_t kPush = LAYOUT == 2 ? 8 : 2; // children of a node
    for (uint32_t i = blockIdx.x * (kBlock / 32) + threadIdx.x / 32; i < n; i += gridDim.x * (kBlock / 32)) {
        float const *q = rays6 + 6 * static_cast<size_t>(i);
        const float3 o = f3(q[0], q[1], q[2]), d = f3(q[3], q[4], q[5]);
        const float t0 = ANY ? tmin[i] : 1e-4f, t1 = ANY ? tmax[i] : 1000.0f;
        SahWalk T;
        WideTrav TW;
        if (LAYOUT == 2)
            wide_begin(TW, o, d, t0, t1, ANY);
        else
            sah_begin(S, T, o, d, t0, t1);
        float cull = t1;
        Hit h; // this lane's nearest
        h.t = INFINITY;
        h.tri = 0xFFFFFFFFu;
        h.b1 = h.b2 = 0.0f;
        bool tie = false, found = false, again = false;
        uint32_t nn = 0, nl = 0; // list lengths, the same in every lane
        if (S.nnodes) {
            if (LAYOUT == 0 && T.leaf()) {
                if (lane == 0)
                    leaves[0] = 0;
                nl = 1;
            } else {
                if (lane == 0)
                    nodes[0] = 0;
                nn = 1;
            }
        }
        __syncwarp();
        while (nn || nl) {
            uint32_t k = nn < 32u ? nn : 32u;
            const uint32_t room_n = (kWarpList - nn) / (kPush - 1), room_l = (kWarpList - nl) / kPush;
            k = k < room_n ? k : room_n;
            k = k < room_l ? k : room_l;
            if (nn && k == 0 && nl == 0) {
                again = true;
                break;
            }
            if (k) {
                const bool on = lane < k;
                const uint32_t item = on ? nodes[nn - 1 - lane] : 0;
                nn -= k;
                __syncwarp();
                if (LAYOUT == 2) {
                    uint32_t hit = 0, imask = 0, base = 0, tri_base = 0, meta_lo = 0, meta_hi = 0, counts = 0;
                    if (on && E8G_CHK(S.check, item < S.nnodes, kChkNode, item)) {
                        uint4 const *np = S.wnodes + 6 * static_cast<size_t>(item);
                        uint4 n0, n1, n2, n3, n4, n5;
                        hd_ld2<true>(np, n0, n1);
                        hd_ld2<true>(np + 2, n2, n3);
                        hd_ld2<true>(np + 4, n4, n5);
                        TW.cull = cull;
                        imask = n0.w >> 24;
                        hit = wide_child_hits(TW, n0, n2, n3, n4) & (imask | n5.y);
                        base = n1.x, tri_base = n1.y, meta_lo = n1.z, meta_hi = n1.w, counts = n5.x;
                    }
                    for (uint32_t j = 8; j-- > 0;) { // the nearest octant on top
                        const uint32_t s = j ^ TW.oct;
                        const bool is = hit >> s & 1u, inner = is && (imask >> s & 1u);
                        const uint32_t mn = __ballot_sync(~0u, inner), ml = __ballot_sync(~0u, is && !inner);
                        if (inner)
                            nodes[nn + __popc(mn & below)] = base + __popc(imask & ((1u << s) - 1u));
                        else if (is)
                            leaves[nl + __popc(ml & below)] =
                                ((counts >> (4u * s)) & 0xFu) << 27 |
                                (tri_base + ((s < 4 ? meta_lo : meta_hi) >> (8u * (s & 3u)) & 0xFFu));
                        nn += __popc(mn);
                        nl += __popc(ml);
                    }
                } else {
                    bool hit0 = false, hit1 = false;
                    uint32_t w0 = 0, w1 = 0;
                    if (on && E8G_CHK(S.check, 2 * static_cast<uint64_t>(item) + 2 < S.nnodes, kChkNode, item)) {
                        float4 l0, h0, l1, h1;
                        float4 const *pair = S.nlo.p + 4 * static_cast<size_t>(item) + 2;
                        ldg_node(pair, l0, h0);
                        ldg_node(pair + 2, l1, h1);
                        float tn0, tn1;
                        hit0 = sah_slab(l0, h0, T.inv, T.oi, t0, cull, tn0);
                        hit1 = sah_slab(l1, h1, T.inv, T.oi, t0, cull, tn1);
                        w0 = sah_word(l0.w, h0.w), w1 = sah_word(l1.w, h1.w);
                        if (hit0 && hit1 && tn0 < tn1) { // the nearer one on top
                            const uint32_t w = w0;
                            w0 = w1;
                            w1 = w;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const bool is = c ? hit1 : hit0;
                        const uint32_t w = c ? w1 : w0;
                        const bool leaf = is && (w & kSahLeaf);
                        const uint32_t mn = __ballot_sync(~0u, is && !leaf), ml = __ballot_sync(~0u, leaf);
                        if (leaf)
                            leaves[nl + __popc(ml & below)] = w & ~kSahLeaf;
                        else if (is)
                            nodes[nn + __popc(mn & below)] = w;
                        nn += __popc(mn);
                        nl += __popc(ml);
                    }
                }
                __syncwarp();
            }
            if (nl && (nl >= 8 || nn == 0 || k == 0)) {
                const uint32_t take = nl < 8u ? nl : 8u;
                bool open = group < take;
                const uint32_t item = open ? leaves[nl - 1 - group] : 0;
                nl -= take;
                __syncwarp();
                uint32_t rec = (LAYOUT == 2 ? item & (kWarpRayTris - 1) : item) + sub;
                const uint32_t end = LAYOUT == 2 ? (item & (kWarpRayTris - 1)) + (item >> 27) : S.ntris;
                while (__any_sync(~0u, open)) {
                    bool test = open && rec < end && E8G_CHK(S.check, rec < S.ntris, kChkTri, rec);
                    float4 a, b, c;
                    if (test) {
                        float4 const *r = S.tri + 3 * static_cast<size_t>(rec);
                        a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2);
                    }
                    if (LAYOUT == 2) {
                        open = open && rec - sub + 4 < end;
                    } else { // a leaf of child pairs ends with its marked record
                        const uint32_t last = __ballot_sync(~0u, test && b.w != 0.0f) >> (4 * group) & 0xFu;
                        test = test && (last & ((1u << sub) - 1u)) == 0;
                        open = open && last == 0 && rec - sub + 4 < end;
                    }
                    rec += 4;
                    float t, b1, b2;
                    if (test && hd_tri_test(o, d, a, b, c, t0, cull, t, b1, b2) && t < INFINITY) {
                        const uint32_t id = __float_as_uint(a.w);
                        if (ANY) {
                            found = true;
                        } else if (t < h.t) {
                            h.t = t;
                            h.tri = id;
                            h.b1 = b1;
                            h.b2 = b2;
                            tie = false;
                        } else if (t == h.t) {
                            tie = true;
                        }
                    }
                }
                if (ANY) {
                    if (__any_sync(~0u, found))
                        break;
                } else { // distances are positive: their bits are in order
                    cull = fminf(cull, __uint_as_float(__reduce_min_sync(~0u, __float_as_uint(h.t))));
                }
            }
        }
        if (ANY) {
            found = __any_sync(~0u, found);
            if (lane == 0 && again)
                found = trace_l<LAYOUT, false>(S, o, d, t0, t1, true, stk_all + threadIdx.x, nullptr).tri != 0xFFFFFFFFu;
            if (lane == 0)
                occ[i] = found ? 1 : 0;
        } else {
            // every lane takes part in the warp operations, whatever it found
            const uint32_t nearest = __reduce_min_sync(~0u, __float_as_uint(h.t));
            const bool mine = h.tri != 0xFFFFFFFFu && __float_as_uint(h.t) == nearest;
            const uint32_t win = __ballot_sync(~0u, mine), ties = __ballot_sync(~0u, mine && tie);
            again = again || __popc(win) > 1 || ties;
            if (again && lane == 0)
                h = trace_l<LAYOUT, false>(S, o, d, t0, t1, false, stk_all + threadIdx.x, nullptr);
            if (again || win == 0 ? lane == 0 : mine)
                store_hit(S, h, hits, i);
        }
        __syncwarp();
    }
}

// One ray per thread: the reference's tree and the linear layout.
template <bool ANY>
__global__ void __launch_bounds__(kBlock) k_trace_plain(DevScene S, float const *rays6, float const *tmin,
                                                        float const *tmax, uint32_t n, HitOut hits, uint8_t *occ) {
    __shared__ uint32_t stk[kStackWords * kBlock];
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float const *r = rays6 + 6 * static_cast<size_t>(i);
    float3 o = f3(r[0], r[1], r[2]), d = f3(r[3], r[4], r[5]);
    if (ANY)
        occ[i] = trace_any<false>(S, o, d, tmin[i], tmax[i], stk + threadIdx.x, nullptr) ? 1 : 0;
    else
        store_hit(S, trace_closest<false>(S, o, d, stk + threadIdx.x, nullptr), hits, i);
}

__global__ void k_resolve(float4 const *accum, uint32_t npix, float inv_spp, float *rgba) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix)
        return;
    float4 a = accum[i];
    reinterpret_cast<float4 *>(rgba)[i] = make_float4(a.x * inv_spp, a.y * inv_spp, a.z * inv_spp, 1.0f);
}

// pt_image_renderer's firefly clamp (renderer.cpp:46-83) over K per-sample images est
// (sample-major, W*H rgb each), accumulated per pixel in sample order like the reference's task
// estimate: an interior pixel whose squared norm exceeds each of its 8 neighbours' by more than
// 1.5 (renderer.h:118) has every channel capped at the neighbours' mean squared norm plus 1.5.
__device__ __forceinline__ float sqnorm(float const *v) {
    float r = 0.0f;
    r += v[0] * v[0];
    r += v[1] * v[1];
    r += v[2] * v[2];
    return r;
}

__global__ void k_firefly(float const *__restrict__ est, uint32_t K, uint32_t w, uint32_t h, float4 *accum) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t npix = w * h;
    if (i >= npix)
        return;
    uint32_t x = i % w, y = i / w;
    bool inner = x > 0 && x < w - 1 && y > 0 && y < h - 1;
    const float diff = 1.5f;
    float4 a = accum[i];
    for (uint32_t k = 0; k < K; k++) {
        float const *e = est + 3 * (static_cast<size_t>(k) * npix + i);
        float v0 = e[0], v1 = e[1], v2 = e[2];
        if (inner) {
            size_t row = 3 * static_cast<size_t>(w);
            float r00 = sqnorm(e - row - 3), r10 = sqnorm(e - row), r20 = sqnorm(e - row + 3);
            float r01 = sqnorm(e - 3), r11 = sqnorm(e), r21 = sqnorm(e + 3);
            float r02 = sqnorm(e + row - 3), r12 = sqnorm(e + row), r22 = sqnorm(e + row + 3);
            bool ff = (r11 - r00) > diff && (r11 - r10) > diff && (r11 - r20) > diff && (r11 - r01) > diff &&
                      (r11 - r21) > diff && (r11 - r02) > diff && (r11 - r12) > diff && (r11 - r22) > diff;
            if (ff) {
                float cap = 1.0f / 8.0f * (r00 + r10 + r20 + r01 + r21 + r02 + r12 + r22) + diff;
                v0 = cap < v0 ? cap : v0;
                v1 = cap < v1 ? cap : v1;
                v2 = cap < v2 ? cap : v2;
            }
        }
        a.x += v0;
        a.y += v1;
        a.z += v2;
    }
    accum[i] = a;
}

static inline int blocks(uint32_t n, int b) { return static_cast<int>((n + b - 1) / b); }

void launch_first_hits(DevScene const &S, uint32_t w, uint32_t h, FirstHit *out, cudaStream_t st) {
    auto *kern = S.layout == 0 ? k_first_hits<0> : S.layout == 1 ? k_first_hits<1> : S.layout == 2 ? k_first_hits<2> : k_first_hits<3>;
    kern<<<blocks(w * h, kBlock), kBlock, 0, st>>>(S, w, h, out);
}
void launch_first_hits_rays(DevScene const &S, float const *rays6, uint32_t n, FirstHit *out, uint32_t sample,
                            uint32_t *pixel, uint32_t *samples, cudaStream_t st) {
    if (!n)
        return;
    auto *kern = S.layout == 0   ? k_first_hits_rays<0>
                 : S.layout == 1 ? k_first_hits_rays<1>
                 : S.layout == 2 ? k_first_hits_rays<2>
                                 : k_first_hits_rays<3>;
    kern<<<blocks(n, kBlock), kBlock, 0, st>>>(S, rays6, n, out);
    k_ray_lists<<<blocks(n, 256), 256, 0, st>>>(n, sample, pixel, samples);
}
void launch_camera_rays(DevScene const &S, uint32_t w, uint32_t h, float *rays6, cudaStream_t st) {
    k_camera_rays<<<blocks(w * h, 256), 256, 0, st>>>(S, w, h, rays6);
}
// A warp per ray for batches of at most kWarpRays rays per resident warp, else an equal share of the batch
// for every resident warp (a closest-hit and an any-hit query of 1,000,003 rays against the
// 327,690-triangle icosphere 0.83 ms).
template <bool ANY>
static void trace_rays(DevScene const &S, float const *rays6, float const *tmin, float const *tmax, uint32_t n,
                       HitOut const &hits, uint8_t *occ, int num_sms, cudaStream_t st) {
    if (!n)
        return;
    if (S.layout != 0 && S.layout != 2) {
        k_trace_plain<ANY><<<blocks(n, kBlock), kBlock, 0, st>>>(S, rays6, tmin, tmax, n, hits, occ);
        return;
    }
    const uint32_t warps = static_cast<uint32_t>(num_sms) * kRayBlocks * (kBlock / 32);
    if (n <= kWarpRays * warps && (S.layout == 0 || S.ntris < kWarpRayTris)) {
        const uint32_t g = (std::min(n, warps) - 1) / (kBlock / 32) + 1;
        if (S.layout == 2)
            k_trace_warp<2, ANY><<<g, kBlock, 0, st>>>(S, rays6, tmin, tmax, n, hits, occ);
        else
            k_trace_warp<0, ANY><<<g, kBlock, 0, st>>>(S, rays6, tmin, tmax, n, hits, occ);
        return;
    }
    const uint32_t chunk = (n - 1) / warps + 1;
    const uint32_t g = ((n - 1) / chunk) / (kBlock / 32) + 1;
    if (S.layout == 2)
        k_trace_rays<2, ANY><<<g, kBlock, 0, st>>>(S, rays6, tmin, tmax, n, chunk, hits, occ);
    else
        k_trace_rays<0, ANY><<<g, kBlock, 0, st>>>(S, rays6, tmin, tmax, n, chunk, hits, occ);
}
void launch_trace_closest(DevScene const &S, float const *rays6, uint32_t n, HitOut const &hits, int num_sms,
                          cudaStream_t st) {
    trace_rays<false>(S, rays6, nullptr, nullptr, n, hits, nullptr, num_sms, st);
}
void launch_trace_any(DevScene const &S, float const *rays6, float const *tmin, float const *tmax, uint32_t n,
                      uint8_t *occ, int num_sms, cudaStream_t st) {
    trace_rays<true>(S, rays6, tmin, tmax, n, HitOut{}, occ, num_sms, st);
}
void launch_resolve(float4 const *accum, uint32_t npix, float inv_spp, float *rgba, cudaStream_t st) {
    k_resolve<<<blocks(npix, 256), 256, 0, st>>>(accum, npix, inv_spp, rgba);
}
void launch_firefly(float const *est, uint32_t K, uint32_t w, uint32_t h, float4 *accum, cudaStream_t st) {
    k_firefly<<<blocks(w * h, 256), 256, 0, st>>>(est, K, w, h, accum);
}

} // namespace e8g

namespace e8g {

// Batched first hits: the pixel index runs over every scene's pixels.
__global__ void __launch_bounds__(kBlock) k_first_hits_batch(BatchDev B, uint64_t total_pix, FirstHit *out) {
    __shared__ uint32_t stk[kStackWords * kBlock];
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= total_pix)
        return;
    uint32_t lo = 0, hi = B.n;
    while (hi - lo > 1) {
        uint32_t mi = (lo + hi) >> 1;
        if (B.pix_prefix[mi] <= i)
            lo = mi;
        else
            hi = mi;
    }
    DevScene const &S = B.scenes[lo];
    RenderArgs const &A = B.args[lo];
    uint32_t px = static_cast<uint32_t>(i - B.pix_prefix[lo]);
    float3 o, d;
    camera_ray(S.cam, px % A.width, px / A.width, A.width, A.height, o, d);
    Hit hit = trace_closest<false>(S, o, d, stk + threadIdx.x, nullptr); // the scene's own layout
    FirstHit f;
    f.d = make_float4(d.x, d.y, d.z, 0.0f);
    int32_t mesh = -1, light = -1;
    float3 p = f3(0, 0, 0), n = f3(0, 0, 0);
    if (hit.tri != 0xFFFFFFFFu) {
        Vert v = make_vert(S, hit);
        if (dot(v.n, neg(d)) > 0) {
            mesh = v.mesh;
            p = v.p;
            n = v.n;
            light = __ldg(&S.mesh_light[mesh]);
        }
    }
    f.p = make_float4(p.x, p.y, p.z, __int_as_float(mesh));
    f.n = make_float4(n.x, n.y, n.z, __int_as_float(light));
    out[i] = f;
}

__global__ void k_resolve_batch(BatchDev B, uint64_t total_pix, float4 const *accum, float *rgba) {
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= total_pix)
        return;
    uint32_t lo = 0, hi = B.n;
    while (hi - lo > 1) {
        uint32_t mi = (lo + hi) >> 1;
        if (B.pix_prefix[mi] <= i)
            lo = mi;
        else
            hi = mi;
    }
    uint32_t spp = B.args[lo].spp;
    float inv = spp ? 1.0f / static_cast<float>(spp) : 0.0f;
    float4 a = accum[i];
    reinterpret_cast<float4 *>(rgba)[i] = make_float4(a.x * inv, a.y * inv, a.z * inv, 1.0f);
}

void launch_first_hits_batch(BatchDev const &B, DevScene const *, RenderArgs const *, uint64_t const *h_pix_prefix,
                             FirstHit *fh_all, cudaStream_t st) {
    uint64_t total = h_pix_prefix[B.n];
    if (total)
        k_first_hits_batch<<<static_cast<unsigned>((total + kBlock - 1) / kBlock), kBlock, 0, st>>>(B, total, fh_all);
}

void launch_resolve_batch(BatchDev const &B, uint64_t total_pix, float4 const *accum_all, float *rgba_all,
                          cudaStream_t st) {
    if (total_pix)
        k_resolve_batch<<<static_cast<unsigned>((total_pix + 255) / 256), 256, 0, st>>>(B, total_pix, accum_all, rgba_all);
}

} // namespace e8g
