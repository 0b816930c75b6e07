// Path-replay adjoint of the product estimator (E8G_MODE_MIS): gradients of a loss on the image
// with respect to every material's albedo (3 channels) and GGX roughness.
//
// Each path is recomputed from its counter-based (Philox) stream; nothing is stored between the
// forward render and the adjoint. The BSDF value f_j used for the continuation at vertex j
// multiplies every contribution gathered after it, i.e. L - L_j with L the path's radiance and
// L_j the radiance gathered before that scatter; the BSDF value of the light sample at vertex j
// multiplies that sample's contribution only. Sampling densities and MIS weights are held fixed
// (weights still sum to one, so the gradient estimate stays unbiased), and since f is linear in
// albedo and d ln f / d r follows from GGX's D and G, each vertex adds
//     dL/d albedo_c += w_c (C_c / albedo_c)        dL/d r += (w . C) d ln f / d r
// with C the contribution it multiplies and w the upstream gradient of the path's pixel / spp.
// One walk does it: light-sample terms are added at once, and the first kScatterList scatters
// are recorded as (material, d ln f / d r, L_j) and added when the walk ends and L is known.
// A path with more scatters than that is walked a second time for the rest (the classic
// two-pass replay), which only paths longer than kScatterList vertices pay.
// Gradients are summed per block in shared memory and flushed with one atomic per material.
// Materials whose parameters do not enter f linearly (mixtures, the fail-safe material) and the
// Oren-Nayar sigma receive no gradient.
#include "../../include/e8g.h"
#include "adjoint.h"
#include "mega_pool.cuh"

namespace e8g {

namespace {

// d ln f / d r of cook_torr at (n, o, i), f = F D G / (4 cos_i cos_o) with alpha^2 = 2 r^2.
__device__ __forceinline__ float ct_dlog_dr(const DevMaterial &m, float3 n, float3 o, float3 i) {
    float3 h = add(i, o);
    if (vequals0(h))
        return 0.0f;
    h = normalize(h);
    float a2 = m.alpha2;
    float ch = dot(n, h);
    float c2 = ch * ch;
    float t2 = (1.0f - c2) / c2;
    float k = 1.0f + t2 / a2;
    float dlnD = -1.0f / a2 + 2.0f * t2 / (a2 * a2 * k);
    float ci = dot(n, i), co = dot(n, o);
    float ti = (1.0f - ci * ci) / (ci * ci), to = (1.0f - co * co) / (co * co);
    float si = sqrtf(1.0f + a2 * ti), so = sqrtf(1.0f + a2 * to);
    float li = (-1.0f + si) / 2.0f, lo = (-1.0f + so) / 2.0f;
    float dli = ti / (4.0f * si), dlo = to / (4.0f * so);
    float dlnG = -(dli + dlo) / (1.0f + li + lo);
    return (dlnD + dlnG) * 4.0f * m.rough;
}

struct GradAcc {
    float *a; // 3 per material (shared memory)
    float *r; // 1 per material
    uint32_t nmat;
};

constexpr uint32_t kScatterList = 8;

struct ScatterRec {
    int32_t mat;  // -1: no gradient (other material types)
    float dlog;   // d ln f / d r (cook_torr), else 0
    float3 L;     // radiance gathered before the scatter
};

// Material index receiving gradients at a vertex of this mesh, or -1.
__device__ __forceinline__ int32_t grad_mat(DevScene const &S, uint32_t nmat, int32_t mesh) {
    int32_t mi = __ldg(&S.mesh_mat[mesh]);
    if (mi < 0 || static_cast<uint32_t>(mi) >= nmat)
        return -1;
    uint32_t t = S.mats[mi].type;
    return (t == E8G_MAT_OREN_NAYAR || t == E8G_MAT_COOK_TORR) ? mi : -1;
}

__device__ __forceinline__ void add_grad_m(GradAcc &g, DevScene const &S, int32_t mi, float dlog, float3 C, float3 w) {
    const DevMaterial &m = S.mats[mi];
    if (m.albedo[0] > 0.0f)
        atomicAdd(&g.a[3 * mi], w.x * C.x / m.albedo[0]);
    if (m.albedo[1] > 0.0f)
        atomicAdd(&g.a[3 * mi + 1], w.y * C.y / m.albedo[1]);
    if (m.albedo[2] > 0.0f)
        atomicAdd(&g.a[3 * mi + 2], w.z * C.z / m.albedo[2]);
    if (m.type == E8G_MAT_COOK_TORR)
        atomicAdd(&g.r[mi], dot(w, C) * dlog);
}

__device__ __forceinline__ float grad_dlog(DevScene const &S, int32_t mi, float3 n, float3 o, float3 i) {
    const DevMaterial &m = S.mats[mi];
    return m.type == E8G_MAT_COOK_TORR ? ct_dlog_dr(m, n, o, i) : 0.0f;
}

// One walk of the MIS path in megakernel/oracle order.
// FIRST: adds the light-sample terms, records the first kScatterList scatters in `rec` and
// counts every scatter in *nscatter; returns L. !FIRST (second walk, L = Ltot known): adds the
// terms of scatters kScatterList and later only.
template <bool FIRST, int LAYOUT>
__device__ float3 replay(DevScene const &S, RenderArgs const &A, FirstHit const &f, uint32_t pixel, uint32_t sample,
                         float3 Ltot, float3 w, GradAcc &g, uint32_t *stk, ScatterRec *rec, uint32_t *nscatter) {
    RngPhiloxMem rng;
    rng.seed(A.seed, pixel, sample);
    float3 p = xyz(f.p), n = xyz(f.n), o = neg(xyz(f.d));
    int32_t mesh = __float_as_int(f.p.w);
    float3 L = f3(0, 0, 0);
    int32_t l0 = __float_as_int(f.n.w);
    if (l0 >= 0)
        L = light_radiance(S, l0, o, n);
    float3 beta = f3(1.0f, 1.0f, 1.0f);
    uint32_t scat = 0;
    for (uint32_t depth = 0;; depth++) {
        if ((A.max_depth && depth >= A.max_depth) || depth >= kHardDepth)
            break;
        if (depth >= A.rr_start) {
            if (rng.next() >= A.rr_prob)
                break;
            beta = divs(beta, A.rr_prob);
        }
        const DevMaterial &m = vert_mat(S, mesh);
        float pmf;
        int light = sample_light(S, rng, pmf);
        Surf ls = mesh_sample(S, __ldg(&S.light_mesh[light]), rng, true);
        float3 l = sub(p, ls.p);
        float r2 = dot(l, l);
        float dist = sqrtf(r2);
        float3 ln = divs(l, dist);
        float cos_l = dot(ls.n, ln);
        float3 wi = neg(ln);
        float cos_x = dot(n, wi);
        if (cos_l > 0.0f && cos_x > 0.0f) {
            float3 fv = bsdf_eval(S, m, n, o, wi);
            if (!vequals0(fv)) {
                float p_l = pmf * ls.area_dens * r2 / cos_l;
                float p_b = bsdf_pdf(S, m, n, o, wi);
                if (trace_l<LAYOUT, false>(S, p, wi, 1e-4f, dist - 1e-3f, true, stk, nullptr).tri == 0xFFFFFFFFu) {
                    float wgt = power_heuristic(p_l, p_b);
                    float3 c = scale(mul(mul(beta, fv), light_rad(S, light)), cos_x * wgt / p_l);
                    L = add(L, c);
                    if (FIRST) {
                        int32_t mi = grad_mat(S, g.nmat, mesh);
                        if (mi >= 0)
                            add_grad_m(g, S, mi, grad_dlog(S, mi, n, o, wi), c, w);
                    }
                }
            }
        }
        float pdf;
        float3 i = bsdf_sample_mis(S, m, rng, pdf, n, o);
        if (!(pdf > 0.0f))
            break;
        float cw = dot(n, i);
        if (cw <= 0.0f)
            break;
        float3 fv = bsdf_eval(S, m, n, o, i);
        if (FIRST) {
            if (scat < kScatterList) {
                int32_t mi = grad_mat(S, g.nmat, mesh);
                rec[scat].mat = mi;
                rec[scat].dlog = mi >= 0 ? grad_dlog(S, mi, n, o, i) : 0.0f;
                rec[scat].L = L;
            }
        } else if (scat >= kScatterList) {
            int32_t mi = grad_mat(S, g.nmat, mesh);
            if (mi >= 0)
                add_grad_m(g, S, mi, grad_dlog(S, mi, n, o, i), sub(Ltot, L), w); // gathered after this scatter
        }
        scat++;
        beta = mul(beta, scale(fv, cw / pdf));
        Hit h = trace_l<LAYOUT, false>(S, p, i, 1e-4f, 1000.0f, false, stk, nullptr);
        if (h.tri == 0xFFFFFFFFu)
            break;
        Vert nv = make_vert(S, h);
        if (dot(nv.n, neg(i)) <= 0.0f)
            break;
        int32_t hl = __ldg(&S.mesh_light[nv.mesh]);
        if (hl >= 0) {
            float cos_l2 = dot(nv.n, neg(i));
            float pl = __ldg(&S.light_pnorm[hl]) / S.total_power;
            float inv_area = 1.0f / __ldg(&S.mesh_area[__ldg(&S.light_mesh[hl])]);
            float p_l = pl * inv_area * (nv.t * nv.t) / cos_l2;
            L = add(L, scale(mul(beta, light_rad(S, hl)), power_heuristic(pdf, p_l)));
        }
        p = nv.p;
        n = nv.n;
        mesh = nv.mesh;
        o = neg(i);
    }
    if (FIRST)
        *nscatter = scat;
    return L;
}

template <int LAYOUT>
__global__ void __launch_bounds__(kBlock) k_adjoint(DevScene S, RenderArgs A, FirstHit const *__restrict__ fh,
                                                    float const *__restrict__ dl_dimage, float inv_spp,
                                                    unsigned long long *work, float *d_albedo, float *d_rough,
                                                    float *path_rgb) {
    __shared__ uint32_t stk_all[kStackOf<LAYOUT> * kBlock];
    extern __shared__ float sgrad[];
    GradAcc g{sgrad, sgrad + 3 * S.nmat, S.nmat};
    for (uint32_t k = threadIdx.x; k < 4 * S.nmat; k += blockDim.x)
        sgrad[k] = 0.0f;
    __syncthreads();
    uint32_t *stk = stk_all + threadIdx.x;
    const uint32_t lane = lane_id();
    while (true) {
        unsigned long long base = 0;
        if (lane == 0)
            base = atomicAdd(work, 32ull);
        base = __shfl_sync(~0u, base, 0);
        if (base >= A.total_paths)
            break;
        uint64_t idx = base + lane;
        if (idx < A.total_paths) {
            uint32_t pixel, sample, out;
            bool ok = path_coords(A, idx, pixel, sample, out);
            if (ok) {
                FirstHit f = fh[pixel];
                if (__float_as_int(f.p.w) >= 0) {
                    float3 w = scale(f3(dl_dimage[3 * static_cast<size_t>(pixel)], dl_dimage[3 * static_cast<size_t>(pixel) + 1],
                                        dl_dimage[3 * static_cast<size_t>(pixel) + 2]),
                                     inv_spp);
                    ScatterRec rec[kScatterList];
                    uint32_t ns = 0;
                    float3 Ltot = replay<true, LAYOUT>(S, A, f, pixel, sample, f3(0, 0, 0), w, g, stk, rec, &ns);
                    uint32_t nl = ns < kScatterList ? ns : kScatterList;
                    for (uint32_t j = 0; j < nl; j++)
                        if (rec[j].mat >= 0)
                            add_grad_m(g, S, rec[j].mat, rec[j].dlog, sub(Ltot, rec[j].L), w);
                    if (ns > kScatterList)
                        replay<false, LAYOUT>(S, A, f, pixel, sample, Ltot, w, g, stk, nullptr, nullptr);
                    if (path_rgb) {
                        path_rgb[3 * idx] = Ltot.x;
                        path_rgb[3 * idx + 1] = Ltot.y;
                        path_rgb[3 * idx + 2] = Ltot.z;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * S.nmat; k += blockDim.x)
        if (sgrad[k] != 0.0f)
            atomicAdd(&d_albedo[k], sgrad[k]);
    for (uint32_t k = threadIdx.x; k < S.nmat; k += blockDim.x)
        if (sgrad[3 * S.nmat + k] != 0.0f)
            atomicAdd(&d_rough[k], sgrad[3 * S.nmat + k]);
}

// ---- the same over block-local path pools (mega_pool.cuh) ----
// k_adjoint walks one path per lane, so a warp waits for the longest of its rays at every vertex and
// for its longest path (4.7 of 32 lanes active). Here the walk's state lives in a pool slot: the
// radiance gathered so far, the last scatter (material, d ln f / d r), the light sample's d ln f / d r
// and the list of scatters with the radiance before each. A light sample's term is added once its
// shadow ray is back; a scatter enters the list when its ray has made a vertex (one whose
// ray left the scene gathers nothing after it); a path's end adds the list. A path that made more
// vertices than the list holds starts over in its slot and adds the later scatters directly, its
// radiance being known.
// Slot arrays beside those of mega_pool.cuh (kPoolRad's w: 1 on the second walk): the last scatter
// (x: material, y: its d ln f / d r, z: the light sample's d ln f / d r), and the list's entries,
// (radiance, d ln f / d r) and the materials four to an array; the second walk keeps the path's whole
// radiance in the first entry.
// One gradient term per lane with `on`, all lanes of the warp calling: the terms of the material that
// most lanes share are summed across the warp and added once, the others by their lanes. Float adds
// in shared memory are compare-and-swap loops, and half of a scene's vertices may lie on one
// material. The sums are of w C; the division by the albedo is the block's last step.
__device__ __forceinline__ void add_grad_warp(GradAcc &g, bool on, int32_t mi, float dlog, float3 C, float3 w) {
    on = on && mi >= 0;
    if (!__ballot_sync(~0u, on))
        return;
    const uint32_t lane = lane_id();
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (on)
        x = make_float4(w.x * C.x, w.y * C.y, w.z * C.z, dot(w, C) * dlog);
    const uint32_t peers = __match_any_sync(~0u, on ? mi : -1);
    const uint32_t best = __reduce_max_sync(~0u, on ? static_cast<uint32_t>(__popc(peers)) << 5 | lane : 0u);
    if (best >> 5 >= 4) {
        const int32_t m = __shfl_sync(~0u, mi, best & 31u);
        const bool mine = on && mi == m;
        float4 y = mine ? x : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int k = 16; k > 0; k >>= 1) {
            y.x += __shfl_xor_sync(~0u, y.x, k);
            y.y += __shfl_xor_sync(~0u, y.y, k);
            y.z += __shfl_xor_sync(~0u, y.z, k);
            y.w += __shfl_xor_sync(~0u, y.w, k);
        }
        if (lane == (best & 31u))
            x = y;
        else if (mine)
            on = false;
    }
    if (on) {
        atomicAdd(&g.a[3 * mi], x.x);
        atomicAdd(&g.a[3 * mi + 1], x.y);
        atomicAdd(&g.a[3 * mi + 2], x.z);
        if (x.w != 0.0f)
            atomicAdd(&g.r[mi], x.w);
    }
}

enum { kAdjScat = kPoolArrays, kAdjRec, kAdjMat = kAdjRec + kScatterList, kAdjArrays = kAdjMat + kScatterList / 4 };

__device__ __forceinline__ float3 pixel_grad(float const *dl_dimage, uint32_t pixel, float inv_spp) {
    float const *d = dl_dimage + 3 * static_cast<size_t>(pixel);
    return scale(f3(d[0], d[1], d[2]), inv_spp);
}

// Measured on the differentiable configuration (327,690 triangles, 256 materials, 512 x 512, 32 spp,
// depth 6), device time of the backward kernel: one path per lane 12.6 ms on the pairs and 19.5 on the
// eight-wide tree; pools 10.7 and 10.4; with the terms summed per warp (add_grad_warp) 8.3 and 8.1.
// 5 / 6 / 7 / 8 blocks per SM: 8.9 / 8.3 / 8.5 / 8.2 on the pairs, 8.2 / 8.1 / 8.2 / 8.7 on the wide tree.
// It is bound as the pooled megakernel is, by issue slots and latency, three quarters of it tracing.
constexpr int kAdjBlocks = 6;
template <int LAYOUT>
__global__ void __launch_bounds__(kBlock, kAdjBlocks)
    k_adjoint_pool(const __grid_constant__ DevScene S, const __grid_constant__ RenderArgs A,
                   FirstHit const *__restrict__ fh, float const *__restrict__ dl_dimage, float inv_spp,
                   unsigned long long *work, float *d_albedo, float *d_rough, float4 *pool, uint32_t slots,
                   uint32_t keep) {
    __shared__ uint32_t stk_all[kStackOf<LAYOUT> * kBlock];
    __shared__ PoolQueue Q;
    extern __shared__ float sgrad[];
    GradAcc g{sgrad, sgrad + 3 * S.nmat, S.nmat};
    for (uint32_t k = threadIdx.x; k < 4 * S.nmat; k += kBlock)
        sgrad[k] = 0.0f;
    uint32_t *stk = stk_all + threadIdx.x;
    float4 *P = pool + static_cast<size_t>(blockIdx.x) * kAdjArrays * slots;
    for (uint32_t s = threadIdx.x; s < slots; s += kBlock)
        Q.ext_st[s] = Q.sh_st[s] = kRayNone;
    if (threadIdx.x == 0)
        Q.n_ext = Q.n_sh = Q.head = Q.over = 0;
    __syncthreads();
    PoolLane L;
    L.cur = kPoolNone;
    L.any = false;
    while (true) {
        for (uint32_t s0 = 0; s0 < slots; s0 += kBlock) {
            __syncthreads(); // warps together in the code, as in k_mega_pool
            const uint32_t s = s0 + threadIdx.x;
            bool at_vertex = false, fresh = false, second = false;
            PoolVertex v;
            RngPhilox rng;
            uint32_t pixel = 0, sample = 0;
            float3 rad = f3(0, 0, 0), before = rad; // the radiance gathered so far, and before the vertex's emission
            const uint32_t es = Q.ext_st[s], sh = Q.sh_st[s];
            const bool open = es != kRayOut && sh != kRayOut;
            const bool back = open && es != kRayNone; // a path whose rays are back
            float4 sc = make_float4(__int_as_float(-1), 0.0f, 0.0f, 0.0f);
            float3 w = f3(0, 0, 0), c = f3(0, 0, 0);
            uint32_t made = 0; // vertices made so far, and scatters with a vertex after them
            uint32_t nl = 0;   // list entries to add: the path ended
            if (back) {
                const float4 ids = P[kPoolIds * slots + s], l4 = P[kPoolRad * slots + s];
                pixel = __float_as_uint(ids.x);
                sample = __float_as_uint(ids.y);
                rad = xyz(l4);
                second = l4.w != 0.0f;
                sc = P[kAdjScat * slots + s];
                w = pixel_grad(dl_dimage, pixel, inv_spp);
                if (sh == kRayHit) { // the light sample is unoccluded
                    c = xyz(P[kPoolShAdd * slots + s]);
                    rad = ::e8g::add(rad, c);
                }
                const float4 dd = P[kPoolDir * slots + s];
                made = __float_as_uint(dd.w);
                if (es == kRayHit) {
                    const float4 hv = P[kPoolHit * slots + s];
                    float3 add = f3(0, 0, 0);
                    at_vertex = __float_as_uint(hv.y) != 0xFFFFFFFFu &&
                                pool_complete<E8G_MODE_MIS>(S, hv, dd, P[kPoolBeta * slots + s], v, add);
                    if (at_vertex) {
                        if (!second && made < kScatterList) {
                            P[(kAdjRec + made) * slots + s] = make_float4(rad.x, rad.y, rad.z, sc.y);
                            reinterpret_cast<float *>(&P[(kAdjMat + made / 4) * slots + s])[made & 3u] = sc.x;
                        }
                        rng = RngSlot<RngPhilox>::load(A, pixel, sample, __float_as_uint(ids.w));
                        before = rad;
                        rad = ::e8g::add(rad, add);
                    }
                }
                if (!at_vertex && !second)
                    nl = made < kScatterList ? made : kScatterList;
            }
            add_grad_warp(g, back && sh == kRayHit && !second, __float_as_int(sc.x), sc.z, c, w);
            if (__ballot_sync(~0u, second && at_vertex && made >= kScatterList)) // the scatters beyond the list
                add_grad_warp(g, second && at_vertex && made >= kScatterList, __float_as_int(sc.x), sc.y,
                              sub(xyz(P[kAdjRec * slots + s]), before), w);
            const uint32_t most = __reduce_max_sync(~0u, nl);
            for (uint32_t j = 0; j < most; j++) {
                float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                int32_t mi = -1;
                if (j < nl) {
                    r = P[(kAdjRec + j) * slots + s];
                    mi = __float_as_int(reinterpret_cast<float const *>(&P[(kAdjMat + j / 4) * slots + s])[j & 3u]);
                }
                add_grad_warp(g, j < nl, mi, r.w, sub(rad, xyz(r)), w);
            }
            if (back && !at_vertex && !second && made > kScatterList) { // walk again for the later scatters
                P[kAdjRec * slots + s] = make_float4(rad.x, rad.y, rad.z, 0.0f);
                second = fresh = at_vertex = true;
            }
            bool want = open && !at_vertex && Q.over == 0;
            if (want)
                second = false;
            while (const uint32_t mask = __ballot_sync(~0u, want)) {
                const uint64_t idx = pool_next_path(work, mask);
                uint32_t out;
                if (want) {
                    if (idx >= A.total_paths) {
                        want = false;
                        Q.over = 1;
                    } else if (path_coords(A, idx, pixel, sample, out)) {
                        fresh = at_vertex = __float_as_int(fh[pixel].p.w) >= 0;
                        want = !at_vertex;
                    }
                }
            }
            __syncthreads();
            if (fresh) {
                const FirstHit f = fh[pixel];
                pool_start(f, v);
                rng = RngSlot<RngPhilox>::fresh(A, 0, pixel, sample);
                const int32_t light = __float_as_int(f.n.w);
                rad = light >= 0 ? light_radiance(S, light, v.o, v.n) : f3(0, 0, 0);
            }
            bool shadow = false, extend = false;
            if (at_vertex) {
                PoolRays q;
                pool_shade<E8G_MODE_MIS>(S, A, v, rng, q);
                shadow = q.shadow;
                extend = q.extend;
                const int32_t mi = shadow || extend ? grad_mat(S, S.nmat, v.mesh) : -1;
                float dl_scat = 0.0f, dl_light = 0.0f;
                if (mi >= 0) {
                    if (shadow && !second)
                        dl_light = grad_dlog(S, mi, v.n, v.o, q.sd);
                    if (extend)
                        dl_scat = grad_dlog(S, mi, v.n, v.o, q.i);
                }
                if (extend)
                    P[kPoolBeta * slots + s] = make_float4(v.beta.x, v.beta.y, v.beta.z, q.pdf);
                P[kPoolDir * slots + s] = make_float4(q.i.x, q.i.y, q.i.z, __uint_as_float(v.depth));
                if (shadow) {
                    P[kPoolShDir * slots + s] = make_float4(q.sd.x, q.sd.y, q.sd.z, q.st);
                    P[kPoolShAdd * slots + s] = make_float4(q.vis.x, q.vis.y, q.vis.z, 0.0f);
                }
                P[kPoolPos * slots + s] = make_float4(v.p.x, v.p.y, v.p.z, 0.0f);
                P[kPoolIds * slots + s] = make_float4(__uint_as_float(pixel), __uint_as_float(sample), 0.0f,
                                                      __uint_as_float(RngSlot<RngPhilox>::store(rng)));
                P[kPoolRad * slots + s] = make_float4(rad.x, rad.y, rad.z, second ? 1.0f : 0.0f);
                P[kAdjScat * slots + s] = make_float4(__int_as_float(mi), dl_scat, dl_light, 0.0f);
            }
            if (open) { // kRayEnd: no extension ray, the path ends once its shadow ray is back
                Q.ext_st[s] = extend ? kRayOut : at_vertex ? kRayEnd : kRayNone;
                Q.sh_st[s] = shadow ? kRayOut : kRayNone;
            }
            pool_push(Q, s, extend, shadow);
        }
        // slots that ended without a shadow ray still have their list to add: one more round
        bool pending = L.cur != kPoolNone;
        for (uint32_t s = threadIdx.x; s < slots; s += kBlock)
            pending = pending || Q.ext_st[s] != kRayNone;
        const int more = __syncthreads_or(pending);
        const uint32_t ne = Q.n_ext, n = ne + Q.n_sh;
        if (n == 0 && Q.over && !more)
            break;
        pool_trace<LAYOUT>(S, L, P, slots, Q, ne, n, stk, keep);
        __syncthreads();
        if (threadIdx.x == 0)
            Q.n_ext = Q.n_sh = Q.head = 0;
        __syncthreads();
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * S.nmat; k += kBlock) {
        const float al = S.mats[k / 3].albedo[k % 3];
        if (sgrad[k] != 0.0f && al > 0.0f)
            atomicAdd(&d_albedo[k], sgrad[k] / al);
    }
    for (uint32_t k = threadIdx.x; k < S.nmat; k += kBlock)
        if (sgrad[3 * S.nmat + k] != 0.0f)
            atomicAdd(&d_rough[k], sgrad[3 * S.nmat + k]);
}

} // namespace

namespace {
// Blocks, slots and bytes of the pooled backward; slots 0 where it does not run: other trees, renders
// below the pooled megakernel's line, and material tables whose sums (16 bytes each) would take more
// shared memory than leaves three blocks to an SM.
AdjointPool plan(DevScene const &S, RenderArgs const &A, int num_sms) {
    AdjointPool p;
    const size_t smem = static_cast<size_t>(S.nmat) * 4 * sizeof(float);
    if ((S.layout != 0 && S.layout != 2) || A.total_paths < (1u << 19) || smem > 64 * 1024)
        return p;
    auto *kern = S.layout == 2 ? k_adjoint_pool<2> : k_adjoint_pool<0>;
    int per_sm = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return p;
    }
    p.grid = num_sms * per_sm;
    p.slots = std::min<uint32_t>(pool_slots(A, num_sms), 512);
    p.bytes = static_cast<size_t>(p.grid) * p.slots * kAdjArrays * sizeof(float4);
    return p;
}
} // namespace

AdjointPool adjoint_pool(DevScene const &S, RenderArgs const &A, int num_sms) { return plan(S, A, num_sms); }

cudaError_t launch_adjoint_pool(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float const *dl_dimage,
                                float inv_spp, unsigned long long *work, float *d_albedo, float *d_rough,
                                AdjointPool const &p, void *pool, cudaStream_t st) {
    const size_t smem = static_cast<size_t>(S.nmat) * 4 * sizeof(float);
    auto *kern = S.layout == 2 ? k_adjoint_pool<2> : k_adjoint_pool<0>;
    kern<<<p.grid, kBlock, smem, st>>>(S, A, fh, dl_dimage, inv_spp, work, d_albedo, d_rough,
                                       static_cast<float4 *>(pool), p.slots, pool_keep(S));
    return cudaGetLastError();
}

cudaError_t launch_adjoint(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float const *dl_dimage,
                           float inv_spp, unsigned long long *work, float *d_albedo, float *d_rough, float *path_rgb,
                           int num_sms, cudaStream_t st) {
    size_t smem = static_cast<size_t>(S.nmat) * 4 * sizeof(float);
    if (smem + kStackWords * kBlock * sizeof(uint32_t) > 200 * 1024)
        return cudaErrorInvalidValue;
    auto kern = S.layout == 1 ? k_adjoint<1>
                              : (S.layout == 2 ? k_adjoint<2> : (S.layout == 3 ? k_adjoint<3> : k_adjoint<0>));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, smem);
    int grid = num_sms * (per_sm > 0 ? per_sm : 1);
    kern<<<grid, kBlock, smem, st>>>(S, A, fh, dl_dimage, inv_spp, work, d_albedo, d_rough, path_rgb);
    return cudaGetLastError();
}

} // namespace e8g
