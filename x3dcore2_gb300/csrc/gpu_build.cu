// BVH build on the device: Morton order, PLOC clustering, SAH leaf collapse, and the SAH-pair node
// layout of the host builder (bvh.h).
//
// 1. Per triangle: exact box, centroid, scene box; a 30-bit Morton code of the centroid in the
//    centroids' box; a stable LSD radix sort of (code, triangle) pairs, 8 bits per pass.
// 2. PLOC (Meister and Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
//    Hierarchy Construction", IEEE TVCG 2018): the sorted triangles are the initial clusters;
//    every round each cluster finds, among the clusters within kPlocRadius positions in the
//    current order, the one whose union box has the smallest surface area (ties to the lower
//    position); mutual nearest neighbours merge into a new node, which takes the lower position,
//    and the cluster array is compacted. The round with the globally cheapest pair always merges
//    it, so the loop ends with one cluster.
// 3. Bottom-up (a thread per triangle, the last child to arrive at a node carries on): triangle
//    counts and the SAH cost min(tri_cost A n, node_cost A + C(left) + C(right)); subtrees of at
//    most max_leaf_prims triangles whose leaf cost is not above their inner cost become leaves.
// 4. Top-down, one launch per level: every node of the level writes its 32-byte record (boxes
//    pushed out exactly as the host builder pushes them out, bvh_boxes.h) at its depth-first
//    preorder slot (the host builder's order: children adjacent, the k-th interior node's at 1 + 2k,
//    from interior-node counts of the subtrees); then a thread per triangle writes its record.
// Every byte of the tree is deterministic: scans decide the clusters' and wide nodes' positions, and the
// flattening's items carry theirs (only the order of a level's work list comes from an atomic).
// Counts stay on the device: rounds and levels follow each other in the stream with grids for the
// most they can hold, and the host reads back every few rounds and at the end. 525 launches and about
// 70 reads made 5.7 ms of the 1.3M-triangle scene's eight-wide build; it is 236 launches, a dozen
// reads and 2.8 ms (pairs 4.3 -> 2.1).
#include "bvh_boxes.h"
#include "gpu_build.h"
#include "launch.h"

#include <algorithm>
#include <cstring>
#include <vector>

namespace e8g {
namespace {

constexpr int kGB = 256;          // threads per block
constexpr int kSortItems = 8;     // keys per thread in the sort
constexpr int kSortTile = kGB * kSortItems;
constexpr int kScanItems = 4;     // elements per thread in the device-wide scan
constexpr int kScanTile = 1024 * kScanItems;
constexpr int kPlocRadius = 24;
constexpr int kLevels = 40;       // entries of the per-level states (trees are at most 32 levels deep)

__device__ __forceinline__ uint32_t ord_key(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Inclusive scan of one value per thread over a block of `threads` threads (a multiple of 32).
template <int THREADS, class T> __device__ __forceinline__ T block_inclusive(T v, T *sh) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T x = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o)
            v += x;
    }
    if (lane == 31)
        sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        T w = lane < THREADS / 32 ? sh[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T x = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o)
                w += x;
        }
        if (lane < THREADS / 32)
            sh[lane] = w;
    }
    __syncthreads();
    T r = v + (warp ? sh[warp - 1] : T(0));
    __syncthreads();
    return r;
}

// ------------------------------------------------------------------ device-wide scan ----
// Exclusive scan in place of n values; sums[] receives one total per tile. Three launches.

__global__ void __launch_bounds__(1024) k_scan_tiles(uint32_t *d, uint32_t n, uint32_t *sums) {
    __shared__ uint32_t sh[32];
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems], t = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? d[base + k] : 0;
        t += v[k];
    }
    uint32_t incl = block_inclusive<1024>(t, sh);
    uint32_t run = incl - t;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n)
            d[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 1023)
        sums[blockIdx.x] = incl;
}

// Scans the tile totals (any count, one block) and writes the grand total to *total.
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t *sums, uint32_t m, uint32_t *total) {
    __shared__ uint32_t sh[32];
    uint32_t carry = 0;
    for (uint32_t b = 0; b < m; b += 1024) {
        uint32_t i = b + threadIdx.x;
        uint32_t v = i < m ? sums[i] : 0;
        uint32_t incl = block_inclusive<1024>(v, sh);
        if (i < m)
            sums[i] = carry + incl - v;
        carry += sh[31]; // the block's total
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *total = carry;
}

__global__ void __launch_bounds__(1024) k_scan_add(uint32_t *d, uint32_t n, uint32_t const *sums) {
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t add = sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n)
            d[base + k] += add;
}

// ------------------------------------------------------------------ radix sort ----

__global__ void __launch_bounds__(kGB) k_sort_hist(uint32_t const *keys, uint32_t n, int shift, uint32_t *hist) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    uint32_t base = blockIdx.x * kSortTile;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        uint32_t i = base + k * kGB + threadIdx.x;
        if (i < n)
            atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x]; // digit-major
}

// Stable scatter of one tile: every key's rank among the equal digits before it (a warp matches 32 keys
// at a time and keeps its own digit counts), one scan of the tile's digit counts, the tile put in
// digit order in shared memory and written from there in runs. Eight one-bit splits with a block scan
// each took 50 us a pass of 1.3M keys, this 21.
__global__ void __launch_bounds__(kGB)
    k_sort_scatter(uint32_t const *kin, uint32_t const *vin, uint32_t *kout, uint32_t *vout, uint32_t n, int shift,
                   uint32_t const *offs) {
    __shared__ uint32_t sk[kSortTile], sv[kSortTile];
    __shared__ uint32_t counts[kGB / 32][256]; // per warp and digit: the count, then where the warp's keys start
    __shared__ uint32_t start[256];
    __shared__ uint32_t sh[32];
    static_assert(kGB == 256, "a thread per digit");
    const uint32_t base = blockIdx.x * kSortTile, lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
    const uint32_t valid = min(static_cast<uint32_t>(kSortTile), n - base);
    for (int w = 0; w < kGB / 32; w++)
        counts[w][threadIdx.x] = 0;
    __syncthreads();
    uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t p = warp * (32 * kSortItems) + k * 32 + lane;
        const bool in = p < valid;
        key[k] = in ? kin[base + p] : 0;
        val[k] = in ? vin[base + p] : 0;
        const uint32_t d = (key[k] >> shift) & 255u;
        const uint32_t peers = __match_any_sync(~0u, in ? d : 256u);
        const uint32_t before = in ? counts[warp][d] : 0;
        rank[k] = before + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (in && lane == 31u - __clz(peers)) // the last of the equal digits
            counts[warp][d] = rank[k] + 1;
        __syncwarp();
    }
    __syncthreads();
    uint32_t sum = 0;
    for (int w = 0; w < kGB / 32; w++) {
        const uint32_t c = counts[w][threadIdx.x];
        counts[w][threadIdx.x] = sum;
        sum += c;
    }
    start[threadIdx.x] = block_inclusive<kGB>(sum, sh) - sum;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        if (warp * (32 * kSortItems) + k * 32 + lane < valid) {
            const uint32_t d = (key[k] >> shift) & 255u, p = start[d] + counts[warp][d] + rank[k];
            sk[p] = key[k];
            sv[p] = val[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t p = k * kGB + threadIdx.x;
        if (p < valid) {
            const uint32_t x = sk[p], d = (x >> shift) & 255u;
            const uint32_t dst = offs[d * gridDim.x + blockIdx.x] + (p - start[d]);
            kout[dst] = x;
            vout[dst] = sv[p];
        }
    }
}

// ------------------------------------------------------------------ primitives ----

__global__ void k_build_init(uint32_t *red) {
    if (threadIdx.x < 12) // [0..2] min, [3..5] max of boxes; [6..8] min, [9..11] max of centroids
        red[threadIdx.x] = (threadIdx.x < 3 || (threadIdx.x >= 6 && threadIdx.x < 9)) ? 0xFFFFFFFFu : 0u;
}

template <int N, bool MAX> __device__ __forceinline__ void reduce_to(uint32_t (&v)[N], uint32_t *red) {
    __shared__ uint32_t sh[kGB / 32][N];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            uint32_t x = __shfl_xor_sync(0xFFFFFFFFu, v[k], o);
            v[k] = MAX ? max(v[k], x) : min(v[k], x);
        }
        if (lane == 0)
            sh[warp][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        uint32_t r = sh[0][threadIdx.x];
        for (int w = 1; w < kGB / 32; w++)
            r = MAX ? max(r, sh[w][threadIdx.x]) : min(r, sh[w][threadIdx.x]);
        if (MAX)
            atomicMax(&red[threadIdx.x], r);
        else
            atomicMin(&red[threadIdx.x], r);
    }
    __syncthreads();
}

// Leaf boxes (node i = triangle i before sorting) and the boxes of all boxes and of all centroids.
__global__ void __launch_bounds__(kGB) k_prim_boxes(uint4 const *tidx, float4 const *vpos, uint32_t nt, float4 *blo,
                                                     float4 *bhi, uint32_t *red) {
    uint32_t mn[6] = {~0u, ~0u, ~0u, ~0u, ~0u, ~0u}, mx[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        uint4 g = tidx[t];
        float4 p0 = vpos[g.x], p1 = vpos[g.y], p2 = vpos[g.z];
        float lo[3] = {fminf(fminf(p0.x, p1.x), p2.x), fminf(fminf(p0.y, p1.y), p2.y), fminf(fminf(p0.z, p1.z), p2.z)};
        float hi[3] = {fmaxf(fmaxf(p0.x, p1.x), p2.x), fmaxf(fmaxf(p0.y, p1.y), p2.y), fmaxf(fmaxf(p0.z, p1.z), p2.z)};
        blo[t] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        bhi[t] = make_float4(hi[0], hi[1], hi[2], 0.0f);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            float c = 0.5f * (lo[a] + hi[a]);
            mn[a] = min(mn[a], ord_key(lo[a]));
            mx[a] = max(mx[a], ord_key(hi[a]));
            mn[3 + a] = min(mn[3 + a], ord_key(c));
            mx[3 + a] = max(mx[3 + a], ord_key(c));
        }
    }
    uint32_t a[3] = {mn[0], mn[1], mn[2]}, b[3] = {mx[0], mx[1], mx[2]};
    uint32_t c[3] = {mn[3], mn[4], mn[5]}, d[3] = {mx[3], mx[4], mx[5]};
    reduce_to<3, false>(a, red);
    reduce_to<3, true>(b, red + 3);
    reduce_to<3, false>(c, red + 6);
    reduce_to<3, true>(d, red + 9);
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void k_morton(float4 const *blo, float4 const *bhi, uint32_t nt, uint32_t const *red, uint32_t *keys,
                         uint32_t *vals) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt)
        return;
    float4 lo = blo[t], hi = bhi[t];
    float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t code = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float cl = key_float(red[6 + a]), ch = key_float(red[9 + a]);
        float ext = ch - cl;
        float u = ext > 0.0f ? (c[a] - cl) / ext : 0.0f;
        uint32_t q = static_cast<uint32_t>(fminf(fmaxf(u * 1024.0f, 0.0f), 1023.0f));
        code |= spread10(q) << (2 - a);
    }
    keys[t] = code;
    vals[t] = t;
}

// Leaf nodes 0..n-1 in sorted order: boxes gathered from the triangle boxes.
__global__ void k_gather_leaves(uint32_t const *order, float4 const *tlo, float4 const *thi, uint32_t n, float4 *blo,
                                float4 *bhi, uint32_t *clusters) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    uint32_t t = order[i];
    blo[i] = tlo[t];
    bhi[i] = thi[t];
    clusters[i] = i;
}

// ------------------------------------------------------------------------ PLOC ----

__device__ __forceinline__ float union_area(float4 a0, float4 a1, float4 b0, float4 b1) {
    float dx = fmaxf(a1.x, b1.x) - fminf(a0.x, b0.x);
    float dy = fmaxf(a1.y, b1.y) - fminf(a0.y, b0.y);
    float dz = fmaxf(a1.z, b1.z) - fminf(a0.z, b0.z);
    return dx * dy + dy * dz + dz * dx;
}

// A round: neighbours, a scan of the merge and keep flags (two counts in one 64-bit word, tile by
// tile), the tile totals, and the merges. The cluster count stays on the device: round r reads
// state[r & 1] and writes the other one, so the host looks only every few rounds (kPlocBatch), with
// grids for the count it last saw. Once kPlocSmall clusters are left a round does nothing.
struct PlocState {
    uint32_t m, base;  // clusters, next tree node
    uint32_t cur;      // which cluster array holds them
    uint32_t rounds;
    uint32_t stuck;    // a round found no mutual pair (non-finite boxes)
};
constexpr int kPlocSmall = 2048; // clusters the one-block kernel takes over at
constexpr int kPlocBatch = 4;

__global__ void k_ploc_start(PlocState *state, uint32_t n) { state[0] = PlocState{n, n, 0, 0, 0}; }

__global__ void __launch_bounds__(kGB) k_ploc_nn(PlocState const *state, uint32_t const *c0, uint32_t const *c1,
                                                  float4 const *blo, float4 const *bhi, int32_t *nn) {
    const uint32_t m = state->m;
    if (m <= static_cast<uint32_t>(kPlocSmall) || blockIdx.x * kGB >= m)
        return;
    uint32_t const *clus = state->cur ? c1 : c0;
    __shared__ float4 slo[kGB + 2 * kPlocRadius], shi[kGB + 2 * kPlocRadius];
    int s0 = static_cast<int>(blockIdx.x * kGB) - kPlocRadius;
    for (int k = threadIdx.x; k < kGB + 2 * kPlocRadius; k += kGB) {
        int idx = s0 + k;
        if (idx >= 0 && idx < static_cast<int>(m)) {
            uint32_t node = clus[idx];
            slo[k] = blo[node];
            shi[k] = bhi[node];
        }
    }
    __syncthreads();
    int i = static_cast<int>(blockIdx.x * kGB + threadIdx.x);
    if (i >= static_cast<int>(m))
        return;
    float4 a0 = slo[threadIdx.x + kPlocRadius], a1 = shi[threadIdx.x + kPlocRadius];
    float best = INFINITY;
    int bj = -1;
    for (int d = -kPlocRadius; d <= kPlocRadius; d++) {
        int j = i + d;
        if (d == 0 || j < 0 || j >= static_cast<int>(m))
            continue;
        float area = union_area(a0, a1, slo[threadIdx.x + kPlocRadius + d], shi[threadIdx.x + kPlocRadius + d]);
        if (area < best) { // increasing j: ties keep the lower position
            best = area;
            bj = j;
        }
    }
    nn[i] = bj;
}

// Cluster i's flags: merged in the high word (the lower position of a mutual pair), kept in the low.
__device__ __forceinline__ uint64_t ploc_flags(int32_t const *nn, uint32_t i) {
    int32_t j = nn[i];
    bool mutual = j >= 0 && nn[j] == static_cast<int32_t>(i);
    uint64_t merged = mutual && static_cast<int32_t>(i) < j, keep = !(mutual && static_cast<int32_t>(i) > j);
    return merged << 32 | keep;
}

__global__ void __launch_bounds__(1024) k_ploc_tiles(PlocState const *state, int32_t const *nn, uint64_t *scan,
                                                     uint64_t *sums) {
    const uint32_t m = state->m;
    if (m <= static_cast<uint32_t>(kPlocSmall) || blockIdx.x * kScanTile >= m)
        return;
    __shared__ uint64_t sh[32];
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint64_t v[kScanItems], t = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < m ? ploc_flags(nn, base + k) : 0;
        t += v[k];
    }
    uint64_t incl = block_inclusive<1024>(t, sh);
    uint64_t run = incl - t;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < m)
            scan[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 1023)
        sums[blockIdx.x] = incl;
}

// Exclusive scan of m tile totals in place, one block; the grand total in every thread.
__device__ __forceinline__ uint64_t scan_totals(uint64_t *sums, uint32_t m, uint64_t *sh) {
    uint64_t carry = 0;
    for (uint32_t b = 0; b < m; b += 1024) {
        uint32_t i = b + threadIdx.x;
        uint64_t v = i < m ? sums[i] : 0;
        uint64_t incl = block_inclusive<1024>(v, sh);
        if (i < m)
            sums[i] = carry + incl - v;
        carry += sh[31]; // the block's total
        __syncthreads();
    }
    return carry;
}

__global__ void __launch_bounds__(1024) k_ploc_sums(PlocState const *state, PlocState *next, uint64_t *sums) {
    __shared__ uint64_t sh[32];
    PlocState s = *state;
    if (s.m > static_cast<uint32_t>(kPlocSmall)) {
        uint64_t total = scan_totals(sums, (s.m - 1) / kScanTile + 1, sh);
        uint32_t merged = static_cast<uint32_t>(total >> 32);
        s.stuck |= merged == 0;
        s.m = static_cast<uint32_t>(total);
        s.base += merged;
        s.cur ^= 1u;
        s.rounds++;
    }
    if (threadIdx.x == 0)
        *next = s;
}

__global__ void __launch_bounds__(kGB) k_ploc_apply(PlocState const *state, uint32_t *c0, uint32_t *c1,
                                                     int32_t const *nn, uint64_t const *scan, uint64_t const *sums,
                                                     float4 *blo, float4 *bhi, int2 *child) {
    const uint32_t m = state->m, i = blockIdx.x * kGB + threadIdx.x;
    if (m <= static_cast<uint32_t>(kPlocSmall) || i >= m)
        return;
    uint32_t const *clus = state->cur ? c1 : c0;
    uint32_t *clus_out = state->cur ? c0 : c1;
    const uint64_t f = ploc_flags(nn, i), at = scan[i] + sums[i / kScanTile];
    if (!static_cast<uint32_t>(f))
        return;
    if (f >> 32) {
        uint32_t node = state->base + static_cast<uint32_t>(at >> 32); // < 2n - 1: every merge removes one cluster
        uint32_t a = clus[i], b = clus[nn[i]];
        child[node] = make_int2(static_cast<int>(a), static_cast<int>(b));
        float4 a0 = blo[a], a1 = bhi[a], b0 = blo[b], b1 = bhi[b];
        blo[node] = make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), 0.0f);
        bhi[node] = make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), fmaxf(a1.z, b1.z), 0.0f);
        clus_out[static_cast<uint32_t>(at)] = node;
    } else {
        clus_out[static_cast<uint32_t>(at)] = clus[i];
    }
}

// The last rounds, once few clusters are left, in one block: the same rounds as the kernels above
// (same neighbour search, tie-breaks and node numbering), without launches between them. The
// clusters' boxes stay in shared memory (279 -> 180 us from 2,048 clusters on, against reading them
// through L1 for every neighbour).
constexpr int kPlocSmallThreads = 1024;
constexpr size_t kPlocFinishShared = 4 * kPlocSmall * sizeof(float4);

__global__ void __launch_bounds__(kPlocSmallThreads)
    k_ploc_finish(uint32_t const *clus_in, uint32_t m, uint32_t base, float4 *blo, float4 *bhi, int2 *child,
                  uint32_t *out_nodes) {
    __shared__ uint32_t ca[kPlocSmall], cb[kPlocSmall];
    __shared__ int32_t nn[kPlocSmall];
    __shared__ uint32_t ms[kPlocSmall], ks[kPlocSmall];
    __shared__ uint32_t sh[32];
    constexpr int per = kPlocSmall / kPlocSmallThreads; // elements per thread in the scans
    extern __shared__ float4 boxes[];
    float4 *lo = boxes, *hi = boxes + kPlocSmall, *lo2 = hi + kPlocSmall, *hi2 = lo2 + kPlocSmall;
    for (uint32_t i = threadIdx.x; i < m; i += kPlocSmallThreads) {
        ca[i] = clus_in[i];
        lo[i] = blo[clus_in[i]];
        hi[i] = bhi[clus_in[i]];
    }
    __syncthreads();
    uint32_t *cur = ca, *nxt = cb;
    int rounds = 0;
    while (m > 1 && rounds++ < 1000000) {
        for (uint32_t i = threadIdx.x; i < m; i += kPlocSmallThreads) {
            float4 a0 = lo[i], a1 = hi[i];
            float best = INFINITY;
            int bj = -1;
            for (int d = -kPlocRadius; d <= kPlocRadius; d++) {
                int j = static_cast<int>(i) + d;
                if (d == 0 || j < 0 || j >= static_cast<int>(m))
                    continue;
                float area = union_area(a0, a1, lo[j], hi[j]);
                if (area < best) {
                    best = area;
                    bj = j;
                }
            }
            nn[i] = bj;
        }
        __syncthreads();
        // merge flags and their exclusive scans (each thread owns `per` consecutive clusters)
        uint32_t mf[per], kf[per], msum = 0, ksum = 0;
#pragma unroll
        for (int k = 0; k < per; k++) {
            uint32_t i = threadIdx.x * per + k;
            uint32_t merged = 0, keep = 0;
            if (i < m) {
                int32_t j = nn[i];
                bool mutual = j >= 0 && nn[j] == static_cast<int32_t>(i);
                merged = mutual && static_cast<int32_t>(i) < j;
                keep = !(mutual && static_cast<int32_t>(i) > j);
            }
            mf[k] = merged;
            kf[k] = keep;
            msum += merged;
            ksum += keep;
        }
        uint32_t mincl = block_inclusive<kPlocSmallThreads>(msum, sh);
        uint32_t mtotal = sh[31];
        __syncthreads();
        uint32_t kincl = block_inclusive<kPlocSmallThreads>(ksum, sh);
        uint32_t ktotal = sh[31];
        __syncthreads();
        uint32_t mrun = mincl - msum, krun = kincl - ksum;
#pragma unroll
        for (int k = 0; k < per; k++) {
            uint32_t i = threadIdx.x * per + k;
            if (i < m) {
                ms[i] = mf[k] ? mrun : 0xFFFFFFFFu;
                ks[i] = kf[k] ? krun : 0xFFFFFFFFu;
            }
            mrun += mf[k];
            krun += kf[k];
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < m; i += kPlocSmallThreads) {
            if (ks[i] == 0xFFFFFFFFu)
                continue;
            if (ms[i] != 0xFFFFFFFFu) {
                uint32_t node = base + ms[i];
                uint32_t a = cur[i], b = cur[nn[i]];
                child[node] = make_int2(static_cast<int>(a), static_cast<int>(b));
                float4 a0 = lo[i], a1 = hi[i], b0 = lo[nn[i]], b1 = hi[nn[i]];
                float4 u0 = make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), 0.0f);
                float4 u1 = make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), fmaxf(a1.z, b1.z), 0.0f);
                blo[node] = lo2[ks[i]] = u0;
                bhi[node] = hi2[ks[i]] = u1;
                nxt[ks[i]] = node;
            } else {
                nxt[ks[i]] = cur[i];
                lo2[ks[i]] = lo[i];
                hi2[ks[i]] = hi[i];
            }
        }
        __syncthreads();
        if (mtotal == 0)
            break; // no mutual pair (non-finite boxes): reported through the node count
        base += mtotal;
        m = ktotal;
        uint32_t *t = cur;
        cur = nxt;
        nxt = t;
        float4 *x = lo, *y = hi;
        lo = lo2, hi = hi2;
        lo2 = x, hi2 = y;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        out_nodes[0] = m == 1 ? base : 0u;
}

// ------------------------------------------------------------- collapse (bottom-up) ----

__global__ void k_tree_parents(int2 const *child, uint32_t n, uint32_t num_nodes, uint32_t *parent) {
    uint32_t node = n + blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= num_nodes)
        return;
    int2 c = child[node];
    parent[c.x] = node;
    parent[c.y] = node;
}

__device__ __forceinline__ float box_area(float4 lo, float4 hi) {
    float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// Triangle counts, SAH cost and leaf decisions; a thread per triangle walks up.
__global__ void k_collapse(uint32_t n, int2 const *child, uint32_t const *parent, float4 const *blo,
                           float4 const *bhi, uint32_t *counter, uint32_t *ntris, uint32_t *icount, float *cost,
                           uint8_t *leaf, uint32_t max_leaf, float tri_cost, float node_cost) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    ntris[i] = 1;
    icount[i] = 0;
    cost[i] = tri_cost * box_area(blo[i], bhi[i]);
    leaf[i] = 1;
    uint32_t node = parent[i];
    while (node != 0xFFFFFFFFu) {
        // the second child to arrive carries on: release of this thread's writes, acquire of the
        // sibling's
        uint32_t old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(&counter[node]) : "memory");
        if (old == 0)
            return;
        int2 c = child[node];
        uint32_t cnt = __ldcg(&ntris[c.x]) + __ldcg(&ntris[c.y]);
        float area = box_area(blo[node], bhi[node]);
        float inner = node_cost * area + __ldcg(&cost[c.x]) + __ldcg(&cost[c.y]);
        float as_leaf = tri_cost * area * static_cast<float>(cnt);
        bool make_leaf = cnt <= max_leaf && as_leaf <= inner;
        ntris[node] = cnt;
        icount[node] = make_leaf ? 0u : 1u + __ldcg(&icount[c.x]) + __ldcg(&icount[c.y]);
        cost[node] = make_leaf ? as_leaf : inner;
        leaf[node] = make_leaf;
        node = parent[node];
    }
}

// ------------------------------------------------------------ flatten (top-down) ----

struct FlatItem {
    uint32_t node, slot, tri_start;
    uint32_t pre; // interior nodes before this one in depth-first preorder
};

struct WideItem {
    uint32_t bn, wn; // binary node, wide node index
};

__global__ void k_flat_start(FlatItem *items, uint32_t *lvl, unsigned long long *leaf_stats, uint32_t root) {
    if (threadIdx.x < kLevels)
        lvl[threadIdx.x] = threadIdx.x == 0;
    if (threadIdx.x < 2)
        leaf_stats[threadIdx.x] = 0;
    if (threadIdx.x == 0)
        items[0] = FlatItem{root, 0, 0, 0};
}

// One level: lvl[level] frontier items (any order: an item carries its node slot and triangle start)
// into lvl[level + 1] items of the next. Grids are for any count, so the levels follow each other
// without the host.
__global__ void __launch_bounds__(kGB)
    k_flat_level(FlatItem const *items, FlatItem *next, uint32_t *lvl, uint32_t level, uint32_t n, int2 const *child,
                 uint8_t const *leaf, uint32_t const *ntris, uint32_t const *icount, float4 const *blo,
                 float4 const *bhi, uint32_t const *red, NodeHalf<float4> nlo, NodeHalf<float4> nhi,
                 uint32_t *leaf_start, unsigned long long *leaf_stats) {
    const uint32_t f = lvl[level], lane = threadIdx.x & 31u;
    float lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        lo[a] = key_float(red[a]);
        hi[a] = key_float(red[3 + a]);
    }
    const float eps = scene_eps(lo, hi);
    for (uint32_t i0 = blockIdx.x * kGB + (threadIdx.x & ~31u); i0 < f; i0 += gridDim.x * kGB) {
        const bool on = i0 + lane < f;
        FlatItem it{};
        bool is_leaf = false;
        if (on) {
            it = items[i0 + lane];
            is_leaf = leaf[it.node] != 0;
        }
        const uint32_t mi = __ballot_sync(~0u, on && !is_leaf), ml = __ballot_sync(~0u, is_leaf);
        uint32_t at = 0;
        if (lane == 0) {
            if (mi)
                at = atomicAdd(&lvl[level + 1], 2u * __popc(mi));
            if (ml) {
                atomicAdd(&leaf_stats[0], static_cast<unsigned long long>(__popc(ml)));
                atomicAdd(&leaf_stats[1], static_cast<unsigned long long>(__popc(ml)) * level);
            }
        }
        at = __shfl_sync(~0u, at, 0) + 2u * __popc(mi & ((1u << lane) - 1u));
        if (!on)
            continue;
        uint32_t link, count;
        if (is_leaf) {
            link = it.tri_start;
            count = ntris[it.node];
            leaf_start[it.node] = link;
        } else {
            // depth-first preorder slots, as the host builder lays nodes out: the k-th interior node in
            // preorder keeps its children at 1 + 2k and 2 + 2k
            link = 1 + 2 * it.pre;
            count = 0;
            int2 c = child[it.node];
            if (at + 1 < 2 * n) { // a malformed tree is refused before a write could leave the buffers
                next[at] = FlatItem{static_cast<uint32_t>(c.x), link, it.tri_start, it.pre + 1};
                next[at + 1] =
                    FlatItem{static_cast<uint32_t>(c.y), link + 1, it.tri_start + ntris[c.x], it.pre + 1 + icount[c.x]};
            }
        }
        if (it.slot >= 2 * n)
            continue;
        const float4 b0 = blo[it.node], b1 = bhi[it.node];
        nlo[it.slot] = make_float4(inflate_lo(b0.x, eps), inflate_lo(b0.y, eps), inflate_lo(b0.z, eps),
                                   __uint_as_float(link));
        nhi[it.slot] = make_float4(inflate_hi(b1.x, eps), inflate_hi(b1.y, eps), inflate_hi(b1.z, eps),
                                   __uint_as_float(count));
    }
}

// A thread per triangle, in Morton order: its leaf is the topmost ancestor that was made one, its place in
// the leaf the number of the leaf's triangles to its left (as parts of a level's walk over its leaves,
// one triangle after the other, the records took 110 us of the 1.3M-triangle scene's build, this 50).
__global__ void __launch_bounds__(kGB)
    k_leaf_tris(uint32_t n, uint32_t max_leaf, int2 const *child, uint32_t const *parent, uint8_t const *leaf,
                uint32_t const *ntris, uint32_t const *leaf_start, uint32_t const *order, uint4 const *tidx,
                float4 const *vpos, float4 *tri) {
    const uint32_t x = blockIdx.x * kGB + threadIdx.x;
    if (x >= n)
        return;
    const uint32_t t = order[x];
    const uint4 g = tidx[t];
    const float4 p0 = vpos[g.x], p1 = vpos[g.y], p2 = vpos[g.z];
    uint32_t top = x, count = 1, rank = 0, left = 0;
    for (uint32_t at = x, p = parent[x]; p != 0xFFFFFFFFu; p = parent[at]) {
        const uint32_t c = ntris[p];
        if (c > max_leaf)
            break;
        const int2 ch = child[p];
        if (static_cast<uint32_t>(ch.y) == at)
            left += ntris[ch.x];
        at = p;
        if (leaf[p]) {
            top = p;
            count = c;
            rank = left;
        }
    }
    const size_t r = leaf_start[top] + static_cast<size_t>(rank);
    if (r >= n)
        return; // (never: every leaf was reached)
    tri[3 * r] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(t));
    tri[3 * r + 1] = make_float4(p1.x - p0.x, p1.y - p0.y, p1.z - p0.z, rank + 1 == count ? 1.0f : 0.0f);
    tri[3 * r + 2] = make_float4(p2.x - p0.x, p2.y - p0.y, p2.z - p0.z, 0.0f);
}

inline uint32_t blocks(uint64_t n, int per) { return n ? static_cast<uint32_t>((n + per - 1) / per) : 1u; }

struct Carver {
    char *p;
    size_t used = 0;
    template <class T> T *take(size_t count) {
        size_t off = (used + 255) & ~size_t(255);
        used = off + count * sizeof(T);
        return p ? reinterpret_cast<T *>(p + off) : nullptr;
    }
};

// A level of the collapse: its frontier's length and the first node and triangle positions of the
// next level (level l reads state[l] and makes state[l + 1]).
struct WideState {
    uint32_t f, next_base, tri_running;
};
struct Scratch {
    uint32_t *red, *keys0, *vals0, *keys1, *vals1, *hist, *sums, *total;
    float4 *tlo, *thi, *blo, *bhi;
    int2 *child;
    uint32_t *clus0, *clus1, *parent, *counter, *ntris, *icount;
    uint64_t *scan, *tile_sums; // two counts per word (PLOC rounds, eight-wide levels)
    PlocState *ploc;            // the rounds' two states
    uint32_t *lvl;              // items per level of the flattening
    WideState *wstate;          // per level of the collapse
    int32_t *nn;
    float *cost;
    uint8_t *leaf;
    FlatItem *fa, *fb;
    unsigned long long *leaf_stats;
    WideItem *wa, *wb;   // eight-wide collapse: frontiers,
    uint32_t *wslots;    // 8 chosen children per frontier node,
    float4 *tri_tmp;     // triangle records in the wide order
};

Scratch carve(void *base, uint32_t n, size_t *bytes) {
    Carver c{static_cast<char *>(base)};
    Scratch s;
    size_t nodes = 2 * static_cast<size_t>(n);
    uint32_t sort_blocks = blocks(n, kSortTile);
    size_t hist_n = 256 * static_cast<size_t>(sort_blocks);
    size_t scan_max = std::max<size_t>(hist_n, n);
    s.red = c.take<uint32_t>(16);
    s.total = c.take<uint32_t>(4);
    s.keys0 = c.take<uint32_t>(n);
    s.vals0 = c.take<uint32_t>(n);
    s.keys1 = c.take<uint32_t>(n);
    s.vals1 = c.take<uint32_t>(n);
    s.hist = c.take<uint32_t>(hist_n);
    s.sums = c.take<uint32_t>(blocks(scan_max, kScanTile) + 1);
    s.tlo = c.take<float4>(n);
    s.thi = c.take<float4>(n);
    s.blo = c.take<float4>(nodes);
    s.bhi = c.take<float4>(nodes);
    s.child = c.take<int2>(nodes);
    s.clus0 = c.take<uint32_t>(n);
    s.clus1 = c.take<uint32_t>(n);
    s.scan = c.take<uint64_t>(n);
    s.tile_sums = c.take<uint64_t>(blocks(n, kScanTile) + 1);
    s.ploc = c.take<PlocState>(2);
    s.lvl = c.take<uint32_t>(kLevels);
    s.wstate = c.take<WideState>(kLevels);
    s.nn = c.take<int32_t>(n);
    s.parent = c.take<uint32_t>(nodes);
    s.counter = c.take<uint32_t>(nodes);
    s.ntris = c.take<uint32_t>(nodes);
    s.icount = c.take<uint32_t>(nodes);
    s.cost = c.take<float>(nodes);
    s.leaf = c.take<uint8_t>(nodes);
    s.fa = c.take<FlatItem>(nodes);
    s.fb = c.take<FlatItem>(nodes);
    s.leaf_stats = c.take<unsigned long long>(2);
    s.wa = c.take<WideItem>(n);
    s.wb = c.take<WideItem>(n);
    s.wslots = c.take<uint32_t>(8 * static_cast<size_t>(n));
    s.tri_tmp = c.take<float4>(3 * static_cast<size_t>(n));
    *bytes = c.used + 256;
    return s;
}

// Exclusive scan of d[0, n) in place; the total lands in *total (device).
void scan(uint32_t *d, uint32_t n, uint32_t *sums, uint32_t *total, cudaStream_t st) {
    uint32_t tiles = blocks(n, kScanTile);
    k_scan_tiles<<<tiles, 1024, 0, st>>>(d, n, sums);
    k_scan_sums<<<1, 1024, 0, st>>>(sums, tiles, total);
    k_scan_add<<<tiles, 1024, 0, st>>>(d, n, sums);
}

// ------------------------------------------------------------ eight-wide collapse ----
// The host collapse (bvh_wide.cpp) level by level: a thread per wide node opens the binary child
// with the largest surface area until eight children are collected, assigns octant slots with the
// same greedy cost and quantizes with the same arithmetic; scans give every node the child and
// triangle bases the host's breadth-first queue gives it, so the bytes equal the host's.

__device__ __forceinline__ float wide_area(float4 lo, float4 hi) {
    float d0 = hi.x - lo.x, d1 = hi.y - lo.y, d2 = hi.z - lo.z;
    if (!(d0 >= 0) || !(d1 >= 0) || !(d2 >= 0))
        return 0.0f;
    return 2.0f * (d0 * d1 + d0 * d2 + d1 * d2);
}

// Children of one wide node in slot order (binary node ids, kNone for an empty slot).
constexpr uint32_t kNone = 0xFFFFFFFFu;

__global__ void k_wide_start(WideItem *items, WideState *state) {
    items[0] = WideItem{0, 0};
    state[0] = WideState{1, 1, 0};
}

// Eight lanes per wide node, one child each (a thread per node with its children and costs in local
// memory took 731 us over the nine levels of the 1.3M-triangle scene, this 313): the child with the largest area is opened until there
// are eight (or none is interior), then children take octant slots greedily by the cost of the octant
// they lie in, the cheapest (child, slot) first. Ties: the lowest child, then the lowest slot.
__global__ void __launch_bounds__(kGB)
    k_wide_plan(WideState const *state, WideItem const *items, NodeHalf<const float4> nlo, NodeHalf<const float4> nhi,
                uint32_t *slots_out, uint64_t *counts) {
    const uint32_t f = state->f, lane = threadIdx.x & 31u, li = lane & 7u, g0 = lane & ~7u;
    for (uint32_t i0 = (blockIdx.x * kGB + (threadIdx.x & ~31u)) / 8; i0 < f; i0 += gridDim.x * (kGB / 8)) {
        const uint32_t i = i0 + lane / 8;
        const bool on = i < f;
        uint32_t id = kNone, n = 0, link = 0, cnt = 1;
        float4 lo = make_float4(0, 0, 0, 0), hi = lo;
        if (on) {
            const uint32_t bn = items[i].bn;
            lo = nlo[bn], hi = nhi[bn];
            const bool interior = __float_as_uint(hi.w) == 0;
            n = interior ? 2u : 1u; // a root that is a leaf is its own child
            id = li < n ? (interior ? __float_as_uint(lo.w) + li : bn) : kNone;
        }
        bool fetch = id != kNone;
        for (int step = 0; step < 7; step++) {
            if (fetch) {
                lo = nlo[id], hi = nhi[id];
                link = __float_as_uint(lo.w);
                cnt = __float_as_uint(hi.w);
            }
            // the interior child with the largest area, the lowest of equals
            float area = id != kNone && cnt == 0 ? wide_area(lo, hi) : -1.0f;
            uint32_t at = li;
            for (int k = 4; k > 0; k >>= 1) {
                float a2 = __shfl_xor_sync(~0u, area, k);
                uint32_t l2 = __shfl_xor_sync(~0u, at, k);
                if (a2 > area || (a2 == area && l2 < at)) {
                    area = a2;
                    at = l2;
                }
            }
            const bool open = on && n < 8 && n > 1 && area > -1.0f;
            const uint32_t l = __shfl_sync(~0u, link, g0 + at);
            fetch = open && (li == at || li == n);
            if (fetch)
                id = li == at ? l : l + 1;
            n += open;
        }
        // (seven rounds: six openings and the fetch of the last pair)
        const bool have = id != kNone;
        float ulo[3] = {INFINITY, INFINITY, INFINITY}, uhi[3] = {-INFINITY, -INFINITY, -INFINITY};
        const float blo[3] = {lo.x, lo.y, lo.z}, bhi[3] = {hi.x, hi.y, hi.z};
        float off[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (have) {
                ulo[a] = blo[a];
                uhi[a] = bhi[a];
            }
            for (int k = 4; k > 0; k >>= 1) {
                ulo[a] = fminf(ulo[a], __shfl_xor_sync(~0u, ulo[a], k));
                uhi[a] = fmaxf(uhi[a], __shfl_xor_sync(~0u, uhi[a], k));
            }
            off[a] = 0.5f * (blo[a] + bhi[a]) - 0.5f * (ulo[a] + uhi[a]);
        }
        float cost[8];
#pragma unroll
        for (int s = 0; s < 8; s++) {
            float c = 0;
#pragma unroll
            for (int a = 0; a < 3; a++)
                c += (s >> a & 1) ? -off[a] : off[a];
            cost[s] = c;
        }
        uint32_t open_slots = n <= 4 ? 0xFu : 0xFFu, slot = kNone;
        for (uint32_t k = 0; k < 8; k++) {
            const bool want = have && slot == kNone;
            float bc = INFINITY;
            uint32_t bs = 8;
#pragma unroll
            for (uint32_t s = 0; s < 8; s++)
                if (want && (open_slots >> s & 1u) && (bs == 8 || cost[s] < bc)) {
                    bc = cost[s] == cost[s] ? cost[s] : INFINITY; // boxes near the float range: any order will do
                    bs = s;
                }
            uint32_t at = want ? li : 8 + li;
            for (int o = 4; o > 0; o >>= 1) {
                float c2 = __shfl_xor_sync(~0u, bc, o);
                uint32_t a2 = __shfl_xor_sync(~0u, at, o);
                if (a2 < 8 && (at >= 8 || c2 < bc || (c2 == bc && a2 < at))) {
                    bc = c2;
                    at = a2;
                }
            }
            const uint32_t taken = __shfl_sync(~0u, bs, g0 + (at & 7u));
            if (at < 8) {
                if (li == at)
                    slot = taken;
                open_slots &= ~(1u << taken);
            }
        }
        uint32_t used = have ? 1u << slot : 0u, ni = have && cnt == 0, nt = have ? cnt : 0u;
        for (int k = 4; k > 0; k >>= 1) {
            used |= __shfl_xor_sync(~0u, used, k);
            ni += __shfl_xor_sync(~0u, ni, k);
            nt += __shfl_xor_sync(~0u, nt, k);
        }
        if (on) {
            if (have)
                slots_out[8 * static_cast<size_t>(i) + slot] = id;
            if (!(used >> li & 1u))
                slots_out[8 * static_cast<size_t>(i) + li] = kNone;
            if (li == 0)
                counts[i] = static_cast<uint64_t>(nt) << 32 | ni;
        }
    }
}

// Scan of a level's (triangles, interior children), tile by tile, then the tile totals.
__global__ void __launch_bounds__(1024) k_wide_tiles(WideState const *state, uint64_t *counts, uint64_t *sums) {
    __shared__ uint64_t sh[32];
    const uint32_t f = state->f;
    for (uint32_t tile = blockIdx.x; tile * kScanTile < f; tile += gridDim.x) {
        uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
        uint64_t v[kScanItems], t = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            v[k] = base + k < f ? counts[base + k] : 0;
            t += v[k];
        }
        uint64_t incl = block_inclusive<1024>(t, sh);
        uint64_t run = incl - t;
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            if (base + k < f)
                counts[base + k] = run;
            run += v[k];
        }
        if (threadIdx.x == 1023)
            sums[tile] = incl;
    }
}

__global__ void __launch_bounds__(1024) k_wide_sums(WideState const *state, WideState *next, uint64_t *sums) {
    __shared__ uint64_t sh[32];
    WideState s = *state;
    const uint64_t total = scan_totals(sums, s.f ? (s.f - 1) / kScanTile + 1 : 0, sh);
    if (threadIdx.x == 0)
        *next = WideState{static_cast<uint32_t>(total), s.next_base + static_cast<uint32_t>(total),
                          s.tri_running + static_cast<uint32_t>(total >> 32)};
}

// Eight lanes per wide node, a slot each: the slot's quantized planes (three lanes compute the grid's
// axes), its triangles' records and its place among the interior children; the
// record is put together in shared memory and written in one piece. (A thread per node with its slots
// in local memory took 274 us over the ten levels of the 1.3M-triangle scene, this 147.)
__global__ void __launch_bounds__(kGB)
    k_wide_emit(WideState const *state, WideItem const *items, uint32_t const *slots_in, uint64_t const *scan,
                uint64_t const *sums, uint32_t n, NodeHalf<const float4> nlo, NodeHalf<const float4> nhi,
                float4 const *tri_bin, float4 *tri_wide, double step_min, uint4 *wide, WideItem *next) {
    __shared__ __align__(16) uint32_t rec[kGB / 8][24];
    const WideState st = *state;
    const int e_min = wide_exponent(step_min);
    const uint32_t lane = threadIdx.x & 31u, s = lane & 7u, g0 = lane & ~7u;
    uint32_t *words = rec[threadIdx.x / 8];
    for (uint32_t i0 = (blockIdx.x * kGB + (threadIdx.x & ~31u)) / 8; i0 < st.f; i0 += gridDim.x * (kGB / 8)) {
        const uint32_t i = i0 + lane / 8;
        const bool on = i < st.f;
        const uint32_t c = on ? slots_in[8 * static_cast<size_t>(i) + s] : kNone;
        const bool have = c != kNone;
        float4 lo4 = make_float4(0, 0, 0, 0), hi4 = lo4;
        if (have)
            lo4 = nlo[c], hi4 = nhi[c];
        const uint32_t cnt = have ? __float_as_uint(hi4.w) : 0u;
        const bool inner = have && cnt == 0;
        // places among the node's interior children and triangles
        const uint32_t in_mask = __ballot_sync(~0u, inner) >> g0 & 0xFFu, leaf_mask = __ballot_sync(~0u, cnt != 0) >> g0 & 0xFFu;
        const uint32_t rank = __popc(in_mask & ((1u << s) - 1u));
        uint32_t toff = cnt;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t y = __shfl_up_sync(~0u, toff, o, 8);
            toff += static_cast<int>(s) >= o ? y : 0u;
        }
        toff -= cnt;
        const uint64_t at = on ? scan[i] + sums[i / kScanTile] : 0;
        const uint32_t int_at = static_cast<uint32_t>(at);
        const uint32_t child_base = st.next_base + int_at, tri_base = st.tri_running + static_cast<uint32_t>(at >> 32);
        if (inner && int_at + rank < n)
            next[int_at + rank] = WideItem{c, child_base + rank};
        const uint32_t first = __float_as_uint(lo4.w);
        for (uint32_t k = 0; k < cnt; k++) {
            const size_t src = 3 * static_cast<size_t>(first + k), dst = 3 * static_cast<size_t>(tri_base + toff + k);
            tri_wide[dst] = tri_bin[src];
            tri_wide[dst + 1] = tri_bin[src + 1];
            tri_wide[dst + 2] = tri_bin[src + 2];
        }
        // the grid: lane a < 3 of the node computes axis a
        const float lo[3] = {lo4.x, lo4.y, lo4.z}, hi[3] = {hi4.x, hi4.y, hi4.z};
        float ulo = 0.0f, uhi = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            float l = have ? lo[a] : INFINITY, h = have ? hi[a] : -INFINITY;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                const float l2 = __shfl_xor_sync(~0u, l, o), h2 = __shfl_xor_sync(~0u, h, o);
                l = l2 < l ? l2 : l;
                h = h < h2 ? h2 : h;
            }
            if (static_cast<int>(s) == a)
                ulo = l, uhi = h;
        }
        float org = 0.0f, inv = 0.0f;
        uint32_t ebyte = 0;
        if (on && s < 3)
            ebyte = wide_grid_axis(ulo, uhi, step_min, e_min, org, inv);
        if (s < 3)
            words[s] = __float_as_uint(org);
        uint32_t ebytes = s < 3 ? ebyte << (8 * s) : 0u;
        uint32_t meta = cnt ? toff << (8 * (s & 3)) : 0u, counts = cnt << (4 * s);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float oa = __shfl_sync(~0u, org, g0 + a), ia = __shfl_sync(~0u, inv, g0 + a);
            uint32_t ql = 0, qh = 0;
            if (have)
                wide_grid_planes(lo[a], hi[a], oa, ia, ql, qh);
            ql <<= 8 * (s & 3), qh <<= 8 * (s & 3);
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                ql |= __shfl_xor_sync(~0u, ql, o);
                qh |= __shfl_xor_sync(~0u, qh, o);
            }
            if ((s & 3u) == 0) {
                words[8 + 2 * a + s / 4] = ql;
                words[14 + 2 * a + s / 4] = qh;
            }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            counts |= __shfl_xor_sync(~0u, counts, o);
            ebytes |= __shfl_xor_sync(~0u, ebytes, o);
            if (o < 4)
                meta |= __shfl_xor_sync(~0u, meta, o);
        }
        if ((s & 3u) == 0)
            words[6 + s / 4] = meta;
        if (s == 0) {
            words[3] = ebytes | in_mask << 24;
            words[4] = child_base;
            words[5] = tri_base;
            words[20] = counts;
            words[21] = leaf_mask;
            words[22] = words[23] = 0;
        }
        __syncwarp();
        const uint32_t wn = on ? items[i].wn : 0;
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t w = __shfl_sync(~0u, wn, 8 * k);
            if (i0 + k < st.f && lane < 6)
                wide[6 * static_cast<size_t>(w) + lane] = reinterpret_cast<uint4 const *>(rec[threadIdx.x / 32 * 4 + k])[lane];
        }
        __syncwarp();
    }
}
} // namespace

size_t gpu_build_scratch_bytes(uint32_t num_tris) {
    size_t bytes = 0;
    carve(nullptr, num_tris, &bytes);
    return bytes;
}

cudaError_t gpu_build_sah_pairs(GpuBuildIn const &in, GpuBuildOut &out, cudaStream_t st) {
    uint32_t n = in.num_tris;
    out = GpuBuildOut{};
    if (n == 0)
        return cudaSuccess;
    size_t bytes = 0;
    Scratch s = carve(in.scratch, n, &bytes);
    uint32_t *host = static_cast<uint32_t *>(in.host_pinned); // 4 words of pinned host memory
    int grid_cap = 8 * in.num_sms;
    // 1. boxes, Morton codes, sort
    k_build_init<<<1, 32, 0, st>>>(s.red);
    k_prim_boxes<<<std::min<uint32_t>(blocks(n, kGB), grid_cap), kGB, 0, st>>>(in.tidx, in.vpos, n, s.tlo, s.thi, s.red);
    k_morton<<<blocks(n, kGB), kGB, 0, st>>>(s.tlo, s.thi, n, s.red, s.keys0, s.vals0);
    uint32_t sort_blocks = blocks(n, kSortTile);
    uint32_t *kin = s.keys0, *vin = s.vals0, *kout = s.keys1, *vout = s.vals1;
    for (int shift = 0; shift < 32; shift += 8) {
        k_sort_hist<<<sort_blocks, kGB, 0, st>>>(kin, n, shift, s.hist);
        scan(s.hist, 256 * sort_blocks, s.sums, s.total, st);
        k_sort_scatter<<<sort_blocks, kGB, 0, st>>>(kin, vin, kout, vout, n, shift, s.hist);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    uint32_t *order = vin; // sorted position -> triangle
    k_gather_leaves<<<blocks(n, kGB), kGB, 0, st>>>(order, s.tlo, s.thi, n, s.blo, s.bhi, s.clus0);
    // 2. PLOC rounds
    k_ploc_start<<<1, 1, 0, st>>>(s.ploc, n);
    auto *hs = static_cast<PlocState *>(in.host_pinned);
    PlocState now{n, n, 0, 0, 0};
    for (uint32_t r = 0; now.m > static_cast<uint32_t>(kPlocSmall);) {
        const uint32_t m0 = now.m, g = blocks(now.m, kGB), tiles = blocks(now.m, kScanTile);
        for (int k = 0; k < kPlocBatch; k++, r++) {
            PlocState *cur = s.ploc + (r & 1), *nxt = s.ploc + (r & 1 ^ 1);
            k_ploc_nn<<<g, kGB, 0, st>>>(cur, s.clus0, s.clus1, s.blo, s.bhi, s.nn);
            k_ploc_tiles<<<tiles, 1024, 0, st>>>(cur, s.nn, s.scan, s.tile_sums);
            k_ploc_sums<<<1, 1024, 0, st>>>(cur, nxt, s.tile_sums);
            k_ploc_apply<<<g, kGB, 0, st>>>(cur, s.clus0, s.clus1, s.nn, s.scan, s.tile_sums, s.blo, s.bhi, s.child);
        }
        cudaError_t e = cudaMemcpyAsync(hs, s.ploc + (r & 1), sizeof(PlocState), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e != cudaSuccess)
            return e;
        now = *hs;
        if (now.stuck || now.m >= m0)
            return cudaErrorUnknown; // no mutual pair (non-finite boxes): host build
    }
    uint32_t base = now.base;
    if (now.m > 1) { // the remaining rounds in one block
        cudaError_t e = cudaFuncSetAttribute(k_ploc_finish, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(kPlocFinishShared));
        if (e != cudaSuccess)
            return e;
        k_ploc_finish<<<1, kPlocSmallThreads, kPlocFinishShared, st>>>(now.cur ? s.clus1 : s.clus0, now.m, base, s.blo,
                                                                       s.bhi, s.child, s.total + 2);
        e = cudaMemcpyAsync(host, s.total + 2, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e != cudaSuccess)
            return e;
        if (host[0] == 0)
            return cudaErrorUnknown; // no mutual pair (non-finite boxes): host build
        base = host[0];
    }
    uint32_t num_nodes = base, root = num_nodes - 1;
    // 3. leaf collapse
    cudaMemsetAsync(s.parent, 0xFF, 4 * static_cast<size_t>(num_nodes), st);
    if (num_nodes > n)
        k_tree_parents<<<blocks(num_nodes - n, kGB), kGB, 0, st>>>(s.child, n, num_nodes, s.parent);
    cudaMemsetAsync(s.counter, 0, 4 * static_cast<size_t>(num_nodes), st);
    k_collapse<<<blocks(n, kGB), kGB, 0, st>>>(n, s.child, s.parent, s.blo, s.bhi, s.counter, s.ntris, s.icount, s.cost,
                                               s.leaf, in.max_leaf, in.tri_cost, in.node_cost);
    // 4. flatten level by level, one level more than the traversal stack allows
    uint32_t *leaf_start = reinterpret_cast<uint32_t *>(s.cost); // per node; the costs are done with
    k_flat_start<<<1, 64, 0, st>>>(s.fa, s.lvl, s.leaf_stats, root);
    const uint32_t levels = std::min<uint32_t>(in.max_depth, kLevels - 2);
    for (uint32_t l = 0; l < levels; l++) {
        const uint32_t g = static_cast<uint32_t>(std::min<uint64_t>(blocks(uint64_t(1) << std::min(l, 31u), kGB),
                                                                    std::min<uint32_t>(blocks(n, kGB), grid_cap)));
        k_flat_level<<<g, kGB, 0, st>>>(l & 1 ? s.fb : s.fa, l & 1 ? s.fa : s.fb, s.lvl, l, n, s.child, s.leaf, s.ntris,
                                        s.icount, s.blo, s.bhi, s.red, in.nlo, in.nhi, leaf_start, s.leaf_stats);
    }
    uint32_t lvl[kLevels], stats[4 + 6];
    cudaError_t e = cudaMemcpyAsync(lvl, s.lvl, sizeof(lvl), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(stats, s.leaf_stats, 16, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(stats + 4, s.red, 24, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return e;
    uint32_t slots = 0, depth = 0;
    for (; depth < levels && lvl[depth]; depth++) {
        if (lvl[depth] > n || slots + lvl[depth] > 2ull * n)
            return cudaErrorUnknown; // a malformed tree
        slots += lvl[depth];
    }
    if (depth == levels && lvl[depth]) { // deeper than the traversal stack: the host builds instead
        out.ok = false;
        return cudaSuccess;
    }
    // every leaf was reached: the triangle records
    k_leaf_tris<<<blocks(n, kGB), kGB, 0, st>>>(n, in.max_leaf, s.child, s.parent, s.leaf, s.ntris, leaf_start, order,
                                                in.tidx, in.vpos, in.tri);
    out.num_nodes = slots;
    unsigned long long leaves = 0, leaf_depth_sum = 0;
    host = stats + 2;
    std::memcpy(&leaf_depth_sum, stats + 2, 8);
    std::memcpy(&leaves, stats, 8);
    for (int a = 0; a < 3; a++) {
        uint32_t lo = host[2 + a], hi = host[5 + a];
        uint32_t ul = (lo & 0x80000000u) ? (lo & 0x7FFFFFFFu) : ~lo;
        uint32_t uh = (hi & 0x80000000u) ? (hi & 0x7FFFFFFFu) : ~hi;
        std::memcpy(&out.scene_lo[a], &ul, 4);
        std::memcpy(&out.scene_hi[a], &uh, 4);
    }
    out.num_leaves = static_cast<uint32_t>(leaves);
    out.max_depth = depth;
    out.avg_leaf_depth = leaves ? static_cast<double>(leaf_depth_sum) / static_cast<double>(leaves) : 0.0;
    out.ploc_rounds = now.rounds;
    out.ok = depth <= in.max_depth;
    return cudaGetLastError();
}

} // namespace e8g

namespace e8g {

cudaError_t gpu_collapse_wide(GpuWideIn const &in, GpuWideOut &out, cudaStream_t st) {
    uint32_t n = in.num_tris;
    out = GpuWideOut{};
    if (n == 0)
        return cudaSuccess;
    size_t bytes = 0;
    Scratch s = carve(in.scratch, n, &bytes);
    double step_min = wide_step_min(in.max_abs);
    k_wide_start<<<1, 1, 0, st>>>(s.wa, s.wstate);
    // the levels follow each other without the host, which looks after kWideBatch of them and then
    // for the few more that a deep tree has
    constexpr uint32_t kWideBatch = 10;
    const uint32_t levels = std::min<uint32_t>(in.max_depth, 31);
    const uint32_t cap = 8 * in.num_sms;
    WideState ws[kLevels];
    uint32_t depth = 0;
    for (uint32_t l = 0; l < levels;) {
        const uint32_t to = std::min<uint32_t>(l + kWideBatch, levels);
        for (; l < to; l++) {
            const uint64_t most = std::min<uint64_t>(n, uint64_t(1) << std::min<uint32_t>(3 * l, 32));
            WideItem *wa = l & 1 ? s.wb : s.wa, *wb = l & 1 ? s.wa : s.wb;
            WideState *cur = s.wstate + l;
            k_wide_plan<<<std::min<uint32_t>(blocks(8 * most, kGB), cap), kGB, 0, st>>>(cur, wa, in.nlo, in.nhi, s.wslots,
                                                                                       s.scan);
            k_wide_tiles<<<std::min<uint32_t>(blocks(most, kScanTile), cap), 1024, 0, st>>>(cur, s.scan, s.tile_sums);
            k_wide_sums<<<1, 1024, 0, st>>>(cur, cur + 1, s.tile_sums);
            k_wide_emit<<<std::min<uint32_t>(blocks(8 * most, kGB), cap), kGB, 0, st>>>(
                cur, wa, s.wslots, s.scan, s.tile_sums, n, in.nlo, in.nhi, in.tri, s.tri_tmp, step_min, in.wide, wb);
        }
        cudaError_t e = cudaMemcpyAsync(ws, s.wstate, sizeof(WideState) * (l + 1), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e != cudaSuccess)
            return e;
        for (; depth < l && ws[depth].f; depth++) {
            if (ws[depth].f > n || ws[depth].next_base > n + 1)
                return cudaErrorUnknown; // a malformed tree
            out.level_start[depth] = ws[depth].next_base - ws[depth].f;
        }
        if (ws[depth].f == 0)
            break;
    }
    if (ws[depth].f) {
        out.ok = false; // too deep for the eight-wide stack: keep the binary tree
        return cudaSuccess;
    }
    const uint32_t next_base = ws[depth].next_base;
    if (ws[depth].tri_running != n)
        return cudaErrorUnknown;
    // the triangle records move to the wide order only now that the collapse succeeded
    cudaError_t e = cudaMemcpyAsync(in.tri, s.tri_tmp, 48 * static_cast<size_t>(n), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess)
        return e;
    out.num_nodes = next_base;
    out.max_depth = depth;
    out.level_start[depth] = next_base;
    out.ok = true;
    return cudaGetLastError();
}

} // namespace e8g
