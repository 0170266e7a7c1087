// bvh_gpu.cu -- GPU build of the 8-wide (or 4-wide) quantised BVH.
//
// Binary hierarchy by parallel locally-ordered clustering (PLOC: Meister and
// Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
// Hierarchy Construction", IEEE TVCG 2018): triangles sorted by 63-bit
// Morton codes of their centroids start as clusters; every iteration each
// cluster finds, among the clusters within kRadius (3) places of it in
// Morton order, the one whose merged box has the least surface area; mutual
// nearest neighbours merge (the merged cluster keeps the left one's place),
// and the list is compacted.  Then the host build's collapse and encoding
// (bvh8.cpp) run level by level: each wide node takes the children the
// collapse chose, assigns them to slots by octant, and quantises their boxes
// outward on a power-of-two grid.  The collapse is
// the host build's SAH-optimal dynamic programme (Ylitie et al., HPG 2017),
// computed bottom-up on the device; it also picks the leaf slots (subtrees
// of at most 3 triangles).  Node and triangle layouts
// are the host build's, so the traversal kernels and every query result are
// unchanged; only the tree differs, and with it the nodes a ray visits.
//
// Triangle boxes get the host build's conservative margin (2^-15 of the
// largest coordinate magnitude, computed in FP64 and rounded outward).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <chrono>
#include <vector>

#include "crt_internal.h"

namespace crt {
namespace {

constexpr uint32_t kSlotTrisMax = 3;  // triangles a leaf slot holds (3-bit count)
constexpr float kTriCost = 0.5f;      // the collapse's cost model, as the host build's
constexpr int kBlock = 256;
// PLOC search radius (clusters on each side).  With the SAH-optimal
// collapse a small radius traces best (C3 / C2, Msamples/s at 64 spp:
// r2 877 / 386, r3 882 / 391, r4 866 / 394, r8 850 / 397, r16 827 / 389,
// r32 809 / 390; the host SAH tree: 888 / 375).
constexpr int kRadius = 3;

struct GBox {
    float lo[3], hi[3];
};

// Binary nodes: internal nodes at 0..n-2 (the root at 0, created last),
// triangle i of the sorted order at n-1+i.  `count` is the node's number of
// triangles; a leaf's `first` is its sorted position.
struct GNode {
    GBox box;
    int32_t left, right, parent;
    uint32_t first, count;
};

// Decisions of the SAH-optimal collapse for one binary node (as DpCollapse
// in bvh8.cpp): as one slot, a leaf slot or a wide node; as a wide node,
// the slots of its left child; with at most i slots, those of the left
// child (0: as with i - 1).
struct GDec {
    uint8_t leaf, wk;
    uint8_t split[9];
    uint8_t pad;
};

// One wide node: the binary node in each slot (-1: empty) and its bases.
struct GWide {
    int32_t child[8];
    uint32_t child_base, tri_base;
};

__device__ __forceinline__ uint32_t float_order(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float order_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}
__device__ __forceinline__ float half_area(const GBox& b) {
    const float dx = fmaxf(b.hi[0] - b.lo[0], 0.f), dy = fmaxf(b.hi[1] - b.lo[1], 0.f),
                dz = fmaxf(b.hi[2] - b.lo[2], 0.f);
    return dx * dy + dy * dz + dz * dx;
}
__device__ __forceinline__ void grow(GBox& a, const GBox& b) {
    for (int k = 0; k < 3; ++k) {
        a.lo[k] = fminf(a.lo[k], b.lo[k]);
        a.hi[k] = fmaxf(a.hi[k], b.hi[k]);
    }
}

// Largest coordinate magnitude, as order-preserving bits of a positive float.
__global__ void k_max_abs(const float* __restrict__ v1, const float* __restrict__ e1, const float* __restrict__ e2,
                          uint32_t n3, uint32_t* out) {
    float m = 0.f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        const float a = v1[i];
        m = fmaxf(m, fmaxf(fabsf(a), fmaxf(fabsf(a + e1[i]), fabsf(a + e2[i]))));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31u) == 0) atomicMax(out, __float_as_uint(m));
}

// Conservative triangle boxes and centroids exactly as the host build forms
// them (FP64 bounds minus / plus the margin, rounded outward to FP32), and
// the centroid bounds, reduced per block before the atomics (one set of six per
// triangle took 300 us of 2.17M triangles' 383 us here).
__global__ void k_tri_boxes(const float* __restrict__ v1, const float* __restrict__ e1, const float* __restrict__ e2,
                            uint32_t n, float margin, GBox* __restrict__ tbox, float* __restrict__ cent,
                            uint32_t* __restrict__ cbounds) {
    uint32_t lo6[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi6[3] = {0u, 0u, 0u};
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        GBox b;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double a = v1[3ull * t + k];
            const double bb = a + (double)e1[3ull * t + k];
            const double c = a + (double)e2[3ull * t + k];
            const double lo = fmin(a, fmin(bb, c)) - (double)margin, hi = fmax(a, fmax(bb, c)) + (double)margin;
            float flo = __double2float_rn(lo), fhi = __double2float_rn(hi);
            if ((double)flo > lo) flo = nextafterf(flo, -FLT_MAX);
            if ((double)fhi < hi) fhi = nextafterf(fhi, FLT_MAX);
            b.lo[k] = flo;
            b.hi[k] = fhi;
            const float cc = 0.5f * (flo + fhi);
            cent[3ull * t + k] = cc;
            lo6[k] = min(lo6[k], float_order(cc));
            hi6[k] = max(hi6[k], float_order(cc));
        }
        tbox[t] = b;
    }
    __shared__ uint32_t sh[6];
    if (threadIdx.x < 6) sh[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t l = __reduce_min_sync(0xFFFFFFFFu, lo6[k]), h = __reduce_max_sync(0xFFFFFFFFu, hi6[k]);
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(&sh[k], l);
            atomicMax(&sh[3 + k], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&cbounds[threadIdx.x], sh[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&cbounds[threadIdx.x], sh[threadIdx.x]);
}

// Spreads the low 21 bits of x to every third bit of a 63-bit code.
__device__ __forceinline__ uint64_t spread21(uint64_t x) {
    x &= 0x1FFFFFull;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// 63-bit Morton codes (21 bits per axis) of the centroids.
__global__ void k_morton(const float* __restrict__ cent, uint32_t n, const uint32_t* __restrict__ cbounds,
                         uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    // one scale for all axes (the centroid bounds' largest extent): Morton
    // cells are cubes, so a flat axis does not get the same weight in the
    // curve as the wide ones
    float lo[3];
    const float top = (float)((1u << 21) - 1u);
    float ext = 0.f;
    for (int k = 0; k < 3; ++k) {
        lo[k] = order_float(cbounds[k]);
        ext = fmaxf(ext, order_float(cbounds[3 + k]) - lo[k]);
    }
    const float sc = ext > 0.f ? top / ext : 0.f;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        uint64_t q[3];
        for (int k = 0; k < 3; ++k) {
            const float f = (cent[3ull * t + k] - lo[k]) * sc;
            q[k] = (uint64_t)fminf(fmaxf(f, 0.f), top);
        }
        keys[t] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
        vals[t] = t;
    }
}

__global__ void k_leaves(const GBox* __restrict__ tbox, const uint32_t* __restrict__ perm, int n,
                         GNode* __restrict__ nodes) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    GNode& lf = nodes[n - 1 + i];
    lf.box = tbox[perm[i]];
    lf.left = lf.right = lf.parent = -1;
    lf.first = (uint32_t)i;
    lf.count = 1;
}

// Clusters left and the next node id of one PLOC iteration.
struct PlocState {
    int32_t m, next_id;
};

// For cluster i of m (in Morton order; tile[k] is cluster t0 + k's box), the
// cluster j within kRadius places whose merged box has the least half area.
// Pairs are ordered by (area, |i - j|, min(i, j) odd, min(i, j)): a total order
// on unordered pairs, so the best pair overall is always mutual and every
// iteration merges; among equal boxes (2k, 2k + 1) pair up, so even a scene of
// identical triangles halves its clusters every iteration.
__device__ __forceinline__ int nearest(const GBox* tile, int t0, int i, int m) {
    const GBox bi = tile[i - t0];
    float best = FLT_MAX;
    int bj = -1, bdist = INT_MAX, bodd = 1, bmin = INT_MAX;
    const int j0 = max(0, i - kRadius), j1 = min(m - 1, i + kRadius);
    for (int j = j0; j <= j1; ++j) {
        if (j == i) continue;
        GBox u = bi;
        grow(u, tile[j - t0]);
        const float d = half_area(u);
        const int dist = abs(i - j), mn = min(i, j), odd = mn & 1;
        const bool better = d < best || (d == best && (dist < bdist || (dist == bdist && (odd < bodd || (odd == bodd && mn < bmin)))));
        if (better) {
            best = d;
            bj = j;
            bdist = dist;
            bodd = odd;
            bmin = mn;
        }
    }
    return bj;
}

// PLOC pairs: i and j pair if each is the other's nearest.  A block also finds the neighbours of the kRadius clusters on either side of
// its own, so it knows which of its clusters pair, writes pair[i] (j or -1) and
// counts its survivors (high word) and new nodes (low word).
__global__ void __launch_bounds__(kBlock) k_ploc_pairs(const int32_t* __restrict__ clusters,
                                                       const PlocState* __restrict__ state,
                                                       const GNode* __restrict__ nodes, int32_t* __restrict__ pair,
                                                       uint64_t* __restrict__ counts, int n, uint32_t* err) {
    constexpr int kTile = kBlock + 4 * kRadius, kNear = kBlock + 2 * kRadius;
    __shared__ GBox tile[kTile];
    __shared__ int near[kNear];
    const int m = state->m;
    const int b0 = (int)(blockIdx.x * kBlock);
    if (b0 >= m) return;   // the whole block
    const int t0 = b0 - 2 * kRadius;   // cluster of tile[0]
    for (int k = (int)threadIdx.x; k < kTile; k += kBlock) {
        const int i = t0 + k;
        if (i < 0 || i >= m) continue;
        const int32_t c = clusters[i];
        if (c < 0 || c > 2 * n - 2) {   // never expected; keeps the read in bounds
            atomicOr(err, 1u);
            tile[k] = GBox{{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        } else {
            tile[k] = nodes[c].box;
        }
    }
    __syncthreads();
    const int n0 = b0 - kRadius;       // cluster of near[0]
    for (int k = (int)threadIdx.x; k < kNear; k += kBlock) {
        const int i = n0 + k;
        int bj = -1;
        if (i >= 0 && i < m) {
            bj = nearest(tile, t0, i, m);
        }
        near[k] = bj;
    }
    __syncthreads();
    const int i = b0 + (int)threadIdx.x;
    bool survive = false, create = false;
    if (i < m) {
        const int j = near[i - n0];
        const bool mutual = j >= 0 && near[j - n0] == i;
        pair[i] = mutual ? j : -1;
        create = mutual && i < j;
        survive = !mutual || i < j;
    }
    const int ns = __syncthreads_count(survive), nc = __syncthreads_count(create);
    if (threadIdx.x == 0) counts[blockIdx.x] = ((uint64_t)ns << 32) | (uint64_t)nc;
}

// Exclusive sums of the block counts in place (one block), and the next
// iteration's state.
__global__ void __launch_bounds__(1024) k_ploc_scan(uint64_t* __restrict__ counts, const PlocState* __restrict__ state,
                                                    PlocState* __restrict__ next, uint32_t* err) {
    __shared__ uint64_t warp_sum[32];
    const int m = state->m, blocks = (m + kBlock - 1) / kBlock;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t carry = 0;
    for (int b0 = 0; b0 < blocks; b0 += 1024) {
        const int b = b0 + (int)threadIdx.x;
        const uint64_t v = b < blocks ? counts[b] : 0;
        uint64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint64_t w = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
                if ((int)lane >= o) w += y;
            }
            warp_sum[lane] = w;
        }
        __syncthreads();
        const uint64_t before = carry + (warp ? warp_sum[warp - 1] : 0) + x - v;
        if (b < blocks) counts[b] = before;
        carry += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const int32_t survivors = (int32_t)(carry >> 32), merges = (int32_t)(uint32_t)carry;
        if (survivors + merges != m || (m > 1 && merges == 0) || state->next_id + 1 < merges) atomicOr(err, 1u);
        next->m = survivors;
        next->next_id = state->next_id - merges;
    }
}

// Creates the merged nodes (ids counting down from next_id) and writes the
// compacted cluster list.
__global__ void __launch_bounds__(kBlock) k_ploc_merge(const int32_t* __restrict__ clusters,
                                                       const int32_t* __restrict__ pair,
                                                       const PlocState* __restrict__ state,
                                                       const uint64_t* __restrict__ counts, GNode* __restrict__ nodes,
                                                       int32_t* __restrict__ out, int n, uint32_t* err) {
    __shared__ uint32_t warp_s[kBlock / 32], warp_c[kBlock / 32];
    const int m = state->m;
    const int b0 = (int)(blockIdx.x * kBlock);
    if (b0 >= m) return;   // the whole block
    const int i = b0 + (int)threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const int j = i < m ? pair[i] : -1;
    const bool create = i < m && j > i, survive = i < m && (j < 0 || j > i);
    const uint32_t bs = __ballot_sync(0xFFFFFFFFu, survive), bc = __ballot_sync(0xFFFFFFFFu, create);
    if (lane == 0) {
        warp_s[warp] = __popc(bs);
        warp_c[warp] = __popc(bc);
    }
    __syncthreads();
    if (!survive) return;
    const uint64_t before = counts[blockIdx.x];
    uint32_t pos = (uint32_t)(before >> 32), made = (uint32_t)before;
    for (uint32_t w = 0; w < warp; ++w) {
        pos += warp_s[w];
        made += warp_c[w];
    }
    const uint32_t below = (1u << lane) - 1u;
    pos += __popc(bs & below);
    made += __popc(bc & below);
    int32_t id = clusters[i];
    if (create) {
        id = state->next_id - (int32_t)made;
        const int32_t l = clusters[i], r = j < m ? clusters[j] : -1;
        if (id < 0 || id > n - 2 || l < 0 || r < 0 || l > 2 * n - 2 || r > 2 * n - 2) {
            atomicOr(err, 1u);   // never expected; keeps every write in bounds
            return;
        }
        GNode nd;
        nd.box = nodes[l].box;
        grow(nd.box, nodes[r].box);
        nd.left = l;
        nd.right = r;
        nd.parent = -1;
        nd.first = 0;
        nd.count = nodes[l].count + nodes[r].count;
        nodes[id] = nd;
        nodes[l].parent = id;
        nodes[r].parent = id;
    }
    if (pos >= (uint32_t)m) {
        atomicOr(err, 1u);
        return;
    }
    out[pos] = id;
}

// The last iterations, from at most kPlocTail clusters to one, in one block: the
// same pairs, ids and order as the three kernels above, with the boxes in shared
// memory.  Those are latency: three dependent launches an iteration, and a host
// wait per kPerSync of them, for 22 of the 47 iterations of 2.17M triangles
// (scene creation 5.3 -> 5.1 ms; 102K triangles 2.18 -> 1.76 ms).
constexpr int kPlocTail = 1024;
__global__ void __launch_bounds__(kPlocTail) k_ploc_tail(const int32_t* __restrict__ clusters,
                                                         const PlocState* __restrict__ state,
                                                         PlocState* __restrict__ next, GNode* __restrict__ nodes,
                                                         int32_t* __restrict__ out, int n, uint32_t* err) {
    __shared__ GBox tile[kPlocTail];
    __shared__ int near[kPlocTail];
    __shared__ int32_t ids[kPlocTail];
    __shared__ uint32_t counts[kPlocTail], warp_s[kPlocTail / 32], warp_c[kPlocTail / 32];
    const int i = (int)threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    int m = min(state->m, kPlocTail);
    int32_t next_id = state->next_id;
    if (i < m) {
        int32_t c = clusters[i];
        if (c < 0 || c > 2 * n - 2) {   // never expected; keeps the accesses in bounds
            atomicOr(err, 1u);
            c = 0;
        }
        ids[i] = c;
        tile[i] = nodes[c].box;
        counts[i] = nodes[c].count;
    }
    __syncthreads();
    while (m > 1) {
        if (i < m) near[i] = nearest(tile, 0, i, m);
        __syncthreads();
        const int j = i < m ? near[i] : -1;
        const bool mutual = j >= 0 && near[j] == i;
        const bool create = mutual && i < j, survive = i < m && (!mutual || i < j);
        const uint32_t bs = __ballot_sync(0xFFFFFFFFu, survive), bc = __ballot_sync(0xFFFFFFFFu, create);
        if (lane == 0) {
            warp_s[warp] = __popc(bs);
            warp_c[warp] = __popc(bc);
        }
        __syncthreads();
        uint32_t pos = __popc(bs & ((1u << lane) - 1u)), made = __popc(bc & ((1u << lane) - 1u)), survivors = 0, merges = 0;
        for (uint32_t w = 0; w < (uint32_t)(m + 31) / 32; ++w) {
            if (w == warp) pos += survivors, made += merges;
            survivors += warp_s[w];
            merges += warp_c[w];
        }
        if (merges == 0 || next_id > n - 2 || next_id + 1 < (int32_t)merges) {   // the whole block; never expected
            if (i == 0) atomicOr(err, 1u);
            break;
        }
        GBox box;
        int32_t id = -1;
        uint32_t count = 0;
        if (survive) {
            id = ids[i];
            box = tile[i];
            count = counts[i];
        }
        if (create) {
            const int32_t l = id, r = ids[j];
            id = next_id - (int32_t)made;
            grow(box, tile[j]);
            count += counts[j];
            GNode nd;
            nd.box = box;
            nd.left = l;
            nd.right = r;
            nd.parent = -1;
            nd.first = 0;
            nd.count = count;
            nodes[id] = nd;
            nodes[l].parent = id;
            nodes[r].parent = id;
        }
        __syncthreads();
        if (survive) {
            ids[pos] = id;
            tile[pos] = box;
            counts[pos] = count;
        }
        m = (int)survivors;
        next_id -= (int32_t)merges;
        __syncthreads();
    }
    if (i < m) out[i] = ids[i];
    if (i == 0) *next = PlocState{m, next_id};
}

__global__ void k_ploc_init(int32_t* __restrict__ clusters, int n, PlocState* __restrict__ state) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) clusters[i] = n - 1 + i;   // every triangle is a cluster
    if (i == 0) *state = PlocState{n, n - 2};
}

// C(x, 1..W) of the collapse, from the children's costs.
template <int W>
__device__ __forceinline__ void dp_node(const GNode& nd, const float* L, const float* R, float* C, GDec& d) {
    const float A = half_area(nd.box);
    const float leafc = nd.count <= kSlotTrisMax ? kTriCost * A * (float)nd.count : FLT_MAX;
    float D[W + 1];
    int K[W + 1];
#pragma unroll
    for (int i = 2; i <= W; ++i) {
        D[i] = FLT_MAX;
        K[i] = 1;
#pragma unroll
        for (int k = 1; k < i; ++k) {
            const float c = L[k - 1] + R[i - k - 1];
            if (c < D[i]) {
                D[i] = c;
                K[i] = k;
            }
        }
    }
    const float wide = A + D[W];
    d.leaf = leafc <= wide;
    d.wk = (uint8_t)K[W];
    C[0] = d.leaf ? leafc : wide;
    d.split[0] = d.split[1] = 0;
#pragma unroll
    for (int i = 2; i <= W; ++i) {
        if (D[i] < C[i - 2]) {
            C[i - 1] = D[i];
            d.split[i] = (uint8_t)K[i];
        } else {
            C[i - 1] = C[i - 2];
            d.split[i] = 0;
        }
    }
#pragma unroll
    for (int i = W + 1; i < 9; ++i) d.split[i] = 0;
    d.pad = 0;
}

// Bottom-up from the leaves: the second child to finish computes its parent.
// cost[8 * node + i - 1] is C(node, i).  (Loops over W known at compile time
// keep the tables in registers: with the leaves 0.91 -> 0.36 ms of 2.17M
// triangles.)
template <int W>
__global__ void k_dp_up(int n, const GNode* __restrict__ nodes, float* cost, GDec* __restrict__ dec, uint32_t* flags,
                        uint32_t* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int leaf = n - 1 + i;
    {
        const float c = kTriCost * half_area(nodes[leaf].box) * (float)nodes[leaf].count;
        float4* to = reinterpret_cast<float4*>(cost + 8ull * leaf);
        __stcg(to, make_float4(c, c, c, c));
        if (W > 4) __stcg(to + 1, make_float4(c, c, c, c));
        GDec d;
        memset(&d, 0, sizeof(d));
        d.leaf = 1;
        dec[leaf] = d;
    }
    int p = nodes[leaf].parent;
    for (int climbed = 0; p >= 0; ++climbed) {
        if (p > n - 2 || climbed >= n) {   // never expected; ends the climb
            atomicOr(err, 8u);
            return;
        }
        __threadfence();
        if (atomicAdd(&flags[p], 1u) == 0) return;   // the sibling subtree is not done yet
        __threadfence();
        const GNode nd = nodes[p];
        if (nd.left < 0 || nd.right < 0 || nd.left > 2 * n - 2 || nd.right > 2 * n - 2) {
            atomicOr(err, 8u);
            return;
        }
        float L[8], R[8], C[8];
        const float4* pl = reinterpret_cast<const float4*>(cost + 8ull * nd.left);
        const float4* pr = reinterpret_cast<const float4*>(cost + 8ull * nd.right);
#pragma unroll
        for (int h = 0; h < W / 4; ++h) {
            const float4 a = __ldcg(pl + h), b = __ldcg(pr + h);
            L[4 * h] = a.x; L[4 * h + 1] = a.y; L[4 * h + 2] = a.z; L[4 * h + 3] = a.w;
            R[4 * h] = b.x; R[4 * h + 1] = b.y; R[4 * h + 2] = b.z; R[4 * h + 3] = b.w;
        }
        GDec d;
        dp_node<W>(nd, L, R, C, d);
        float4* to = reinterpret_cast<float4*>(cost + 8ull * p);
#pragma unroll
        for (int h = 0; h < W / 4; ++h) __stcg(to + h, make_float4(C[4 * h], C[4 * h + 1], C[4 * h + 2], C[4 * h + 3]));
        dec[p] = d;
        p = nd.parent;
    }
}

__device__ __forceinline__ bool wide_slot(const GDec* dec, int32_t x) { return dec[x].leaf == 0; }

// One wide node per 8 lanes: the collapse's children, slots by octant.  The
// first lane expands the decisions; then lane c holds child c.  (One thread per
// node kept children and slots in local memory: 0.55 -> 0.32 ms over the levels of
// 2.17M triangles, and 0.86 -> 0.23 ms for k_emit, which now also runs once.)
__global__ void __launch_bounds__(kBlock) k_choose(const int32_t* __restrict__ front, uint32_t F,
                                                   const GNode* __restrict__ nodes, const GDec* __restrict__ dec,
                                                   int max_children, GWide* __restrict__ recs,
                                                   uint64_t* __restrict__ counts, int n, uint32_t* err) {
    __shared__ int32_t kids[kBlock];
    const uint32_t f = (uint32_t)(((uint64_t)blockIdx.x * kBlock + threadIdx.x) >> 3);
    const uint32_t lane = threadIdx.x & 7u, group = threadIdx.x & ~7u;
    const uint32_t mask = 0xFFu << (threadIdx.x & 24u);
    if (f >= F) return;   // whole groups of 8
    const int32_t x = front[f];
    int nch = 0;
    if (lane == 0) {
        int32_t* ch = kids + group;
        if (x < 0 || x > 2 * n - 2) {
            atomicOr(err, 16u);
        } else if (!wide_slot(dec, x)) {
            ch[nch++] = x;                        // a root of at most 3 triangles
        } else {
            // expand (node, slots) pairs left to right, as DpCollapse::expand
            int32_t sn[16];
            int sb[16];
            int sp = 0;
            sn[sp] = nodes[x].right;
            sb[sp++] = max_children - dec[x].wk;
            sn[sp] = nodes[x].left;
            sb[sp++] = dec[x].wk;
            while (sp > 0) {
                const int32_t y = sn[--sp];
                int i = sb[sp];
                if (y < 0 || y > 2 * n - 2 || i < 1 || i > max_children) { atomicOr(err, 16u); break; }
                while (i > 1 && dec[y].split[i] == 0) --i;
                if (i == 1) {
                    if (nch < max_children) ch[nch++] = y;
                    else { atomicOr(err, 16u); break; }
                } else {
                    const int k = dec[y].split[i];
                    if (sp + 2 > 16 || k < 1 || k >= i) { atomicOr(err, 16u); break; }
                    sn[sp] = nodes[y].right;
                    sb[sp++] = i - k;
                    sn[sp] = nodes[y].left;
                    sb[sp++] = k;
                }
            }
        }
    }
    nch = __shfl_sync(mask, nch, 0, 8);
    __syncwarp(mask);
    const bool used = (int)lane < nch;
    const int32_t c = used ? kids[threadIdx.x] : -1;
    GBox cb;
    for (int k = 0; k < 3; ++k) { cb.lo[k] = FLT_MAX; cb.hi[k] = -FLT_MAX; }
    uint32_t tris = 0;
    bool wide = false;
    if (used) {
        cb = nodes[c].box;
        wide = wide_slot(dec, c);
        tris = wide ? 0u : nodes[c].count;
    }
    float dd[3];
    for (int k = 0; k < 3; ++k) {
        float lo = cb.lo[k], hi = cb.hi[k];
        for (int o = 1; o < 8; o <<= 1) {
            lo = fminf(lo, __shfl_xor_sync(mask, lo, o, 8));
            hi = fmaxf(hi, __shfl_xor_sync(mask, hi, o, 8));
        }
        dd[k] = 0.5f * (cb.lo[k] + cb.hi[k]) - 0.5f * (lo + hi);
    }
    // greedy: the best (child, free slot) pair each round; ties to the lowest
    // child, then the lowest slot
    uint32_t taken = 0;
    int slot = -1;
    for (int round = 0; round < nch; ++round) {
        float best = -FLT_MAX;
        int bs = -1;
        if (used && slot < 0)
            for (int s = 0; s < 8; ++s) {
                if ((taken >> s) & 1u) continue;
                const float sc = ((s & 1) ? dd[0] : -dd[0]) + ((s & 2) ? dd[1] : -dd[1]) + ((s & 4) ? dd[2] : -dd[2]);
                if (sc > best || bs < 0) { best = sc; bs = s; }
            }
        float top = bs < 0 ? -FLT_MAX : best;
        int who = bs < 0 ? 8 : (int)lane;
        for (int o = 1; o < 8; o <<= 1) {
            const float t = __shfl_xor_sync(mask, top, o, 8);
            const int w = __shfl_xor_sync(mask, who, o, 8);
            if (w < 8 && (who == 8 || t > top || (t == top && w < who))) { top = t; who = w; }
        }
        const int s = __shfl_sync(mask, bs, who & 7, 8);
        taken |= 1u << (s & 7);
        if ((int)lane == who) slot = s;
    }
    recs[f].child[lane] = -1;
    __syncwarp(mask);
    if (used && slot >= 0) recs[f].child[slot] = c;
    uint64_t both = ((uint64_t)(wide ? 1u : 0u) << 32) | tris;
    for (int o = 1; o < 8; o <<= 1) both += __shfl_xor_sync(mask, both, o, 8);
    if (lane == 0) counts[f] = both;
}

// The next level's frontier, in slot order, and the level's child and triangle
// bases.
__global__ void __launch_bounds__(kBlock) k_front(GWide* __restrict__ recs, uint32_t F, uint32_t next_base,
                                                  uint32_t tri_level_base, const uint64_t* __restrict__ offsets,
                                                  const GDec* __restrict__ dec, int32_t* __restrict__ next_front,
                                                  uint32_t cap_nodes, uint32_t* err) {
    const uint32_t f = (uint32_t)(((uint64_t)blockIdx.x * kBlock + threadIdx.x) >> 3);
    const uint32_t lane = threadIdx.x & 7u;
    if (f >= F) return;   // whole groups of 8
    const uint32_t shift = threadIdx.x & 24u, mask = 0xFFu << shift;
    const int32_t c = recs[f].child[lane];
    const bool wide = c >= 0 && wide_slot(dec, c);
    const uint32_t w = (__ballot_sync(mask, wide) >> shift) & 0xFFu;
    const uint64_t off = offsets[f];
    const uint32_t k = (uint32_t)(off >> 32) + __popc(w & ((1u << lane) - 1u));
    if (wide) {
        if (next_base + k < cap_nodes) next_front[k] = c;
        else atomicOr(err, 2u);
    }
    if (lane == 0) {
        recs[f].child_base = next_base + (uint32_t)(off >> 32);
        recs[f].tri_base = tri_level_base + (uint32_t)off;
    }
}

// Encodes the wide nodes (both device encodings) and writes the triangle
// records of the leaf slots: 8 lanes per node, lane s for slot s.
__global__ void __launch_bounds__(kBlock) k_emit(const GWide* __restrict__ recs, uint32_t N,
                                                 const GNode* __restrict__ nodes, const GDec* __restrict__ dec,
                                                 const uint32_t* __restrict__ perm, const float* __restrict__ v1,
                                                 const float* __restrict__ e1, const float* __restrict__ e2,
                                                 DevNodeQ16* __restrict__ out, Bvh8FloatNode* __restrict__ fout,
                                                 DevTriA* __restrict__ tris_a, DevTriB* __restrict__ tris_b,
                                                 uint32_t n_tris, uint32_t* err) {
    const uint32_t f = (uint32_t)(((uint64_t)blockIdx.x * kBlock + threadIdx.x) >> 3);
    const uint32_t s = threadIdx.x & 7u;
    if (f >= N) return;   // whole groups of 8
    const uint32_t mask = 0xFFu << (threadIdx.x & 24u);
    const int32_t c = recs[f].child[s];
    const uint32_t child_base = recs[f].child_base, tri_base = recs[f].tri_base;
    GBox cb;
    for (int k = 0; k < 3; ++k) { cb.lo[k] = FLT_MAX; cb.hi[k] = -FLT_MAX; }
    uint32_t bits = 0, count = 0;
    if (c >= 0) {
        cb = nodes[c].box;
        if (wide_slot(dec, c)) bits = 1u << s;
        else {
            count = min(nodes[c].count, kSlotTrisMax);
            bits = ((1u << count) - 1u) << (8 + 3 * s);
        }
    }
    const uint32_t slots = __reduce_or_sync(mask, bits);
    float p[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float lo = cb.lo[k];
        for (int o = 1; o < 8; o <<= 1) lo = fminf(lo, __shfl_xor_sync(mask, lo, o, 8));
        p[k] = lo;
        fout[f].planes[k][0][s] = cb.lo[k];
        fout[f].planes[k][1][s] = cb.hi[k];
        // a word holds slots s and s + 4; an empty slot's planes are inverted
        uint32_t l = 0x7F7Fu, h = 0xFF7Fu;
        if (c >= 0) {
            l = plane16((double)cb.lo[k] - (double)lo, false, s >= 4);
            h = plane16((double)cb.hi[k] - (double)lo, true, s >= 4);
        }
        const uint32_t l4 = __shfl_xor_sync(mask, l, 4, 8), h4 = __shfl_xor_sync(mask, h, 4, 8);
        if (s < 4) {
            out[f].planes[k][0][s] = l | (l4 << 16);
            out[f].planes[k][1][s] = h | (h4 << 16);
        }
    }
    if (s == 0) {
        out[f].px = p[0];
        out[f].py = p[1];
        out[f].pz = p[2];
        out[f].child_base = fout[f].child_base = child_base;
        out[f].tri_base = fout[f].tri_base = tri_base;
        out[f].slots = fout[f].slots = slots;
        out[f].pad[0] = out[f].pad[1] = fout[f].pad = 0;
    }
    out[f].pad2[s] = 0;
    if (!count) return;
    // the subtree's triangles, left to right (at most kSlotTrisMax)
    uint32_t at = tri_base + __popc((slots >> 8) & ((1u << (3 * s)) - 1u)), found = 0;
    int32_t stack[2 * kSlotTrisMax];
    int sp = 0;
    stack[sp++] = c;
    while (sp > 0) {
        const int32_t x = stack[--sp];
        if (x < 0 || x > 2 * (int32_t)n_tris - 2) { atomicOr(err, 4u); break; }
        const GNode& g = nodes[x];
        if (g.left >= 0) {
            if (sp + 2 > 2 * (int)kSlotTrisMax) { atomicOr(err, 4u); break; }
            stack[sp++] = g.right;
            stack[sp++] = g.left;
            continue;
        }
        if (found == count || at >= n_tris) { atomicOr(err, 4u); break; }
        const uint32_t t = perm[g.first];
        tris_a[at] = DevTriA{{v1[3ull * t], v1[3ull * t + 1], v1[3ull * t + 2]}, t,
                             {e1[3ull * t], e1[3ull * t + 1], e1[3ull * t + 2]}, e2[3ull * t]};
        tris_b[at] = DevTriB{e2[3ull * t + 1], e2[3ull * t + 2]};
        ++at;
        ++found;
    }
    if (found != count) atomicOr(err, 4u);
}

uint32_t blocks(uint64_t n) { return (uint32_t)std::max<uint64_t>(1, (n + kBlock - 1) / kBlock); }

// Where a build's temporaries lie in its scratch.  The first part serves in
// turn the boxes and sort keys, the collapse's costs, and the collapse's levels.
struct Scratch {
    size_t sort_bytes = 0, scan_bytes = 0;
    size_t tbox, cent, keys, vals, keys2, sort, cost, recs, cnt, off, fa, fb, scan;
    size_t perm, nodes, ca, cb, pair, counts, dec, flags, small, bytes;

    cudaError_t init(uint32_t n) {
        cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                                        (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0, 63);
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr, (int)n + 1);
        if (e != cudaSuccess) return e;
        const size_t n1 = n, nn2 = 2 * n1 - 1;
        Arena mem;
        tbox = mem.take(n1 * sizeof(GBox)), cent = mem.take(n1 * 12), keys = mem.take(n1 * 8), vals = mem.take(n1 * 4);
        keys2 = mem.take(n1 * 8), sort = mem.take(sort_bytes);
        size_t end = mem.at;
        mem.at = 0;
        cost = mem.take(nn2 * 8 * sizeof(float));
        end = std::max(end, mem.at);
        mem.at = 0;
        recs = mem.take(n1 * sizeof(GWide)), cnt = mem.take((n1 + 1) * 8), off = mem.take((n1 + 1) * 8);
        fa = mem.take(n1 * 4), fb = mem.take(n1 * 4), scan = mem.take(scan_bytes);
        mem.at = std::max(end, mem.at);
        perm = mem.take(n1 * 4), nodes = mem.take(nn2 * sizeof(GNode)), ca = mem.take(n1 * 4), cb = mem.take(n1 * 4);
        pair = mem.take(n1 * 4), counts = mem.take((n1 / kBlock + 1) * 8), dec = mem.take(nn2 * sizeof(GDec));
        flags = mem.take(n1 * 4), small = mem.take(64);
        bytes = mem.at;
        return cudaSuccess;
    }
};

}  // namespace

size_t bvh_gpu_scratch(uint32_t n) {
    Scratch L;
    if (n == 0 || n >= (1u << 30)) return 0;   // build_bvh_gpu refuses these
    return L.init(n) == cudaSuccess ? L.bytes : 0;
}

// Builds the BVH of n triangles (device arrays v1/e1/e2, [n][3]) into nodes,
// fnodes and tris (device, allocated here; tris holds n DevTriA, then n
// DevTriB); fills max_depth and the node count.  scratch: bvh_gpu_scratch(n)
// bytes, 256-byte aligned.  Returns CRT_OK or an error with its message set.
int build_bvh_gpu(const float* d_v1, const float* d_e1, const float* d_e2, uint32_t n, uint32_t max_levels,
                  int max_children, void* scratch, DevBuf& nodes_out, DevBuf& fnodes_out, DevBuf& tris_out, uint32_t* num_nodes,
                  uint32_t* max_depth, bool* fnodes_ok, cudaStream_t s) {
    if (n == 0) return set_error(CRT_ERR_INVALID, "scene has no triangles");
    if (n >= (1u << 30)) return set_error(CRT_ERR_LIMIT, "GPU BVH build: at most 2^30 triangles");
    const int ni = (int)n;
    const size_t n1 = n, nn2 = 2 * n1 - 1;
    Scratch L;
    CRT_CUDA(L.init(n));
    char* base = static_cast<char*>(scratch);
    uint32_t* err = reinterpret_cast<uint32_t*>(base + L.small);       // word 0: error bits, 1: largest magnitude
    uint32_t* cbounds = err + 2;                                       // words 2-7: centroid bounds
    PlocState* ploc = reinterpret_cast<PlocState*>(base + L.small + 32);
    const uint32_t init[8] = {0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    CRT_CUDA(cudaMemcpyAsync(err, init, sizeof(init), cudaMemcpyHostToDevice, s));
    k_max_abs<<<blocks(3ull * n) < 1024 ? blocks(3ull * n) : 1024, kBlock, 0, s>>>(d_v1, d_e1, d_e2, 3 * n, err + 1);
    uint32_t mb = 0;
    CRT_CUDA(cudaMemcpyAsync(&mb, err + 1, 4, cudaMemcpyDeviceToHost, s));
    CRT_CUDA(cudaStreamSynchronize(s));
    float maxabs;
    std::memcpy(&maxabs, &mb, 4);
    const float margin = (float)std::ldexp(std::max(1.0, (double)maxabs), -15);

    GBox* tbox = reinterpret_cast<GBox*>(base + L.tbox);
    float* cent = reinterpret_cast<float*>(base + L.cent);
    uint64_t* keys = reinterpret_cast<uint64_t*>(base + L.keys);
    uint64_t* keys2 = reinterpret_cast<uint64_t*>(base + L.keys2);
    uint32_t* vals = reinterpret_cast<uint32_t*>(base + L.vals);
    uint32_t* perm = reinterpret_cast<uint32_t*>(base + L.perm);
    k_tri_boxes<<<std::min<uint32_t>(blocks(n), 1216), kBlock, 0, s>>>(d_v1, d_e1, d_e2, n, margin, tbox, cent, cbounds);
    k_morton<<<std::min<uint32_t>(blocks(n), 4096), kBlock, 0, s>>>(cent, n, cbounds, keys, vals);
    CRT_CUDA(cub::DeviceRadixSort::SortPairs(base + L.sort, L.sort_bytes, keys, keys2, vals, perm, ni, 0, 63, s));
    GNode* gn = reinterpret_cast<GNode*>(base + L.nodes);
    k_leaves<<<blocks(n), kBlock, 0, s>>>(tbox, perm, ni, gn);
    int32_t root = ni - 1;   // a lone triangle is its own root
    if (n > 1) {
        // PLOC iterations over the cluster list (Morton order), ping-ponged.
        // The list's length stays on the device; the host reads it after every
        // few iterations, to shrink the grid and to end.  (Neighbours, flags, a
        // library scan, the merge and a host read each iteration: 2.6 ms of 2.17M
        // triangles' build; three kernels and a read every fourth: 1.1.)
        constexpr int kPerSync = 4;
        int32_t* cur = reinterpret_cast<int32_t*>(base + L.ca);
        int32_t* nxt = reinterpret_cast<int32_t*>(base + L.cb);
        int32_t* pair = reinterpret_cast<int32_t*>(base + L.pair);
        uint64_t* counts = reinterpret_cast<uint64_t*>(base + L.counts);
        k_ploc_init<<<blocks(n), kBlock, 0, s>>>(cur, ni, ploc);
        PlocState at{ni, ni - 2};
        for (uint32_t iter = 0; at.m > 1;) {
            const int32_t before = at.m;
            if (before <= kPlocTail) {
                k_ploc_tail<<<1, kPlocTail, 0, s>>>(cur, ploc + (iter & 1u), ploc + ((iter + 1u) & 1u), gn, nxt, ni, err);
                std::swap(cur, nxt);
                ++iter;
            } else {
                for (int k = 0; k < kPerSync; ++k, ++iter) {
                    const PlocState* st = ploc + (iter & 1u);
                    k_ploc_pairs<<<blocks(before), kBlock, 0, s>>>(cur, st, gn, pair, counts, ni, err);
                    k_ploc_scan<<<1, 1024, 0, s>>>(counts, st, ploc + ((iter + 1u) & 1u), err);
                    k_ploc_merge<<<blocks(before), kBlock, 0, s>>>(cur, pair, st, counts, gn, nxt, ni, err);
                    std::swap(cur, nxt);
                }
            }
            uint32_t e = 0;
            CRT_CUDA(cudaMemcpyAsync(&at, ploc + (iter & 1u), sizeof(at), cudaMemcpyDeviceToHost, s));
            CRT_CUDA(cudaMemcpyAsync(&root, cur, 4, cudaMemcpyDeviceToHost, s));   // with one cluster left, the root
            CRT_CUDA(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, s));
            CRT_CUDA(cudaStreamSynchronize(s));
            if (e || at.m < 1 || at.m >= before)
                return set_error(CRT_ERR_CUDA, "GPU BVH build: inconsistent clustering step");
        }
        if (root != 0 || at.next_id != -1) return set_error(CRT_ERR_CUDA, "GPU BVH build: clustering left no single root");
    }
    // the collapse's costs and decisions, bottom-up
    float* cost = reinterpret_cast<float*>(base + L.cost);
    GDec* dec = reinterpret_cast<GDec*>(base + L.dec);
    uint32_t* flags = reinterpret_cast<uint32_t*>(base + L.flags);
    CRT_CUDA(cudaMemsetAsync(flags, 0, n1 * 4, s));
    (max_children == 4 ? k_dp_up<4> : k_dp_up<8>)<<<blocks(n), kBlock, 0, s>>>(ni, gn, cost, dec, flags, err);
    CRT_CUDA(cudaGetLastError());
    {   // the collapse follows child links: stop here if any were not set
        uint32_t e = 0;
        CRT_CUDA(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, s));
        CRT_CUDA(cudaStreamSynchronize(s));
        if (e) return set_error(CRT_ERR_CUDA, "GPU BVH build: inconsistent hierarchy (" + std::to_string(e) + ")");
    }

    // ---- collapse level by level, then encode all nodes at once ------------
    const uint32_t cap_nodes = n;   // a wide node holds >= 1 triangle of its own subtree
    GWide* recs = reinterpret_cast<GWide*>(base + L.recs);
    uint64_t* cnt = reinterpret_cast<uint64_t*>(base + L.cnt);
    uint64_t* off = reinterpret_cast<uint64_t*>(base + L.off);
    int32_t* cur = reinterpret_cast<int32_t*>(base + L.fa);
    int32_t* nxt = reinterpret_cast<int32_t*>(base + L.fb);
    CRT_CUDA(cudaMemcpyAsync(cur, &root, 4, cudaMemcpyHostToDevice, s));
    uint32_t F = 1, level_base = 0, tri_base = 0, depth = 0;
    while (F > 0) {
        if (++depth > max_levels) return set_error(CRT_ERR_LIMIT, "BVH deeper than the traversal stack allows");
        k_choose<<<blocks(8ull * F), kBlock, 0, s>>>(cur, F, gn, dec, max_children, recs + level_base, cnt, ni, err);
        // exclusive sums over F + 1 entries: the last is the level's totals
        CRT_CUDA(cudaMemsetAsync(cnt + F, 0, 8, s));
        CRT_CUDA(cub::DeviceScan::ExclusiveSum(base + L.scan, L.scan_bytes, cnt, off, (int)F + 1, s));
        const uint32_t next_base = level_base + F;
        k_front<<<blocks(8ull * F), kBlock, 0, s>>>(recs + level_base, F, next_base, tri_base, off, dec, nxt,
                                                    cap_nodes, err);
        uint64_t totals = 0;
        uint32_t e = 0;
        CRT_CUDA(cudaMemcpyAsync(&totals, off + F, 8, cudaMemcpyDeviceToHost, s));
        CRT_CUDA(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, s));
        CRT_CUDA(cudaStreamSynchronize(s));
        CRT_CUDA(cudaGetLastError());
        if (e) return set_error(CRT_ERR_CUDA, "GPU BVH build: inconsistent tree (" + std::to_string(e) + ")");
        level_base = next_base;
        tri_base += (uint32_t)totals;
        F = (uint32_t)(totals >> 32);
        if ((uint64_t)level_base + F > cap_nodes) return set_error(CRT_ERR_LIMIT, "GPU BVH node count overflow");
        std::swap(cur, nxt);
    }
    if (tri_base != n) return set_error(CRT_ERR_CUDA, "GPU BVH lost triangles");
    CRT_CUDA(nodes_out.alloc((size_t)level_base * sizeof(DevNodeQ16)));
    CRT_CUDA(fnodes_out.alloc((size_t)level_base * sizeof(Bvh8FloatNode)));
    CRT_CUDA(tris_out.alloc(n1 * (sizeof(DevTriA) + sizeof(DevTriB))));
    k_emit<<<blocks(8ull * level_base), kBlock, 0, s>>>(
        recs, level_base, gn, dec, perm, d_v1, d_e1, d_e2, nodes_out.as<DevNodeQ16>(), fnodes_out.as<Bvh8FloatNode>(),
        tris_out.as<DevTriA>(), reinterpret_cast<DevTriB*>(tris_out.as<DevTriA>() + n), n, err);
    uint32_t errbits = 0;
    CRT_CUDA(cudaMemcpyAsync(&errbits, err, 4, cudaMemcpyDeviceToHost, s));
    CRT_CUDA(cudaStreamSynchronize(s));
    CRT_CUDA(cudaGetLastError());
    if (errbits) return set_error(CRT_ERR_CUDA, "GPU BVH build: inconsistent tree (" + std::to_string(errbits) + ")");
    *num_nodes = level_base;
    *max_depth = depth;
    *fnodes_ok = level_base <= (1u << 24);
    return CRT_OK;
}

}  // namespace crt
