// crt_device.cuh -- device code shared by the closest-hit, megakernel,
// wavefront and adjoint kernels (sm_103a).
//
// Arithmetic contract: every translation unit that includes this header is
// compiled with -fmad=false, so each float multiply and add rounds
// separately exactly like the reference's host pass; the slab tests use
// explicit fmaf() where fusing is wanted.  Division and square root are
// IEEE round-to-nearest (no fast-math).
#pragma once

#include <cfloat>
#include <cstdint>
#include <cuda_runtime.h>

#include "bvh8.h"

namespace crt {

#define CRT_D __device__ __forceinline__

constexpr float kEps = 0.00001f;      // EPSILON   (src/include/geometry.h:9)
constexpr float kEps2 = 0.000005f;    // EPSILON_2 (src/include/geometry.h:10)
constexpr int kNoTexture = -1;

enum Bsdf : int { DIFFUSE = 0, SPECULAR = 1, DIFFSPEC = 2, MICROFACET = 3, REFRACTIVE = 4, EMISSIVE = 5 };

// Traversal stack: the first entries of each thread's stack live in shared
// memory (kStackShared by default, or the launch's chosen depth, at most
// kStackSharedMax), the rest in local memory, which only very deep trees
// touch.  A traversal never holds more than kMaxLevels entries.
constexpr int kStackShared = 16;
constexpr int kStackSharedMax = 32;
constexpr int kMaxLevels = 64;
constexpr uint32_t kMaxNodeVisits = 1u << 20;   // default watchdog per traversal
constexpr uint32_t kVisitCeiling = 1u << 30;    // largest limit; the counter starts at ceiling - limit

enum ErrorBits : uint32_t { ERR_WATCHDOG = 1u, ERR_STACK = 2u };

// ---------------------------------------------------------------------------
// Device view of a scene (all arrays in HBM, 16-byte aligned).
// ---------------------------------------------------------------------------
struct DevScene {
    const DevNodeQ16* nodes;       // 16-bit planes
    const Bvh8FloatNode* fnodes;   // the same nodes with FP32 planes, or null
    const DevTriA* tris_a;         // intersection records in leaf order: v1, face, e1, e2.x
    const DevTriB* tris_b;         //                                     and e2.yz
    const float4* shade;       // 3 float4 per face: n1.xyz n2.x | n2.yz n3.xy | n3.z area mat 0
    const float4* uvs;         // 2 float4 per face: uv1 uv2 | uv3 0 0
    const float4* mats;        // 4 float4 per material: kd tex | ka bsdf | ks ns | ni diffuse 0 0
    const float4* light_geo;   // 3 float4 per light: v1 face | e1 area | e2 material
    const float4* texels;      // rgb0 per texel, with the zero padding
    const uint2* tex_dims;
    const uint32_t* tex_offsets;
    uint32_t tex_total;
    uint32_t n_lights;
    float lights_area;
    uint32_t n_faces;
    uint32_t max_visits;       // node visits a traversal may make (watchdog), <= kVisitCeiling
    uint32_t* error;           // ErrorBits, sticky until crt_scene_clear_errors
};

struct Camera {
    float3 eye, dir, up, right;
    float fov, aspect, aperture, focus;
    int xpixels, ypixels;
};

// ---------------------------------------------------------------------------
// float3 helpers in the reference's operation order (src/include/linalg.h)
// ---------------------------------------------------------------------------
CRT_D float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
CRT_D float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
CRT_D float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
CRT_D float3 operator*(float3 a, float3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
CRT_D float3 operator*(float3 a, float b) { return f3(a.x * b, a.y * b, a.z * b); }
CRT_D float3 operator/(float3 a, float b) { return f3(a.x / b, a.y / b, a.z / b); }
CRT_D float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
CRT_D float3 cross(float3 a, float3 b) {
    return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
CRT_D float3 normalize(float3 v) {
    float n = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
    return f3(v.x / n, v.y / n, v.z / n);
}
CRT_D float max_component(float3 v) { float m = v.x > v.y ? v.x : v.y; return m > v.z ? m : v.z; }
CRT_D float3 xyz(float4 v) { return f3(v.x, v.y, v.z); }

template <typename T>
CRT_D T ldg(const T* p) { return __ldg(p); }

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11) and the per-sample stream.
// Key = seed; counter = (draw / 4, sample, pixel, view).  A draw is
// (x >> 8) * 2^-24 in [0, 1).
// ---------------------------------------------------------------------------
CRT_D uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

struct Rng {
    uint2 key;
    uint32_t sample, pixel, view;
    uint32_t n;          // draws consumed
    uint4 buf;

    CRT_D void init(uint64_t seed, uint32_t view_, uint32_t pixel_, uint32_t sample_, uint32_t n0 = 0) {
        key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
        sample = sample_;
        pixel = pixel_;
        view = view_;
        n = n0;
        if (n & 3u) buf = philox4x32_10(make_uint4(n >> 2, sample, pixel, view), key);
    }
    // Sampler::getNextFloat (src/renderer/renderer.cu:72-78).
    CRT_D float next() {
        uint32_t lane = n & 3u;
        if (lane == 0) buf = philox4x32_10(make_uint4(n >> 2, sample, pixel, view), key);
        uint32_t x = lane == 0 ? buf.x : (lane == 1 ? buf.y : (lane == 2 ? buf.z : buf.w));
        ++n;
        return (float)(x >> 8) * 0x1p-24f;
    }
};

// ---------------------------------------------------------------------------
// Moller-Trumbore, Triangle::intersect (src/geometry/geometry.cu:38-65), in
// the reference's operation order with explicitly rounded operations, so t,
// u, v are bit-identical to the CPU path.  Returns FLT_MAX on a miss.
// ---------------------------------------------------------------------------
CRT_D float mt_intersect(float3 o, float3 d, float3 v1, float3 e1, float3 e2, float& ou, float& ov) {
    float px = __fsub_rn(__fmul_rn(d.y, e2.z), __fmul_rn(d.z, e2.y));
    float py = __fsub_rn(__fmul_rn(d.z, e2.x), __fmul_rn(d.x, e2.z));
    float pz = __fsub_rn(__fmul_rn(d.x, e2.y), __fmul_rn(d.y, e2.x));
    float det = __fadd_rn(__fadd_rn(__fmul_rn(e1.x, px), __fmul_rn(e1.y, py)), __fmul_rn(e1.z, pz));
    if (fabsf(det) < kEps) return FLT_MAX;
    float inv_det = __frcp_rn(det);
    float tx = __fsub_rn(o.x, v1.x), ty = __fsub_rn(o.y, v1.y), tz = __fsub_rn(o.z, v1.z);
    float u = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(tx, px), __fmul_rn(ty, py)), __fmul_rn(tz, pz)), inv_det);
    if (u < 0.f || u > 1.f) return FLT_MAX;
    float qx = __fsub_rn(__fmul_rn(ty, e1.z), __fmul_rn(tz, e1.y));
    float qy = __fsub_rn(__fmul_rn(tz, e1.x), __fmul_rn(tx, e1.z));
    float qz = __fsub_rn(__fmul_rn(tx, e1.y), __fmul_rn(ty, e1.x));
    float v = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(d.x, qx), __fmul_rn(d.y, qy)), __fmul_rn(d.z, qz)), inv_det);
    if (v < 0.f || __fadd_rn(u, v) > 1.f) return FLT_MAX;
    float t = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(e2.x, qx), __fmul_rn(e2.y, qy)), __fmul_rn(e2.z, qz)), inv_det);
    if (t > kEps) { ou = u; ov = v; return t; }
    return FLT_MAX;
}

// ---------------------------------------------------------------------------
// 8-wide BVH traversal.
// ---------------------------------------------------------------------------
struct Hit {
    float t;
    int32_t face;
    float u, v;
};

// Counting traversals: node visits and triangle tests.
struct TraversalStats {
    uint32_t nodes, tris;
};

// Per-thread stack: shared-memory part (stride = threads per block) and a
// local-memory overflow part.  The overflow array is the kernel's own
// variable: as a member, its dynamic indexing would keep the whole struct, the
// stack pointer included, in local memory (8.4M queries into the
// 2.17M-triangle scene: 6.80 ms so, 5.65 ms as it is).
using StackSpill = uint2[kMaxLevels];
struct Stack {
    uint2* sh;           // this thread's first shared entry; entries are `stride` apart
    uint2* spill;
    uint32_t stride;     // threads per block
    int depth;           // entries kept in shared memory
    int sp;

    CRT_D Stack(uint2* base, StackSpill& overflow, uint32_t threads, int shared_depth)
        : sh(base + threadIdx.x), spill(overflow), stride(threads), depth(shared_depth), sp(0) {}
    CRT_D void push(uint2 e) {
        if (sp < depth) sh[sp * stride] = e;
        else spill[sp - depth] = e;
        ++sp;
    }
    CRT_D uint2 pop() {
        --sp;
        return sp < depth ? sh[sp * stride] : spill[sp - depth];
    }
};

CRT_D float safe_rcp(float d) {
    float a = fabsf(d);
    return 1.0f / copysignf(a > 0x1p-80f ? a : 0x1p-80f, d);
}

// 256-bit read-only load (sm_100 and later) as four pairs of floats; p is
// 32-byte aligned.
CRT_D void ld256(const void* p, uint64_t (&v)[4]) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}

// Pairs of floats in one 64-bit register and their fused multiply-add (one
// instruction on sm_100 and later, each half rounded as fmaf).
CRT_D uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
CRT_D float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
CRT_D uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Three-input min / max (PTX ISA 8.8, sm_100 and later): one instruction each.
CRT_D float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
CRT_D float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Resumable traversal of one ray.  step() visits one node (popping the
// stack first when the current group is exhausted) and tests the triangles
// of the leaves it hits; it returns true when the ray is finished.  Kernels
// that keep a lane busy with a new ray as soon as its old one finishes drive
// step() directly; traverse() runs a ray to completion.
//
// Mode CLOSEST: nearest hit with the lowest-face tie rule, h.t starts at tmax.
// Mode OCCLUDED: finishes as soon as a face other than `target` is hit with
// t < h.t, or t == h.t and face < target (exactly the faces that would make
// the closest hit differ from `target`); `occluded` is then true.
//
// What bounds it (ncu, bounce 1 of the 1080p frame, 64 registers, 32 warps per
// SM, 14-15 of 32 lanes active): issue slots with the quantised nodes (77% of
// cycles issue, the ALU pipe 56% busy), L1 with the FP32 ones.  So a visit is kept
// short on the ALU pipe: two planes per multiply-add, the eight misses collected
// by sign with one funnel shift each, the nearest child found by narrowing the
// slot mask instead of permuting it, triangles of the hit leaves selected by
// spreading slot bits to the three bits each owns.  Against the previous form
// (compare and set per child, octant permutation, a loop over leaf slots, 8-bit
// planes converted one by one, nodes of 80 and 208 bytes with the triangles in
// three loads each): 1080p x 256 424 -> 351 ms with FP32 nodes, 1001x563 x 32
// mixed scene 49.3 -> 36.8 ms with quantised ones, 1M queries 531 -> 416 us.
template <bool OCCLUDED, bool COUNT, bool WHOLE_LEAF = true, bool F32 = false>
struct Traversal {
    float3 o, d;
    float ix, iy, iz, tmin;
    uint32_t oct;
    uint2 grp;          // child base, internal mask << 8 | children still to visit (slots)
    uint32_t tri_base;  // triangles of the last visited node still to test,
    uint32_t tri_mask;  //   three bits per slot,
    uint32_t tri_all;   //   among all the node's triangles
    uint32_t visits;
    int32_t target;
    bool occluded;
    Hit h;

    // max_visits: the scene's watchdog limit (DevScene::max_visits); the
    // counter starts at kVisitCeiling - max_visits so that every visit
    // compares against a constant.
    CRT_D void init(float3 o_, float3 d_, float tmin_, float tmax, int32_t target_, Stack& st,
                    uint32_t max_visits) {
        o = o_;
        d = d_;
        ix = safe_rcp(d.x);
        iy = safe_rcp(d.y);
        iz = safe_rcp(d.z);
        tmin = tmin_;
        oct = (signbit(d.x) ? 1u : 0u) | (signbit(d.y) ? 2u : 0u) | (signbit(d.z) ? 4u : 0u);
        grp = make_uint2(0u, (1u << 8) | 1u);   // root = slot 0 of a virtual parent
        tri_base = tri_mask = tri_all = 0;
        visits = kVisitCeiling - max_visits;
        target = target_;
        occluded = false;
        h.t = tmax;
        h.face = -1;
        h.u = h.v = 0.f;
        st.sp = 0;
    }

    // One pending triangle test.  Returns true if it ends an occlusion query.
    CRT_D bool test_triangle(const DevScene& S, TraversalStats* stats) {
        const uint32_t low = tri_mask & (0u - tri_mask);
        tri_mask ^= low;
        const uint32_t i = tri_base + __popc(tri_all & (low - 1u));
        uint64_t a[4];
        ld256(S.tris_a + i, a);
        const float2 b = ldg(reinterpret_cast<const float2*>(S.tris_b + i));
        const float2 a0 = unpack2(a[0]), a1 = unpack2(a[1]), a2 = unpack2(a[2]), a3 = unpack2(a[3]);
        if (COUNT) stats->tris++;
        float u, v;
        const float t = mt_intersect(o, d, f3(a0.x, a0.y, a1.x), f3(a2.x, a2.y, a3.x), f3(a3.y, b.x, b.y), u, v);
        const int32_t face = (int32_t)__float_as_uint(a1.y);
        if (t == FLT_MAX || !(t > tmin)) return false;
        if (OCCLUDED) {
            if (face != target && (t < h.t || (t == h.t && face < target))) {
                occluded = true;
                return true;
            }
        } else if (t < h.t || (t == h.t && h.face >= 0 && face < h.face)) {
            h.t = t;
            h.face = face;
            h.u = u;
            h.v = v;
        }
        return false;
    }

    // One unit of work: the next pending triangle of the last visited node,
    // else one node visit.  Lanes of a warp that are testing triangles and
    // lanes that are visiting nodes each do one unit per step, so a leaf
    // with many triangles does not hold the other lanes back.
    // With WHOLE_LEAF a step is one node visit followed by all of its
    // triangle tests.
    CRT_D bool step(const DevScene& S, Stack& st, TraversalStats* stats) {
        if (WHOLE_LEAF) {
            if (visit(S, st, stats)) return true;
            while (tri_mask)
                if (test_triangle(S, stats)) return true;
            return false;
        }
        if (tri_mask) return test_triangle(S, stats);
        return visit(S, st, stats);
    }

    // Shifts the two children's miss bits into `miss` (the higher slot
    // first): a child is missed when its interval [near, far], clipped to
    // [tmin, h.t], is empty, that is, when far - near is negative.
    CRT_D void slab_pair(uint64_t nx, uint64_t ny, uint64_t nz, uint64_t fx, uint64_t fy, uint64_t fz,
                         uint32_t& miss) const {
        const float2 ax = unpack2(nx), ay = unpack2(ny), az = unpack2(nz);
        const float2 bx = unpack2(fx), by = unpack2(fy), bz = unpack2(fz);
        const float d1 = min3f(bx.y, by.y, fminf(bz.y, h.t)) - max3f(ax.y, ay.y, fmaxf(az.y, tmin));
        const float d0 = min3f(bx.x, by.x, fminf(bz.x, h.t)) - max3f(ax.x, ay.x, fmaxf(az.x, tmin));
        miss = __funnelshift_l(__float_as_uint(d1), miss, 1);
        miss = __funnelshift_l(__float_as_uint(d0), miss, 1);
    }

    // Slab tests of the 8 children of a quantised node: planes are 16-bit
    // floats relative to the node origin, t = plane * (1/d) + (origin - o) *
    // (1/d).  A word holds slot k in its low and slot k + 4 in its high half;
    // shifted left it is slot k's plane, and as it stands slot k + 4's to within
    // the low half, which the encoding has rounded past (DevNodeQ16).  So the
    // planes cost one shift for two, and pairs of words feed the two-wide
    // multiply-adds as they were loaded.
    CRT_D uint32_t test_children_q16(const DevScene& S, uint32_t node, uint32_t& child_base,
                                     uint32_t& tri_base_new, uint32_t& slots) const {
        // a node is 32-byte aligned: bit 4 of the address picks lo or hi
        const uintptr_t at = reinterpret_cast<uintptr_t>(S.nodes + node);
        auto load = [](uintptr_t p) { return ldg(reinterpret_cast<const uint4*>(p)); };
        const uintptr_t x = at | ((oct & 1u) << 4), y = at | ((oct & 2u) << 3), z = at | ((oct & 4u) << 2);
        uint64_t hd[4];
        ld256(reinterpret_cast<const void*>(at), hd);
        const uint4 nx = load(x + 32), ny = load(y + 64), nz = load(z + 96);
        const uint4 fx = load((x ^ 16) + 32), fy = load((y ^ 16) + 64), fz = load((z ^ 16) + 96);
        const float2 h0 = unpack2(hd[0]), h1 = unpack2(hd[1]), h2 = unpack2(hd[2]);
        child_base = __float_as_uint(h1.y);
        tri_base_new = __float_as_uint(h2.x);
        slots = __float_as_uint(h2.y);
        const float cx = (h0.x - o.x) * ix, cy = (h0.y - o.y) * iy, cz = (h1.x - o.z) * iz;
        const uint64_t ix2 = pack2(ix, ix), iy2 = pack2(iy, iy), iz2 = pack2(iz, iz);
        const uint64_t cx2 = pack2(cx, cx), cy2 = pack2(cy, cy), cz2 = pack2(cz, cz);
        auto raw = [](uint32_t a, uint32_t b) { return pack2(__uint_as_float(a), __uint_as_float(b)); };
        auto low = [&](uint32_t a, uint32_t b) { return raw(a << 16, b << 16); };
        uint32_t miss = 0;
        slab_pair(fma2(raw(nx.z, nx.w), ix2, cx2), fma2(raw(ny.z, ny.w), iy2, cy2), fma2(raw(nz.z, nz.w), iz2, cz2),
                  fma2(raw(fx.z, fx.w), ix2, cx2), fma2(raw(fy.z, fy.w), iy2, cy2), fma2(raw(fz.z, fz.w), iz2, cz2), miss);
        slab_pair(fma2(raw(nx.x, nx.y), ix2, cx2), fma2(raw(ny.x, ny.y), iy2, cy2), fma2(raw(nz.x, nz.y), iz2, cz2),
                  fma2(raw(fx.x, fx.y), ix2, cx2), fma2(raw(fy.x, fy.y), iy2, cy2), fma2(raw(fz.x, fz.y), iz2, cz2), miss);
        slab_pair(fma2(low(nx.z, nx.w), ix2, cx2), fma2(low(ny.z, ny.w), iy2, cy2), fma2(low(nz.z, nz.w), iz2, cz2),
                  fma2(low(fx.z, fx.w), ix2, cx2), fma2(low(fy.z, fy.w), iy2, cy2), fma2(low(fz.z, fz.w), iz2, cz2), miss);
        slab_pair(fma2(low(nx.x, nx.y), ix2, cx2), fma2(low(ny.x, ny.y), iy2, cy2), fma2(low(nz.x, nz.y), iz2, cz2),
                  fma2(low(fx.x, fx.y), ix2, cx2), fma2(low(fy.x, fy.y), iy2, cy2), fma2(low(fz.x, fz.y), iz2, cz2), miss);
        return miss;
    }

    // Slab tests of the 8 children of a node with FP32 planes:
    // t = plane * (1/d) - o * (1/d) in one fused multiply-add per plane.  Four
    // slots at a time, in 128-bit loads: holding all 48 planes at once (256-bit
    // loads) takes 72-80 registers and lost 3-7% on the 1080p frame.
    CRT_D uint32_t test_children_f32(const DevScene& S, uint32_t node, uint32_t& child_base,
                                     uint32_t& tri_base_new, uint32_t& slots) const {
        const float ox = -o.x * ix, oy = -o.y * iy, oz = -o.z * iz;
        const uint64_t ix2 = pack2(ix, ix), iy2 = pack2(iy, iy), iz2 = pack2(iz, iz);
        const uint64_t ox2 = pack2(ox, ox), oy2 = pack2(oy, oy), oz2 = pack2(oz, oz);
        uint32_t miss = 0;
        auto four = [&](float4 nx, float4 ny, float4 nz, float4 fx, float4 fy, float4 fz) {
            slab_pair(fma2(pack2(nx.z, nx.w), ix2, ox2), fma2(pack2(ny.z, ny.w), iy2, oy2),
                      fma2(pack2(nz.z, nz.w), iz2, oz2), fma2(pack2(fx.z, fx.w), ix2, ox2),
                      fma2(pack2(fy.z, fy.w), iy2, oy2), fma2(pack2(fz.z, fz.w), iz2, oz2), miss);
            slab_pair(fma2(pack2(nx.x, nx.y), ix2, ox2), fma2(pack2(ny.x, ny.y), iy2, oy2),
                      fma2(pack2(nz.x, nz.y), iz2, oz2), fma2(pack2(fx.x, fx.y), ix2, ox2),
                      fma2(pack2(fy.x, fy.y), iy2, oy2), fma2(pack2(fz.x, fz.y), iz2, oz2), miss);
        };
        // node offsets stay below 2^32 (indices are below 2^24)
        const char* base = reinterpret_cast<const char*>(S.fnodes);
        constexpr uint32_t kSize = sizeof(Bvh8FloatNode);
        const uint32_t lo = node * kSize, hi = node * kSize + 32u;
        const uint32_t x = (oct & 1u) << 5, y = (oct & 2u) << 4, z = (oct & 4u) << 3;
        auto load = [&](uint32_t k, uint32_t off) { return ldg(reinterpret_cast<const float4*>(base + k + off)); };
        const float4 hd = load(192, lo);
#pragma unroll
        for (int h = 16; h >= 0; h -= 16)
            four(load(h, lo + x), load(64 + h, lo + y), load(128 + h, lo + z), load(h, hi - x), load(64 + h, hi - y),
                 load(128 + h, hi - z));
        child_base = __float_as_uint(hd.x);
        tri_base_new = __float_as_uint(hd.y);
        slots = __float_as_uint(hd.z);
        return miss;
    }

    // Visits the next node: pops the stack first when the current group is
    // exhausted; returns true when nothing is left.
    CRT_D bool visit(const DevScene& S, Stack& st, TraversalStats* stats) {
        uint32_t m = grp.y & 0xFFu;
        if (m == 0) {
            if (st.sp == 0) return true;
            grp = st.pop();
            m = grp.y & 0xFFu;
        }
        // the nearest child in octant order: of the slots left, the one with
        // the least slot ^ oct, narrowed one bit of the slot number at a time
        const uint32_t m4 = m & ((oct & 4u) ? 0xF0u : 0x0Fu);
        m = m4 ? m4 : m;
        const uint32_t m2 = m & ((oct & 2u) ? 0xCCu : 0x33u);
        m = m2 ? m2 : m;
        const uint32_t m1 = m & ((oct & 1u) ? 0xAAu : 0x55u);
        m = m1 ? m1 : m;
        const uint32_t node = grp.x + __popc((grp.y >> 8) & (m - 1u));
        grp.y ^= m;
        if (grp.y & 0xFFu) {
            if (st.sp >= kMaxLevels) { atomicOr(S.error, ERR_STACK); return true; }
            st.push(grp);
        }
        if (++visits > kVisitCeiling) { atomicOr(S.error, ERR_WATCHDOG); return true; }
        if (COUNT) stats->nodes++;
        uint32_t child_base, tri_base_new, slots;
        const uint32_t miss = F32 ? test_children_f32(S, node, child_base, tri_base_new, slots)
                                  : test_children_q16(S, node, child_base, tri_base_new, slots);
        // Empty slots hold inverted boxes and have no triangle bits.  The
        // hit leaf slots spread to three bits each select their triangles.
        const uint32_t imask = slots & 0xFFu;
        grp = make_uint2(child_base, (imask << 8) | (imask & ~miss));
        uint32_t x = ~(miss | imask) & 0xFFu;
        x = (x * 257u) & 0x00F00Fu;
        x = (x * 17u) & 0x0C30C3u;
        x = (x * 5u) & 0x249249u;
        tri_base = tri_base_new;
        tri_all = slots >> 8;
        tri_mask = (x * 7u) & tri_all;
        return false;
    }
};

template <bool OCCLUDED, bool COUNT, bool F32 = false>
CRT_D bool traverse(const DevScene& S, float3 o, float3 d, float tmin, Hit& h, int32_t target,
                    Stack& st, TraversalStats* stats) {
    Traversal<OCCLUDED, COUNT, true, F32> T;
    T.init(o, d, tmin, h.t, target, st, S.max_visits);
    while (!T.step(S, st, stats)) {
    }
    if (!OCCLUDED) h = T.h;
    return T.occluded;
}

// ---------------------------------------------------------------------------
// Estimator pieces (src/renderer/renderer.cu:119-262 and helpers)
// ---------------------------------------------------------------------------
struct Material {
    float3 kd, ka, ks;
    float ns, ni, diffuse;
    int bsdf, tex;
};

CRT_D Material load_material(const DevScene& S, uint32_t m) {
    const float4* p = S.mats + 4ull * m;
    float4 a = ldg(p), b = ldg(p + 1), c = ldg(p + 2), d = ldg(p + 3);
    Material r;
    r.kd = xyz(a); r.tex = __float_as_int(a.w);
    r.ka = xyz(b); r.bsdf = __float_as_int(b.w);
    r.ks = xyz(c); r.ns = c.w;
    r.ni = d.x; r.diffuse = d.y;
    return r;
}

struct Shading {
    float3 n1, n2, n3;
    float area;
    uint32_t material;
};

CRT_D Shading load_shading(const DevScene& S, uint32_t face) {
    const float4* p = S.shade + 3ull * face;
    float4 a = ldg(p), b = ldg(p + 1), c = ldg(p + 2);
    Shading s;
    s.n1 = xyz(a);
    s.n2 = f3(a.w, b.x, b.y);
    s.n3 = f3(b.z, b.w, c.x);
    s.area = c.y;
    s.material = __float_as_uint(c.z);
    return s;
}

// Triangle::getNormal (src/geometry/geometry.cu:67-71).
CRT_D float3 shading_normal(const Shading& s, float u, float v) {
    float w = 1.f - u - v;
    return normalize(s.n1 * w + s.n2 * u + s.n3 * v);
}

// sampleTexture, host branch (src/renderer/renderer.cu:92-115): bilinear at
// (u*W, v*H) without a half-texel offset or wrap; neighbours at i+1 / j+1
// read the next texel of the flattened array, which ends in zero padding.
CRT_D float3 sample_texture(const DevScene& S, int tex, float u, float v) {
    const uint2 dim = ldg(S.tex_dims + tex);
    const uint32_t off = ldg(S.tex_offsets + tex);
    const uint32_t avail = S.tex_total - off;
    const float pu = u * (float)dim.x;
    const float pv = v * (float)dim.y;
    const uint32_t i = (uint32_t)truncf(pu);
    const uint32_t j = (uint32_t)truncf(pv);
    const float fu = floorf(pu), fv = floorf(pv), cu = ceilf(pu), cv = ceilf(pv);
    const uint32_t ia = j * dim.x + i + 1, ib = j * dim.x + i;
    const uint32_t ic = (j + 1) * dim.x + i + 1, id = (j + 1) * dim.x + i;
    const float4* p = S.texels + off;
    const float3 z = f3(0.f, 0.f, 0.f);
    const float3 ta = ia < avail ? xyz(ldg(p + ia)) : z, tb = ib < avail ? xyz(ldg(p + ib)) : z;
    const float3 tc = ic < avail ? xyz(ldg(p + ic)) : z, td = id < avail ? xyz(ldg(p + id)) : z;
    const float3 a1 = ta * (pu - fu);
    const float3 a2 = tb * (cu - pu);
    const float3 b1 = tc * (pu - fu);
    const float3 b2 = td * (cu - pu);
    return (a1 + a2) * (cv - pv) + (b1 + b2) * (pv - fv);
}

struct Ray {
    float3 o, d;
};

// tentFilter + Camera::computeCameraRay (src/geometry/camera.cu:13-57).
CRT_D Ray camera_ray(const Camera& c, int i, int j, Rng& rng) {
    const float r1 = 2.f * rng.next();
    const float r2 = 2.f * rng.next();
    const float dx = r1 < 1.f ? sqrtf(r1) - 1.f : 1.f - sqrtf(2.f - r1);
    const float dy = r2 < 1.f ? sqrtf(r2) - 1.f : 1.f - sqrtf(2.f - r2);
    // (float)((double)a - 0.5) equals the float subtraction: a - 0.5 is exact in double
    const float ni = (((float)i + dx) / (float)c.xpixels) - 0.5f;
    const float nj = 0.5f - (((float)j + dy) / (float)c.ypixels);
    float3 dir = c.dir;
    float3 origin = c.eye;
    dir = dir + c.right * c.fov * c.aspect * ni;
    dir = dir + c.up * c.fov * nj;
    if (c.aperture > 0.0f) {
        const float q1 = (float)((double)rng.next() - 3.14159265358979323846);
        const float q2 = rng.next() - 0.5f;
        float s, co;
        sincosf(q1, &s, &co);
        const float rj = co * q2 * c.aperture;
        const float uj = s * q2 * c.aperture;
        origin = origin + (c.right * rj + c.up * uj);
        const float3 focal = c.eye + dir * c.focus;
        dir = focal - origin;
    }
    Ray r;
    r.o = origin;
    r.d = normalize(dir);
    return r;
}

// Diffuse direction of sampleDiffuseBSDF (src/renderer/renderer.cu:375-402).
CRT_D float3 diffuse_direction(float3 normal, Rng& rng) {
    const float r1 = (float)(6.283185307179586 * (double)rng.next());   // 2 * M_PI * xi
    const float r2 = rng.next();
    const float r2sq = sqrtf(r2);
    const float3 w = normal;
    const float3 u = normalize(cross(fabsf(w.x) > 0.1f ? f3(0.f, 1.f, 0.f) : f3(1.f, 0.f, 0.f), w));
    const float3 v = cross(w, u);
    float s, c;
    sincosf(r1, &s, &c);
    return normalize(u * c * r2sq + v * s * r2sq + w * sqrtf(1.f - r2));
}

struct Fresnel {
    float pr, pt;
    float3 tdir;
};

// getFresnelReflectance (src/renderer/renderer.cu:464-493), including its
// R0 = (etai - etat)^2 / (etat + etai) * (etat + etai) grouping.
CRT_D Fresnel fresnel(float3 incident, float3 normal, float ior) {
    float cosi = dot(incident, normal);
    float etai = 1.f, etat = ior;
    float3 n = normal;
    if (cosi < 0.0f) cosi = -cosi;
    else { float tmp = etai; etai = etat; etat = tmp; n = normal * -1.0f; }
    const float eta = etai / etat;
    const float k = 1.f - eta * eta * (1.f - cosi * cosi);
    Fresnel f;
    f.tdir = f3(0.f, 0.f, 0.f);
    if (k < 0.f) { f.pr = 1.0f; f.pt = 0.0f; return f; }
    f.tdir = incident * eta + n * (eta * cosi - sqrtf(k));
    const float R0 = (etai - etat) * (etai - etat) / (etat + etai) * (etat + etai);
    const float c = 1.f - dot(f.tdir, normal);
    const float Re = R0 + (1.f - R0) * c * c * c * c * c;
    f.pr = Re;
    f.pt = 1.f - Re;
    return f;
}

struct LightGeo {
    float3 v1, e1, e2;
    float area;
    uint32_t face, material;
};

CRT_D LightGeo load_light(const DevScene& S, uint32_t i) {
    const float4* p = S.light_geo + 3ull * i;
    float4 a = ldg(p), b = ldg(p + 1), c = ldg(p + 2);
    LightGeo l;
    l.v1 = xyz(a); l.face = __float_as_uint(a.w);
    l.e1 = xyz(b); l.area = b.w;
    l.e2 = xyz(c); l.material = __float_as_uint(c.w);
    return l;
}

// Light pick of samplePixel (src/renderer/renderer.cu:218-219).
CRT_D uint32_t pick_light(const DevScene& S, float xi) {
    const float rn = xi * ((float)S.n_lights - .00001f);
    uint32_t li = (uint32_t)truncf(rn);
    return li < S.n_lights ? li : S.n_lights - 1;
}

// Triangle::getRandomPointOn (src/geometry/geometry.cu:73-80).
CRT_D float3 light_point(const LightGeo& l, float pu, float pv) {
    if (pu + pv >= 1.0f) { pu = 1.0f - pu; pv = 1.0f - pv; }
    return l.v1 + l.e1 * pu + l.e2 * pv;
}

// Contribution of estimateDirectLighting after a successful shadow test
// (src/renderer/renderer.cu:436-443): ka_light * A |cos| / (d^2 A_total).
// Geometry weight of a light sample: the contribution is lcolor * weight.
CRT_D float light_weight(const DevScene& S, const LightGeo& l, float t, float lu, float lv, float3 dir) {
    const Shading ls = load_shading(S, l.face);
    const float d2 = t * t;
    const float cost = fabsf(dot(shading_normal(ls, lu, lv), dir * -1.0f));
    return l.area / (d2 * S.lights_area) * cost;
}

CRT_D float3 light_contribution(const DevScene& S, const LightGeo& l, float3 lcolor, float t,
                                float lu, float lv, float3 dir) {
    return f3(0.f, 0.f, 0.f) + lcolor * light_weight(S, l, t, lu, lv, dir);
}

}  // namespace crt
