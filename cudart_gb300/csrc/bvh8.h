// bvh8.h -- host build of the 8-wide BVH with quantised child bounds.
//
// Replaces the reference's binary SAH build (src/geometry/bvh.cpp:65-323,
// 32-byte LinearBVHNode, two 1-D textures on the GPU) with:
//   1. a binned surface-area-heuristic binary build down to single
//      triangles (exact SAH sweep for ranges of at most 32);
//   2. an SAH-optimal collapse to 8-wide (or 4-wide) nodes by dynamic
//      programming (Ylitie et al., HPG 2017), which also groups triangles
//      into leaf slots of at most 3 (the reference's maxTrisInNode,
//      bvh.cpp:62);
//   3. child slots ordered by octant so that visiting slot k ^ octant(ray)
//      is approximately front to back;
//   4. child boxes quantised to 8 bits per plane relative to the node
//      origin with a power-of-two scale, rounded outward (conservative).
// Every triangle box is widened by a margin proportional to the scene's
// coordinate magnitude before the build, so the GPU's rounded slab tests
// never cull a triangle that the exact Moller-Trumbore test accepts.
#pragma once

#include <cstdint>
#include <cstring>
#include <vector>

namespace crt {

// 80-byte node as the host build makes it and crt_scene_export_bvh returns it.
struct alignas(16) Bvh8Node {
    float px, py, pz;          // quantisation origin
    uint8_t ex, ey, ez;        // biased exponents of the per-axis scale 2^(e-127)
    uint8_t imask;             // bit s: slot s is an internal node
    uint32_t child_base;       // index of the first internal child
    uint32_t tri_base;         // index of the first triangle record of the leaves
    uint8_t meta[8];           // 0 empty, 0x80 internal, else (count << 5) | offset
    uint8_t qlo[3][8];         // [axis][slot]
    uint8_t qhi[3][8];
};
static_assert(sizeof(Bvh8Node) == 80, "node layout");

// Device layouts.  What bounds the reads is the L1 data banks: 32 lanes that
// read 16 bytes at the same place of 32 different nodes take 34 cycles when the
// nodes lie a multiple of 128 bytes apart (every lane meets the same banks), and
// 12 at a distance that moves from bank to bank (144 or 208 bytes; 160: 14.6).
//
// `slots` holds the internal mask in bits 0-7 and, in bits 8-31, three bits
// per slot for its triangles (none for an internal or empty slot).  A node's
// triangle records follow one another in slot order, so triangle bit b is
// record tri_base + (bits set below b).
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t slots_word(uint8_t imask, const uint8_t meta[8]) {
    uint32_t w = imask;
    for (int s = 0; s < 8; ++s)
        if (!((imask >> s) & 1)) w |= ((1u << (meta[s] >> 5)) - 1u) << (8 + 3 * s);
    return w;
}

// The quantised node: child planes as 16-bit floats (the upper half of an FP32
// number) relative to the node origin; four 32-byte sectors.  A word holds
// the planes of slots k (low half) and k + 4 (high half).  The traversal uses
// the word as it is for slot k + 4, so that plane's value lies anywhere in
// [h, h | 0xFFFF]: a lo plane is rounded down until its largest reading is low
// enough, a hi plane up to the first whose least reading is high enough.
// Slot k's are rounded plainly.  All planes are >= 0; an empty slot's lo is the
// largest 16-bit float and its hi the lowest.  A hi plane beyond FLT_MAX reads
// as infinite or NaN: the slab test's minimum passes over both.
// 160 bytes apart: the banks vary, and lo and hi differ in one address bit.
struct alignas(32) DevNodeQ16 {
    float px, py, pz;
    uint32_t child_base, tri_base, slots, pad[2];
    uint32_t planes[3][2][4];  // [axis][lo, hi][k]
    uint32_t pad2[8];
};
static_assert(sizeof(DevNodeQ16) == 160, "node layout");

#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t plane16(double v, bool hi, bool high_half) {
    if (!(v > 0.0)) v = 0.0;
    float f = (float)v;
    uint32_t u;
    memcpy(&u, &f, 4);
    uint32_t h = u >> 16;                       // at or below f (f >= 0)
    auto value = [](uint32_t bits) {
        float x;
        memcpy(&x, &bits, 4);
        return (double)x;
    };
    if (hi) {
        while (value(h << 16) < v) ++h;
    } else {
        // (not above v, and a number: past FLT_MAX a high half would read as infinite or NaN)
        while (h > 0 && !(value((h << 16) | (high_half ? 0xFFFFu : 0u)) <= v)) --h;
    }
    return h;
}

// Writes one slot of a quantised node: planes relative to its origin.
#ifdef __CUDACC__
__host__ __device__
#endif
inline void set_planes16(DevNodeQ16& n, int axis, int slot, double lo, double hi) {
    const int k = slot & 3, sh = slot < 4 ? 0 : 16;
    uint32_t& l = n.planes[axis][0][k];
    uint32_t& h = n.planes[axis][1][k];
    l = (l & ~(0xFFFFu << sh)) | (plane16(lo, false, sh != 0) << sh);
    h = (h & ~(0xFFFFu << sh)) | (plane16(hi, true, sh != 0) << sh);
}

#ifdef __CUDACC__
__host__ __device__
#endif
inline void clear_planes16(DevNodeQ16& n) {
    for (int a = 0; a < 3; ++a)
        for (int k = 0; k < 4; ++k) {
            n.planes[a][0][k] = 0x7F7F7F7Fu;
            n.planes[a][1][k] = 0xFF7FFF7Fu;
        }
}

// The same node with full-precision child planes, read as thirteen 16-byte
// loads; byte offsets fit 32 bits for any index below 2^24.
struct alignas(16) Bvh8FloatNode {
    float planes[3][2][8];     // [axis][lo, hi][slot]; empty slot: lo = FLT_MAX, hi = -FLT_MAX
    uint32_t child_base, tri_base, slots, pad;
};
static_assert(sizeof(Bvh8FloatNode) == 208, "float node layout");

// Intersection record, 40 bytes in two arrays: one 256-bit and one 64-bit load.
struct alignas(32) DevTriA {
    float v1[3];
    uint32_t face;
    float e1[3], e2x;
};
struct alignas(8) DevTriB {
    float e2y, e2z;
};
static_assert(sizeof(DevTriA) == 32 && sizeof(DevTriB) == 8, "triangle layout");

// 48-byte triangle record of the host build and of crt_scene_export_bvh: v1.xyz + face index (bits), e1.xyz, e2.xyz.
struct alignas(16) TriRecord {
    float v1[3];
    uint32_t face;
    float e1[3];
    float pad1;
    float e2[3];
    float pad2;
};
static_assert(sizeof(TriRecord) == 48, "triangle layout");

struct Bvh8 {
    std::vector<Bvh8Node> nodes;
    std::vector<Bvh8FloatNode> fnodes;   // the same nodes with FP32 planes
    bool fnodes_ok = true;               // false beyond 2^24 nodes
    std::vector<TriRecord> tris;     // in leaf order
    uint32_t max_depth = 0;
    float margin = 0.f;
};

// v1/e1/e2: [n][3] floats as the scene computes them (e = v - v1, in FP32).
// Returns false (with msg) if the scene is empty or the tree exceeds
// max_levels levels.
// max_children: 8, or 4 for a narrower tree stored in the same node layout.
bool build_bvh8(const float* v1, const float* e1, const float* e2, uint32_t n,
                uint32_t max_levels, Bvh8& out, const char** msg, int max_children = 8);

}  // namespace crt
