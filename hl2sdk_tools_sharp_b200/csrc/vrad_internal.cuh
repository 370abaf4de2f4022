// vrad_internal.cuh -- device-side layout shared by the scene build and the
// traversal kernels of libvrad_cuda.
//
// Scene layout in HBM.  The triangles are split by the sky bit of their id
// into two BVHs, opaque and sky, each laid out as below (structure of
// arrays, every record 16-byte aligned so each is one or more 128-bit
// loads); tri_id is shared and indexed by the original triangle index.
//
//   tri0[i]  float4 (nx, ny, nz, d)          plane of the i-th triangle in
//   tri1[i]  float4 (e0, e1, e2, e3)         BVH leaf order: the reference's
//   tri2[i]  float4 (e4, e5, idx, meta)      KdTriangle, 48 B
//            idx  = original triangle index (int bits), the tie-break key
//            meta = drop axis (bits 0-1) | sky (bit 2) | FCACHETRI flags << 8
//   tri_id[orig]  int  the caller's id, read only for skip_id and outputs
//
// The nodes of a scene of up to kOctantTriangles triangles lie in eight
// copies, one per octant of a ray's direction (bit a set: the direction's
// axis a is negative), 2 x `inner` nodes each (1 KB an inner node); in a copy
// every box is stored as the planes such a ray meets first (near) and last
// (far), and child 0 is the child it meets first.  A larger scene has the
// first `inner` nodes of octant 0's copy alone (64 B an inner node), near the
// low planes and far the high ones:
//   node[k]  4 x float4 = 64 B, two child boxes and two child references:
//            n0 = child 0 (near.x, near.y, far.x, far.y)
//            n1 = child 1 (near.x, near.y, far.x, far.y)
//            n2 = (c0 near.z, c0 far.z, c1 near.z, c1 far.z)
//            n3 = (ref0, ref1, -, -)
//            ref >= 0 is an inner node; ref < 0 is a leaf, ~ref packing
//            (first triangle << 3) | (count - 1), so a leaf holds 1..8.
//            n3.z is -1.
// Of eight copies, nodes inner .. 2 inner - 1 lead from a subtree up to the rest of the tree:
// node inner + k has as its children the sibling of node k and the sibling
// of k's parent (an empty box where there is none), and n3.z the node that
// leads on from k's grandparent, -1 when the two children complete the
// tree.
#pragma once

#include <cstdint>
#include <type_traits>

#include "../../include/vrad_cuda.h"

namespace vrad {

constexpr int kMaxLeaf = 8;
constexpr int kStackDepth = 64;
constexpr uint32_t kTraceIdSky = 0x01000000u;   // TraceId.Sky (MapTools/Rad/TraceId.cs)
constexpr float kKdEps = 1.0e-10f;              // KdRayTracer.cs:1209-1230
constexpr float kKdHuge = 1.0e23f;              // KdRayTracer.cs:985
// Scenes of more triangles keep one copy of the nodes: where the two walks
// take as long for warps of neighbouring rays (walk_one's table).
constexpr int32_t kOctantTriangles = 20000;

struct DeviceBvh {
    const float4 *tri0;
    const float4 *tri1;
    const float4 *tri2;
    const float4 *nodes;
    int32_t ntris;  // 0: empty, never traversed
    int32_t depth;  // inner nodes on the longest root-to-leaf path
    int32_t inner;  // the tree's inner nodes
};

struct DeviceScene {
    DeviceBvh opaque;
    DeviceBvh sky;
    const int32_t *tri_id;
    bool one_copy;  // of the nodes: the kernels' ONE
    // The traversal stack's entries per thread (kernels size their shared
    // memory by it).  A walk holds at most one entry per inner node of the
    // path below the subtree it is in, and two more while it climbs: the
    // deeper tree's depth plus two.  The build refuses a tree deeper than
    // kStackDepth, so a walk needs no check of its own.
    __host__ __device__ int32_t stack_depth() const {
        const int32_t d = opaque.depth > sky.depth ? opaque.depth : sky.depth;
        return d + 2;
    }
};

// f(std::true_type or std::false_type): a launch of the kernel for the scene's
// copies of the nodes.
template <typename F>
auto by_copies(const DeviceScene &s, F &&f) {
    return s.one_copy ? f(std::true_type{}) : f(std::false_type{});
}

enum TraceMode : int { kModeAny = 0, kModeClosest = 1, kModeSkyPass = 2 };

struct TraceParams {
    float tmin;
    int32_t skip_id;
    int32_t mode;
};

__host__ __device__ inline int32_t leaf_ref(int32_t first, int32_t count) {
    return ~((first << 3) | (count - 1));
}

}  // namespace vrad
