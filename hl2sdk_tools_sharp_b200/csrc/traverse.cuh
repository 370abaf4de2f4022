// traverse.cuh -- the per-ray BVH walk shared by the trace kernels
// (trace.cu) and the fused lighting kernels (direct.cu).
//
// Per-triangle arithmetic is the reference's KdRayTracer.IntersectTriangle
// (MapTools/Tracing/KdRayTracer.cs:1194-1267) operation for operation, each
// an explicitly rounded intrinsic, so an accepted/rejected decision and a
// hit distance are the CPU's bits.  The walk tests every triangle whose
// padded box the segment meets, which includes every triangle the
// predicate can accept.
#pragma once

#include "vrad_internal.cuh"

namespace vrad {

constexpr int kBlock = 128;       // threads per CTA of every traversal kernel
constexpr uint32_t kFull = 0xffffffffu;

struct RayState {
    float ox, oy, oz, dx, dy, dz;
    float ix, iy, iz;      // 1/d with zeros saturated to +-2^60
    float nox, noy, noz;   // -o/d, for the FMA slab test
    // The direction's octant: the copy of the nodes the walk reads (of eight).
    __device__ __forceinline__ int octant() const {
        return (int)((__float_as_uint(ix) >> 31) | ((__float_as_uint(iy) >> 31) << 1) |
                     ((__float_as_uint(iz) >> 31) << 2));
    }
};

__device__ inline float recip_saturate(float a) {
    // ReciprocalSaturateExact (KdRayTracer.cs:1446): a zero keeps its sign
    // and becomes 2^-60 before the divide.
    if (a == 0.0f) a = __uint_as_float(__float_as_uint(a) | 0x21800000u);
    return __frcp_rn(a);
}

__device__ inline float sel3(int axis, float x, float y, float z) {
    return axis == 0 ? x : (axis == 1 ? y : z);
}

// The FP64 recheck's flag (vrad_trace_visibility_recheck): set when a
// triangle's FP32 predicate values lie within `m` of a decision boundary --
// an edge value near 0, their sum near 1, or t near either end of the
// segment [tlo, thi] -- and no farther than `m` outside on the others.
struct NearCheck {
    float m, tlo, thi;
    bool near;
};

// The predicate.  Returns true with the exact t when the triangle accepts
// the ray (|d.n| > eps, eps < t < 1e23, both edge values >= eps, their sum
// <= 1).  With FLAG the near-boundary test runs first; the decision itself
// is the same arithmetic either way.
template <bool FLAG = false>
__device__ __forceinline__ bool kd_hit(const DeviceBvh &s, int k, const RayState &r, float &t_out,
                                       uint32_t &meta_out, int32_t &orig_out, NearCheck *nc = nullptr) {
    const float4 A = __ldg(&s.tri0[k]);
    float ddotn = __fmul_rn(r.dx, A.x);
    ddotn = __fadd_rn(__fmul_rn(r.dy, A.y), ddotn);
    ddotn = __fadd_rn(__fmul_rn(r.dz, A.z), ddotn);
    float odotn = __fmul_rn(r.ox, A.x);
    odotn = __fadd_rn(__fmul_rn(r.oy, A.y), odotn);
    odotn = __fadd_rn(__fmul_rn(r.oz, A.z), odotn);
    const float num = __fsub_rn(A.w, odotn);
    // t > eps needs num and ddotn of one sign; this rejects without the
    // divide exactly where the divide's sign would (|ddotn| > eps > 0).
    if (!(ddotn > kKdEps || ddotn < -kKdEps)) return false;
    if constexpr (FLAG) {
        const float4 B = __ldg(&s.tri1[k]);
        const float4 C = __ldg(&s.tri2[k]);
        const int drop = __float_as_uint(C.w) & 3;
        const int c0 = drop == 2 ? 0 : drop + 1;
        const int c1 = drop == 0 ? 2 : drop - 1;
        const float t = __fdiv_rn(num, ddotn);
        const float h1 = __fadd_rn(sel3(c0, r.ox, r.oy, r.oz), __fmul_rn(t, sel3(c0, r.dx, r.dy, r.dz)));
        const float h2 = __fadd_rn(sel3(c1, r.ox, r.oy, r.oz), __fmul_rn(t, sel3(c1, r.dx, r.dy, r.dz)));
        const float b0 = __fadd_rn(__fadd_rn(__fmul_rn(B.x, h1), __fmul_rn(B.y, h2)), B.z);
        const float b1 = __fadd_rn(__fadd_rn(__fmul_rn(B.w, h1), __fmul_rn(C.x, h2)), C.y);
        const float m = nc->m, tm = m * fmaxf(1.0f, fabsf(nc->thi));
        const float sum = __fadd_rn(b0, b1);
        const bool out = b0 < -m || b1 < -m || sum > 1.0f + m || t < nc->tlo - tm || t > nc->thi + tm;
        const bool in = b0 > m && b1 > m && sum < 1.0f - m && t > nc->tlo + tm && t < nc->thi - tm;
        if (!out && !in) nc->near = true;
    }
    if ((__float_as_uint(num) ^ __float_as_uint(ddotn)) & 0x80000000u) return false;
    const float t = __fdiv_rn(num, ddotn);
    if (!(t > kKdEps) || !(t < kKdHuge)) return false;
    const float4 B = __ldg(&s.tri1[k]);
    const float4 C = __ldg(&s.tri2[k]);
    const uint32_t meta = __float_as_uint(C.w);
    const int drop = meta & 3;
    const int c0 = drop == 2 ? 0 : drop + 1;
    const int c1 = drop == 0 ? 2 : drop - 1;
    const float h1 = __fadd_rn(sel3(c0, r.ox, r.oy, r.oz), __fmul_rn(t, sel3(c0, r.dx, r.dy, r.dz)));
    const float h2 = __fadd_rn(sel3(c1, r.ox, r.oy, r.oz), __fmul_rn(t, sel3(c1, r.dx, r.dy, r.dz)));
    float b0 = __fmul_rn(B.x, h1);
    b0 = __fadd_rn(b0, __fmul_rn(B.y, h2));
    b0 = __fadd_rn(b0, B.z);
    if (!(b0 >= kKdEps)) return false;
    float b1 = __fmul_rn(B.w, h1);
    b1 = __fadd_rn(b1, __fmul_rn(C.x, h2));
    b1 = __fadd_rn(b1, C.y);
    if (!(b1 >= kKdEps)) return false;
    if (!(__fadd_rn(b1, b0) <= 1.0f)) return false;
    t_out = t;
    meta_out = meta;
    orig_out = __float_as_int(C.z);
    return true;
}

// a * b + c per half, each half rounded once: one issue slot for the two.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(r)
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
          "l"(*reinterpret_cast<const unsigned long long *>(&b)),
          "l"(*reinterpret_cast<const unsigned long long *>(&c)));
    return *reinterpret_cast<const float2 *>(&r);
}

// Whether the segment meets one box within [lo, hi]: p = (near.x, near.y,
// far.x, far.y), z = (near.z, far.z) as the ray's octant orders them.
__device__ __forceinline__ bool box_hit(const float4 &p, float zn, float zf, const RayState &r, float lo, float hi) {
    const float2 ixy = make_float2(r.ix, r.iy), nxy = make_float2(r.nox, r.noy);
    const float2 n = fma2(make_float2(p.x, p.y), ixy, nxy), f = fma2(make_float2(p.z, p.w), ixy, nxy);
    const float2 z = fma2(make_float2(zn, zf), make_float2(r.iz, r.iz), make_float2(r.noz, r.noz));
    return fmaxf(fmaxf(fmaxf(n.x, n.y), z.x), lo) <= fminf(fminf(fminf(f.x, f.y), z.y), hi);
}

// The same for planes as they lie (low, high), and where the segment enters.
__device__ __forceinline__ bool box_meet(const float4 &p, float zl, float zh, const RayState &r, float lo, float hi,
                                         float &enter) {
    const float2 ixy = make_float2(r.ix, r.iy), nxy = make_float2(r.nox, r.noy);
    const float2 a = fma2(make_float2(p.x, p.y), ixy, nxy), b = fma2(make_float2(p.z, p.w), ixy, nxy);
    const float2 z = fma2(make_float2(zl, zh), make_float2(r.iz, r.iz), make_float2(r.noz, r.noz));
    enter = fmaxf(fmaxf(fminf(a.x, b.x), fminf(a.y, b.y)), fmaxf(fminf(z.x, z.y), lo));
    return enter <= fminf(fminf(fmaxf(a.x, b.x), fmaxf(a.y, b.y)), fminf(fmaxf(z.x, z.y), hi));
}

// The deepest inner node whose box, and every box above it, holds the point
// (of two children that do, the one with the smaller box): where walk()
// best starts for segments from there.
__device__ inline int start_node(const DeviceBvh &s, float x, float y, float z) {
    if (s.ntris == 0) return 0;
    auto inside = [&](const float4 &p, float zn, float zf) {
        return x >= p.x && x <= p.z && y >= p.y && y <= p.w && z >= zn && z <= zf;
    };
    auto half_area = [](const float4 &p, float zn, float zf) {
        const float a = p.z - p.x, b = p.w - p.y, c = zf - zn;
        return a * b + b * c + c * a;
    };
    int at = 0;
    while (true) {
        const float4 *nd = s.nodes + 4 * at;  // octant 0: near is low, far is high
        const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2);
        const int2 ref = __ldg(reinterpret_cast<const int2 *>(nd + 3));
        const bool i0 = inside(a, c.x, c.y), i1 = inside(b, c.z, c.w);
        if (!i0 && !i1) return at;
        const bool second = i1 && (!i0 || half_area(b, c.z, c.w) < half_area(a, c.x, c.y));
        const int next = second ? ref.y : ref.x;
        if (next < 0) return at;
        at = next;
    }
}

// The triangles of the leaf `ref`.  Accepts a hit (t, orig) when t >= tmin and
// (t, orig) is lexicographically below the current best (thi, best_orig);
// best_orig = -1 makes the window half-open, [tmin, thi).  ANY stops at the
// first acceptance; otherwise the best is kept.  Returns whether anything was
// accepted.
template <bool ANY, bool FLAG>
__device__ __forceinline__ bool test_leaf(const DeviceBvh &s, const int32_t *__restrict__ tri_id, const RayState &r,
                                          float tmin, int32_t skip_id, int ref, float &thi, int32_t &best_orig,
                                          uint32_t &best_meta, NearCheck *nc, int *at) {
    const int packed = ~ref;
    const int first = packed >> 3;
    const int count = (packed & 7) + 1;
    bool hit = false;
    for (int k = first; k < first + count; k++) {
        float t;
        uint32_t meta;
        int32_t orig;
        if (!kd_hit<FLAG>(s, k, r, t, meta, orig, nc)) continue;
        if (!(t >= tmin)) continue;
        if (!(t < thi || (t == thi && orig < best_orig))) continue;
        if (skip_id != -1 && __ldg(&tri_id[orig]) == skip_id) continue;
        hit = true;
        thi = t;
        best_orig = orig;
        best_meta = meta;
        if (at) *at = k;
        if (ANY) return true;
    }
    return hit;
}

// One walk of one BVH: the leaves whose boxes the segment meets within
// [tmin, thi], which shrinks with every hit that is kept.  Returns whether
// anything was accepted.
//
// walk_octants, for scenes of up to kOctantTriangles triangles: of two
// children the segment meets, the one nearer along its octant's diagonal is
// entered first.
//
// UP: the walk starts with the subtree of inner node `start`, then takes the
// nodes that lead up from it (vrad_internal.cuh), each holding the next two
// siblings of the path to the root.  Whatever the start, subtree and
// siblings are the whole tree, so the answer does not depend on it.  A
// segment that starts near its origin's leaf and is blocked there never
// visits the top of the tree: on the 8x8 room grid 6.8 nodes and 5.1
// siblings a transfer ray against 15.9 nodes from the root, 6.1 and 3.7 a
// sky ray against 13.1.  Without UP it starts at the root: a caller that
// traces few rays from a point does not earn the search for the start.
//
// What bounds it: a visit hands every lane its own copy of the node, 56
// bytes a lane through L1's 128 bytes a clock (14 cycles a warp, however
// coherent its rays; k_transfer 88 % of that rate), then issue slots.  Hence
// boxes stored as the near and far planes of the ray's octant, children in
// its order (six packed FMAs and eight min/max a visit; no swap of planes,
// no order to compare), and an inner loop that takes all lanes through
// nodes until each has a leaf or is done, so that the triangle test runs
// once for the warp.  Against a walk of canonical nodes from the root: the
// 8x8 room grid's transfer build 62.4 -> 54.3 ms by the octants and the loop,
// 47.6 ms with UP; the 4x4 grid's direct light with a soft sun 40.5 -> 23.9
// ms with all three; 4.2 M closest hits 375 -> 291 us.  Four-wide nodes of the
// same layout gave 57.8 ms for the transfer build, one 32-byte load for two
// 16-byte ones nothing.
template <bool ANY, int STRIDE = kBlock, bool UP = false, bool FLAG = false>
__device__ __forceinline__ bool walk_octants(const DeviceBvh &s, const int32_t *__restrict__ tri_id,
                                     const RayState &r, float tmin, int32_t skip_id, int start, int *stack,
                                     float &thi, int32_t &best_orig, uint32_t &best_meta,
                                     NearCheck *nc = nullptr, int *at = nullptr) {
    constexpr int kEnd = INT32_MIN;
    const float4 *nodes = s.nodes + 8 * (size_t)(r.octant() * s.inner);
    bool hit = false;
    int sp = 0;
    int ref = start;
    if (UP && start > 0) {
        stack[0] = s.inner + start;
        sp = 1;
    }
    while (true) {
        float lo = tmin, hi = thi;
        if constexpr (FLAG) {
            // The recheck also wants the triangles just past either end.
            const float tm = nc->m * fmaxf(1.0f, fabsf(thi));
            lo -= tm;
            hi += tm;
        }
        while (ref >= 0) {
            const float4 *nd = nodes + 4 * ref;
            const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2);
            const int2 child = __ldg(reinterpret_cast<const int2 *>(nd + 3));
            if (UP && ref >= s.inner) {
                const int next = __ldg(reinterpret_cast<const int *>(nd + 3) + 2);
                if (next >= 0) {
                    stack[sp * STRIDE] = next;
                    sp++;
                }
            }
            const bool h0 = box_hit(a, c.x, c.y, r, lo, hi), h1 = box_hit(b, c.z, c.w, r, lo, hi);
            ref = child.y;
            if (h0) {
                if (h1) {
                    stack[sp * STRIDE] = child.y;
                    sp++;
                }
                ref = child.x;
            } else if (!h1) {
                ref = kEnd;
                if (sp) {
                    sp--;
                    ref = stack[sp * STRIDE];
                }
            }
        }
        if (ref == kEnd) return hit;
        if (test_leaf<ANY, FLAG>(s, tri_id, r, tmin, skip_id, ref, thi, best_orig, best_meta, nc, at)) {
            hit = true;
            if (ANY) return true;
        }
        if (sp == 0) return hit;
        sp--;
        ref = stack[sp * STRIDE];
    }
}

// The same walk from the root over one copy of the nodes, for scenes of more
// than kOctantTriangles triangles: of two children the segment meets, the one
// that it enters first, or with FAR the other (the gather's segments, measured
// below).
//
// What bounds it: the nodes come from L2, and a ray visits thirty and more of
// them.  Eight copies leave L1 little to keep, and past 100 k triangles fill
// the L2; and where a ray seldom meets a triangle, lanes that wait for one
// another's leaves cost more than tests at part of the warp.  Triangle soups
// (2 M rays, ms; octants, then this, any hit and closest; rays in random
// directions, then warps of neighbouring rays):
//   10 k   1.07 1.13, 0.94 1.03;   0.39 0.40, 0.37 0.39
//   20 k   1.26 1.33, 1.13 1.24;   0.50 0.51, 0.49 0.52
//   100 k  1.67 1.82, 1.55 1.74;   0.90 0.97, 0.82 0.92
//   400 k  2.52 2.89, 1.96 2.21;   1.56 1.73, 1.28 1.44
//   1.5 M  3.93 4.36, 2.68 3.18;   2.00 2.34, 1.75 2.05
// Light passes of the room grids with so many small triangles added: 4x4 grid,
// 5 k in all 44.8 and 46.4 ms, 18 k 92.1 and 81.8, 102 k 130 and 108, 1.5 M
// 504 and 355; 8x8 grid, 9 k 84.4 and 99.9, 17 k 133 and 146, 29 k 179 and
// 180.  Started from the origin's leaf as walk_octants' UP, the 1.5 M took 444
// with the nearer child first and 452 with the farther.
template <bool ANY, int STRIDE, bool FAR, bool FLAG>
__device__ __forceinline__ bool walk_one(const DeviceBvh &s, const int32_t *__restrict__ tri_id, const RayState &r,
                                         float tmin, int32_t skip_id, int *stack, float &thi, int32_t &best_orig,
                                         uint32_t &best_meta, NearCheck *nc, int *at) {
    bool hit = false;
    int sp = 0;
    int ref = 0;
    while (true) {
        if (ref >= 0) {
            const float4 *nd = s.nodes + 4 * (size_t)ref;
            const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2);
            const int2 child = __ldg(reinterpret_cast<const int2 *>(nd + 3));
            float lo = tmin, hi = thi, e0, e1;
            if constexpr (FLAG) {
                // The recheck also wants the triangles just past either end.
                const float tm = nc->m * fmaxf(1.0f, fabsf(thi));
                lo -= tm;
                hi += tm;
            }
            const bool h0 = box_meet(a, c.x, c.y, r, lo, hi, e0), h1 = box_meet(b, c.z, c.w, r, lo, hi, e1);
            if (h0 && h1) {
                const bool second = FAR ? e1 > e0 : e1 < e0;
                stack[sp * STRIDE] = second ? child.x : child.y;
                sp++;
                ref = second ? child.y : child.x;
                continue;
            }
            if (h0) {
                ref = child.x;
                continue;
            }
            if (h1) {
                ref = child.y;
                continue;
            }
        } else if (test_leaf<ANY, FLAG>(s, tri_id, r, tmin, skip_id, ref, thi, best_orig, best_meta, nc, at)) {
            hit = true;
            if (ANY) return true;
        }
        if (sp == 0) return hit;
        sp--;
        ref = stack[sp * STRIDE];
    }
}

// UP and start are walk_octants', FAR walk_one's.
template <bool ONE, bool ANY, int STRIDE = kBlock, bool UP = false, bool FLAG = false, bool FAR = false>
__device__ __forceinline__ bool walk(const DeviceBvh &s, const int32_t *__restrict__ tri_id, const RayState &r, float tmin,
                                     int32_t skip_id, int start, int *stack, float &thi, int32_t &best_orig,
                                     uint32_t &best_meta, NearCheck *nc = nullptr, int *at = nullptr) {
    if constexpr (ONE)
        return walk_one<ANY, STRIDE, FAR, FLAG>(s, tri_id, r, tmin, skip_id, stack, thi, best_orig, best_meta, nc, at);
    else
        return walk_octants<ANY, STRIDE, UP, FLAG>(s, tri_id, r, tmin, skip_id, start, stack, thi, best_orig, best_meta,
                                                   nc, at);
}

// One ray against the scene.  Modes:
//   kModeAny      any accepted hit in [tmin, reach), opaque or sky;
//   kModeClosest  the smallest (t, original index) in [tmin, reach);
//   kModeSkyPass  blocked iff that smallest hit exists and is opaque: the
//                 nearest sky hit (t_s, i_s) is found first, then any
//                 opaque hit below it decides, so the opaque walk stops at
//                 its first acceptance.
// start: where the opaque tree's walk starts (start_node of the ray's
// origin, or 0).  The sky tree is small and flat: its walk starts at the
// root.  kModeAny leaves in *at (when given) the opaque triangle that was
// hit, by its place in the tree's arrays; a sky hit leaves it as it is.
// FAR: which child the opaque any-hit walk over one copy enters first.
template <bool ONE, int MODE, int STRIDE = kBlock, bool UP = false, bool FAR = false>
__device__ __forceinline__ void trace_ray(const DeviceScene &s, const RayState &r, float tmin,
                                          float reach, int32_t skip_id, int start, int *stack,
                                          bool &hit, float &best_t,
                                          int32_t &best_orig, uint32_t &best_meta, int *at = nullptr) {
    best_t = reach;
    best_orig = -1;
    best_meta = 0;
    hit = false;
    if (MODE == kModeAny) {
        if (s.opaque.ntris)
            hit = walk<ONE, true, STRIDE, UP, false, FAR>(s.opaque, s.tri_id, r, tmin, skip_id, start, stack, best_t, best_orig, best_meta,
                                         nullptr, at);
        if (!hit && s.sky.ntris)
            hit = walk<ONE, true, STRIDE>(s.sky, s.tri_id, r, tmin, skip_id, 0, stack, best_t, best_orig, best_meta);
    } else if (MODE == kModeClosest) {
        if (s.opaque.ntris)
            hit = walk<ONE, false, STRIDE, UP>(s.opaque, s.tri_id, r, tmin, skip_id, start, stack, best_t, best_orig, best_meta);
        if (s.sky.ntris)
            hit |= walk<ONE, false, STRIDE>(s.sky, s.tri_id, r, tmin, skip_id, 0, stack, best_t, best_orig, best_meta);
    } else {
        if (s.sky.ntris)
            walk<ONE, false, STRIDE>(s.sky, s.tri_id, r, tmin, skip_id, 0, stack, best_t, best_orig, best_meta);
        // Blocked iff an opaque hit sorts before the nearest sky hit.
        if (s.opaque.ntris)
            hit = walk<ONE, true, STRIDE, UP, false, FAR>(s.opaque, s.tri_id, r, tmin, skip_id, start, stack, best_t, best_orig, best_meta);
    }
}


// kModeAny with the FP64 recheck's flag: the same walks and answer as
// trace_ray<kModeAny>, every box widened by the margin at both ends.
template <bool ONE, int STRIDE = kBlock>
__device__ __forceinline__ void trace_ray_flagged(const DeviceScene &s, const RayState &r, float tmin, float reach,
                                                  int32_t skip_id, int *stack, bool &hit, NearCheck &nc) {
    float best_t = reach;
    int32_t best_orig = -1;
    uint32_t best_meta = 0;
    hit = false;
    if (s.opaque.ntris)
        hit = walk<ONE, true, STRIDE, false, true>(s.opaque, s.tri_id, r, tmin, skip_id, 0, stack, best_t, best_orig, best_meta,
                                       &nc);
    if (!hit && s.sky.ntris)
        hit = walk<ONE, true, STRIDE, false, true>(s.sky, s.tri_id, r, tmin, skip_id, 0, stack, best_t, best_orig, best_meta, &nc);
}

// How many octants the directions of the warp's `live` lanes lie in.
__device__ __forceinline__ int octants_of(unsigned live, const RayState &r) {
    const int oct = r.octant();
    if (__all_sync(live, oct == __shfl_sync(live, oct, __ffs(live) - 1))) return 1;
    const unsigned same = __match_any_sync(live, oct);
    return __popc(__ballot_sync(live, (same & ((1u << (threadIdx.x & 31)) - 1u)) == 0));
}

__device__ __forceinline__ RayState make_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
    RayState r;
    r.ox = ox;
    r.oy = oy;
    r.oz = oz;
    r.dx = dx;
    r.dy = dy;
    r.dz = dz;
    r.ix = recip_saturate(dx);
    r.iy = recip_saturate(dy);
    r.iz = recip_saturate(dz);
    r.nox = -ox * r.ix;
    r.noy = -oy * r.iy;
    r.noz = -oz * r.iz;
    return r;
}

}  // namespace vrad
