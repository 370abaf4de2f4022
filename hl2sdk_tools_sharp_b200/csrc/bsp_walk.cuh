// bsp_walk.cuh -- the BSP surface walk as device functions: stock vrad's
// CLightSurface over EnumerateNodesAlongRay, shared by the closest-hit
// kernel (bsp_trace.cu) and the leaf ambient sample (ambient.cu).
//
// Reference behaviour restated (muflub/hl2sdk_tools_sharp,
// MapTools/Tracing/BspSurfaceTracer.cs, and its leaf-ambient twin
// MapTools/Rad/Ambient/AmbientRayTracer.cs:107-464):
//   the walk (BspSurfaceTracer.cs:233-357, AmbientRayTracer.cs:148-275):
//     front-to-back over the map's BSP tree, one plane test per node (the
//     axial shortcut reads the component), a ray straddling a node within
//     TEST_EPSILON (1/32) of it descends the near side first with the split
//     pending on a stack;
//   EnumerateLeaf (:408-464 / :330-400): the leaf's faces, backface cull,
//     the crossing fraction inside the leaf's segment and below the best so
//     far, the lightmap rectangle test, whose offsets into the rectangle are
//     the hit's luxel coordinates (m_LuxelCoord);
//   EnumerateNode (:365-406 / :279-328): a pending split's on-node faces at
//     the split point, lit faces first (the first hit ends the walk), then
//     sky faces by their windings (the last that passes ends it; a sky hit
//     has no luxel);
// Correct mode (exact normalise in the sky test), every float operation an
// explicitly rounded intrinsic in the reference's order, so a face, a
// fraction and a luxel coordinate are stock's bits.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "bsp_trace.cuh"

namespace vrad {
namespace bspwalk {

constexpr float kTestEpsilon = 0.03125f;  // TEST_EPSILON
constexpr int kStack = 64;

struct Walk {
    float ox, oy, oz, dx, dy, dz;
    float hit_frac, min_frac;
    int32_t surface;
    bool has_luxel;
    float luxel_s, luxel_t;
};

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// TestPointAgainstSurface: inside the face's lightmap rectangle; ds and dt
// are the point's offsets from the rectangle's mins.
__device__ __forceinline__ bool in_surface(const float4 *__restrict__ surface, float px, float py, float pz, float &ds,
                                           float &dt) {
    const float4 S = __ldg(&surface[1]), T = __ldg(&surface[2]), R = __ldg(&surface[3]);
    const float sc = __fadd_rn(dot3(px, py, pz, S.x, S.y, S.z), S.w);
    const float tc = __fadd_rn(dot3(px, py, pz, T.x, T.y, T.z), T.w);
    if (sc < R.x || tc < R.y) return false;
    ds = __fsub_rn(sc, R.x);
    dt = __fsub_rn(tc, R.y);
    return ds <= R.z && dt <= R.w;
}

__device__ __forceinline__ void normalise3(float &x, float &y, float &z) {
    const float len = __fsqrt_rn(dot3(x, y, z, x, y, z));
    if (len == 0.0f) {
        x = y = z = 0.0f;
        return;
    }
    x = __fdiv_rn(x, len);
    y = __fdiv_rn(y, len);
    z = __fdiv_rn(z, len);
}

struct V3 {
    float x, y, z;
};

// Cross(edge, to_pt) of the edge from a to b and the point p (Vec3.Cross's
// operand order).
__device__ __forceinline__ V3 edge_cross(const float4 &a, const float4 &b, float px, float py, float pz) {
    const float ex = __fsub_rn(b.x, a.x), ey = __fsub_rn(b.y, a.y), ez = __fsub_rn(b.z, a.z);
    const float tx = __fsub_rn(px, a.x), ty = __fsub_rn(py, a.y), tz = __fsub_rn(pz, a.z);
    return {__fsub_rn(__fmul_rn(ey, tz), __fmul_rn(ez, ty)), __fsub_rn(__fmul_rn(ez, tx), __fmul_rn(ex, tz)),
            __fsub_rn(__fmul_rn(ex, ty), __fmul_rn(ey, tx))};
}
__device__ __forceinline__ float one_norm(const V3 &v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); }

// TestPointAgainstSkySurface: every edge's normal on the first edge's side,
// by the sign of the normalised crosses' dot product.  The crosses are
// normalised (a square root and six divides an edge) only where their plain
// dot product does not settle that sign: both products' rounding is below
// 1e-6 of the one-norms' product, a hundredth of the margin here, as long
// as no square over- or underflows.
__device__ inline bool in_sky(const DeviceBsp &g, int face, float px, float py, float pz) {
    const int2 run = __ldg(&g.sky_run[face]);
    if (run.y < 2) return false;
    const float4 *p = g.sky_points + run.x;
    const float4 p0 = __ldg(&p[0]);
    float4 at = __ldg(&p[1]);
    V3 first = edge_cross(p0, at, px, py, pz);
    const float n0 = one_norm(first);
    bool unit = false;  // first is normalised
    for (int i = 1; i < run.y; i++) {
        const float4 next = i + 1 < run.y ? __ldg(&p[i + 1]) : p0;
        V3 c = edge_cross(at, next, px, py, pz);
        at = next;
        const float n1 = one_norm(c);
        if (!unit && n0 > 1e-12f && n0 < 1e12f && n1 > 1e-12f && n1 < 1e12f) {
            const float d = dot3(c.x, c.y, c.z, first.x, first.y, first.z);
            if (fabsf(d) > 1e-4f * n0 * n1) {
                if (d < 0.0f) return false;
                continue;
            }
        }
        if (!unit) normalise3(first.x, first.y, first.z);
        unit = true;
        normalise3(c.x, c.y, c.z);
        if (dot3(c.x, c.y, c.z, first.x, first.y, first.z) < 0.0f) return false;
    }
    return true;
}

// The face lists are short but for a few (a floor's node holds 103 faces on
// dm_lockdown, a leaf 147), and a lane that works through one alone holds
// its warp.  Where at most kFewLong lanes have a list of kLong faces or
// more, the whole warp tests each of those lists, 32 faces at a time; where
// more lanes have one (rays that go the same way) each lane does its own.
constexpr int kLong = 16, kFewLong = 8;

// The lanes whose list the warp takes together.
__device__ __forceinline__ unsigned long_lists(int count) {
    const unsigned m = __ballot_sync(0xffffffffu, count >= kLong);
    return __popc(m) <= kFewLong ? m : 0u;
}

// EnumerateNode for every lane with a node (node >= 0), whole warps: done is
// set where the walk ends.
__device__ inline void visit_nodes(const DeviceBsp &g, Walk &c, int node, float f, bool &done) {
    int solid = 0, sky = 0, at = 0;
    float px = 0.0f, py = 0.0f, pz = 0.0f;
    if (node >= 0) {
        const float4 B = __ldg(&g.nodes[2 * node + 1]);
        const int packed = __float_as_int(B.w);
        solid = packed & 0x7FFF;
        sky = (packed >> 15) & 0x7FFF;
        at = __float_as_int(B.z);
        if (solid | sky) {
            px = __fadd_rn(c.ox, __fmul_rn(f, c.dx));
            py = __fadd_rn(c.oy, __fmul_rn(f, c.dy));
            pz = __fadd_rn(c.oz, __fmul_rn(f, c.dz));
        }
    }
    const int lane = threadIdx.x & 31;
    unsigned together = long_lists(solid);
    const bool mine = !((together >> lane) & 1u);
    int hit = -1;
    float ds = 0.0f, dt = 0.0f;
    for (; together; together &= together - 1) {
        const int l = __ffs(together) - 1;
        const float x = __shfl_sync(0xffffffffu, px, l), y = __shfl_sync(0xffffffffu, py, l),
                    z = __shfl_sync(0xffffffffu, pz, l);
        const int n = __shfl_sync(0xffffffffu, solid, l), first = __shfl_sync(0xffffffffu, at, l);
        for (int i = 0; i < n; i += 32) {
            float s = 0.0f, t = 0.0f;
            const bool in = i + lane < n && in_surface(g.node_surf + 4 * (size_t)(first + i + lane), x, y, z, s, t);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (!m) continue;
            const int w = __ffs(m) - 1;  // the first in list order
            s = __shfl_sync(0xffffffffu, s, w);
            t = __shfl_sync(0xffffffffu, t, w);
            if (lane == l) {
                hit = i + w;
                ds = s;
                dt = t;
            }
            break;
        }
    }
    if (mine) {
        const float4 *surf = g.node_surf + 4 * (size_t)at;
        for (int i = 0; i < solid; i++)
            if (in_surface(surf + 4 * i, px, py, pz, ds, dt)) {
                hit = i;
                break;
            }
    }
    if (hit >= 0) {
        c.hit_frac = f;
        c.surface = __ldg(&g.node_faces[at + hit]);
        c.has_luxel = true;
        c.luxel_s = ds;
        c.luxel_t = dt;
        done = true;
    } else if (sky) {
        int sky_hit = -1;
        for (int i = 0; i < sky; i++) {
            const int face = __ldg(&g.node_faces[at + solid + i]);
            if (in_sky(g, face, px, py, pz)) sky_hit = face;
        }
        c.surface = sky_hit;
        done = sky_hit != -1;
    }
}

// One face of a leaf: the crossing fraction inside the leaf's segment, above
// the floor and below `best`, and the point inside the face.
__device__ __forceinline__ bool leaf_face(const float4 *__restrict__ surf, float ox, float oy, float oz, float dx,
                                          float dy, float dz, float start, float end, float best, float min_frac,
                                          float &mid, float &ds, float &dt) {
    const float4 P = __ldg(surf);
    const float ddn = dot3(dx, dy, dz, P.x, P.y, P.z);
    if (ddn > 0.0f) return false;
    const float sdn = dot3(ox, oy, oz, P.x, P.y, P.z);
    const float front = __fsub_rn(__fadd_rn(sdn, __fmul_rn(start, ddn)), P.w);
    const float back = __fsub_rn(__fadd_rn(sdn, __fmul_rn(end, ddn)), P.w);
    const bool side = front < 0.0f;
    if ((back < 0.0f) == side) return false;
    const float f = __fdiv_rn(front, __fsub_rn(front, back));
    mid = __fadd_rn(__fmul_rn(start, __fsub_rn(1.0f, f)), __fmul_rn(end, f));
    if (mid >= best || mid < min_frac) return false;
    const float px = __fadd_rn(ox, __fmul_rn(mid, dx)), py = __fadd_rn(oy, __fmul_rn(mid, dy)),
                pz = __fadd_rn(oz, __fmul_rn(mid, dz));
    return in_surface(surf, px, py, pz, ds, dt);
}

// EnumerateLeaf for every lane with a leaf (leaf >= 0), whole warps: done is
// set where the walk ends.  The nearest accepted face is the answer, the
// first in list order among equals.
__device__ inline void visit_leaves(const DeviceBsp &g, Walk &c, int leaf, float start, float end, bool &done) {
    int2 run = make_int2(0, 0);
    if ((unsigned)leaf < (unsigned)g.nleaves) run = __ldg(&g.leaf_run[leaf]);
    const int lane = threadIdx.x & 31;
    unsigned together = long_lists(run.y);
    const bool mine = !((together >> lane) & 1u);
    int hit = -1;
    float best = c.hit_frac, bs = 0.0f, bt = 0.0f;
    for (; together; together &= together - 1) {
        const int l = __ffs(together) - 1;
        auto from = [&](float v) { return __shfl_sync(0xffffffffu, v, l); };
        const float ox = from(c.ox), oy = from(c.oy), oz = from(c.oz), dx = from(c.dx), dy = from(c.dy),
                    dz = from(c.dz), s0 = from(start), s1 = from(end), lim = from(best), low = from(c.min_frac);
        const int n = __shfl_sync(0xffffffffu, run.y, l), first = __shfl_sync(0xffffffffu, run.x, l);
        // Each lane's nearest of its faces (every 32nd), then the warp's.
        int mi = INT32_MAX;
        float mm = lim, ms = 0.0f, mt = 0.0f;
        for (int i = lane; i < n; i += 32) {
            float mid, ds, dt;
            if (leaf_face(g.leaf_surf + 4 * (size_t)(first + i), ox, oy, oz, dx, dy, dz, s0, s1, mm, low, mid, ds, dt)) {
                mm = mid;
                mi = i;
                ms = ds;
                mt = dt;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, mm, o), os = __shfl_xor_sync(0xffffffffu, ms, o),
                        ot = __shfl_xor_sync(0xffffffffu, mt, o);
            const int oi = __shfl_xor_sync(0xffffffffu, mi, o);
            if (oi != INT32_MAX && (mi == INT32_MAX || om < mm || (om == mm && oi < mi))) {
                mm = om;
                mi = oi;
                ms = os;
                mt = ot;
            }
        }
        if (lane == l && mi != INT32_MAX) {
            hit = mi;
            best = mm;
            bs = ms;
            bt = mt;
        }
    }
    if (mine) {
        for (int i = 0; i < run.y; i++) {
            float mid, ds, dt;
            if (leaf_face(g.leaf_surf + 4 * (size_t)(run.x + i), c.ox, c.oy, c.oz, c.dx, c.dy, c.dz, start, end, best,
                          c.min_frac, mid, ds, dt)) {
                hit = i;
                best = mid;
                bs = ds;
                bt = dt;
            }
        }
    }
    if (hit >= 0) {
        c.hit_frac = best;
        c.surface = __ldg(&g.leaf_faces[run.x + hit]);
        c.has_luxel = true;
        c.luxel_s = bs;
        c.luxel_t = bt;
        done = true;
    }
}

struct Pending {
    int visit, far_child;
    float split, end;
};

// The whole walk from c's origin along c's delta, for the lanes with live
// set; every lane of the warp calls it.  Returns false when the lane's walk
// needed more than kStack pending splits (c then holds no answer).
__device__ inline bool walk(const DeviceBsp &g, Walk &c, bool live) {
    Pending stack[kStack];
    int sp = 0, node = 0;
    float start = 0.0f, end = 1.0f;
    bool done = !live, ok = true;
    while (__any_sync(0xffffffffu, !done)) {
        while (!done && node >= 0) {
            const float4 A = __ldg(&g.nodes[2 * node]), B = __ldg(&g.nodes[2 * node + 1]);
            const int packed = __float_as_int(B.w);
            const unsigned axis = (unsigned)packed >> 30;
            float sdn, ddn;
            if (axis == 3) {
                sdn = dot3(c.ox, c.oy, c.oz, A.x, A.y, A.z);
                ddn = dot3(c.dx, c.dy, c.dz, A.x, A.y, A.z);
            } else if (axis == 0) {
                sdn = c.ox;
                ddn = c.dx;
            } else if (axis == 1) {
                sdn = c.oy;
                ddn = c.dy;
            } else {
                sdn = c.oz;
                ddn = c.dz;
            }
            const float front = __fsub_rn(__fadd_rn(sdn, __fmul_rn(start, ddn)), A.w);
            const float back = __fsub_rn(__fadd_rn(sdn, __fmul_rn(end, ddn)), A.w);
            const int child0 = __float_as_int(B.x), child1 = __float_as_int(B.y);
            if (front <= -kTestEpsilon && back <= -kTestEpsilon) {
                node = child1;
                continue;
            }
            if (front >= kTestEpsilon && back >= kTestEpsilon) {
                node = child0;
                continue;
            }
            const bool side = front < 0.0f;
            float split;
            if (ddn == 0.0f) {
                split = 1.0f;
            } else {
                split = __fdiv_rn(__fsub_rn(A.w, sdn), ddn);
                if (split < 0.0f) split = 0.0f;
                else if (split > 1.0f) split = 1.0f;
            }
            if (sp >= kStack) {
                ok = false;
                done = true;
                break;
            }
            stack[sp++] = Pending{node, side ? child0 : child1, split, end};
            node = side ? child1 : child0;
            end = split;
        }
        __syncwarp();
        visit_leaves(g, c, done ? -1 : -node - 1, start, end, done);
        Pending e{-1, 0, 0.0f, 0.0f};
        if (!done) {
            if (sp == 0) done = true;
            else e = stack[--sp];
        }
        visit_nodes(g, c, e.visit, e.split, done);
        node = e.far_child;
        start = e.split;
        end = e.end;
    }
    return ok;
}

}  // namespace bspwalk
}  // namespace vrad
