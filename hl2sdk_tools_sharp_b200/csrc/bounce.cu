// bounce.cu -- the radiosity bounce: the patches' direct light, the
// transfers (candidate pairs, their rays and form factors), the bounces,
// and the tables the final pass reads the bounced light through.
//
// Reference behaviour restated (muflub/hl2sdk_tools_sharp, MapTools/Rad):
//   PatchLighting.BuildPatchLights / AddSampleToPatch  Light/PatchLighting.cs:65-249
//   Radiosity.MoveDirectLightToEmission / GatherLight /
//             CollectLight / BounceAsync               Bounce/Radiosity.cs:132-316
//   VisMatrix.ReceiverOrder / FacesInRow / Enumerator.Run /
//             TestPatchToFace / TestPatchToPatch /
//             TransferRay / MakeTransfers / MakeTransfer /
//             MakeScales                               Bounce/VisMatrix.cs:180-1004
//   FormFactors.DiffToDiff / PolyToDiff                Bounce/FormFactors.cs:58-140
//   DetMathF.Asin (correctly rounded)                  MapFormats/Numerics/DetMathF.cs:141-164
//   FinalLightFace.BuildPatchRadial / AddFacePatches /
//             PatchLightmapCoordRange                  Final/FinalLightFace.cs:393-540
// with the reference's default settings: no compliance quirks (the
// receiver's plane normal in the plane test, true divides in the transfer
// rays, sines above one clamped), the exact normalise, bounces > 0.
//
// Every float operation of those routines is an explicitly rounded
// intrinsic, in the reference's association order, and every sum runs in
// the reference's order, so the transfers, the patch light and the stop
// decision are the reference's bits.
//
// Kernels of one light pass (after the direct gather):
//   k_patch_samples   one thread per patch: the face's samples that overlap
//                     it, in sample order (AddSampleToPatch), averaged and
//                     moved to emission
//   k_parents         one block per face: the parents level by level, bottom
//                     up (the direct light's area blends; after each bounce
//                     CollectLight's; the warm start's)
//   k_candidates      one lane per receiver, one walk per warp: the candidate
//                     sources in the enumerator's order (a counting launch
//                     at the upload, a writing one)
//   k_transfer        one thread per candidate: the transfer ray, traced
//                     in-thread, and MakeTransfer for an open pair (by groups
//                     of receivers where there are many)
//   k_transfer_count / k_transfer_write  one warp per receiver: the
//                     accepted pairs compacted in order, capped at
//                     MaxPatches, and MakeScales' ordered sum
//   k_sell_*          the transfer lists copied into slices of 32 receivers
//                     sorted by window and count (SELL-32), once per pass
//   k_gather          one thread per receiver (in the slices' order):
//                     GatherLight's ordered sum from its slice lane, then
//                     CollectLight's leaf update, and fp64 sums of the light
//                     the bounce added, with absolute sums that bound the
//                     reference's float sum
//   k_exact_*         the reference's sequential float sum, run only when
//                     the bound cannot settle the stop rule

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "bounce.cuh"
#include "device_pool.h"
#include "context.cuh"
#include "final.cuh"
#include "detmath.cuh"
#include "mlp.cuh"
#include "patches.h"
#include "traverse.cuh"
#include "world.h"

namespace vrad {

namespace {

constexpr int kBounceBlock = 128;
constexpr int kEnumStack = 64;  // patch tree depth the candidate walk holds

// ---- float and double-double helpers ----------------------------------------

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(const float4 &a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ F3 add3(F3 a, F3 b) { return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)}; }
__device__ __forceinline__ F3 sub3(F3 a, F3 b) { return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)}; }
__device__ __forceinline__ F3 mul3(F3 a, float s) { return {__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)}; }
__device__ __forceinline__ float dot3(F3 a, F3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ F3 cross3(F3 a, F3 b) {
    return {__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
            __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x))};
}
// Vec3.Normalise: exact length, three true divides, zero for zero.
__device__ __forceinline__ F3 normalise3(F3 a, float &len) {
    len = __fsqrt_rn(dot3(a, a));
    if (len == 0.0f) return {0.0f, 0.0f, 0.0f};
    return {__fdiv_rn(a.x, len), __fdiv_rn(a.y, len), __fdiv_rn(a.z, len)};
}

// ---- the patches' direct light ----------------------------------------------

// AddSampleToPatch for one leaf patch over its face's samples, in sample
// order, then BuildPatchLights' average and MoveDirectLightToEmission: the
// leaf's direct light, its emission and what it shoots; the bounced total
// starts from zero.  The parents' sums that the reference pushes up are
// replaced by the area blend of their children's averages before anything
// reads them, so only that blend is built (k_parents).
//
// A face has hundreds of samples and a leaf a few cells of them, so where
// the face's samples lie in cell order the leaf looks at the cells in
// reach alone (box, k_patch_boxes): every sample that can pass the overlap
// test lies there, and the cells come in sample order.  On the 8x8 grid of
// rooms a pass takes 235 us, with all of the face's samples 3.1 ms.
__global__ void k_patch_samples(BounceView v, const int4 *__restrict__ box, const int32_t *__restrict__ face_cells,
                                const float4 *__restrict__ frames, const int32_t *__restrict__ cell_sample,
                                const float4 *__restrict__ sample_light, float4 *__restrict__ direct,
                                float4 *__restrict__ total, float4 *__restrict__ emit, float4 *__restrict__ shoot) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.npatches) return;
    total[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int4 tr = __ldg(&v.tree[p]);
    if (tr.y != -1) return;
    float lx = 0.0f, ly = 0.0f, lz = 0.0f, area = 0.0f;
    if (tr.w == 0) {
        const float4 mn = __ldg(&v.mins[p]), mx = __ldg(&v.maxs[p]);
        const int f = __float_as_int(mn.w);
        auto sample = [&](int k) {
            const float4 L = __ldg(&sample_light[k]);
            // VectorAvg: a float divide by 3.
            if (__fdiv_rn(__fadd_rn(__fadd_rn(L.x, L.y), L.z), 3.0f) < 1.0f) return;
            const float a = __ldg(&v.sample_area[k]);
            const float4 P = __ldg(&v.sample_pos[k]);
            const float radius = (float)__ddiv_rn((double)__fsqrt_rn(a), 2.0);
            if (mn.x > __fadd_rn(P.x, radius) || mx.x < __fsub_rn(P.x, radius)) return;
            if (mn.y > __fadd_rn(P.y, radius) || mx.y < __fsub_rn(P.y, radius)) return;
            if (mn.z > __fadd_rn(P.z, radius) || mx.z < __fsub_rn(P.z, radius)) return;
            area = __fadd_rn(area, a);
            lx = __fadd_rn(lx, __fmul_rn(a, L.x));
            ly = __fadd_rn(ly, __fmul_rn(a, L.y));
            lz = __fadd_rn(lz, __fmul_rn(a, L.z));
        };
        const int4 bx = __ldg(&box[p]);
        if (bx.x >= 0) {
            const int base = __ldg(&face_cells[f]), w = __float_as_int(__ldg(&frames[5 * f].w));
            for (int t = bx.y; t < bx.w; t++)
                for (int s = bx.x; s < bx.z; s++) {
                    const int k = __ldg(&cell_sample[base + s + t * w]);
                    if (k >= 0) sample(k);
                }
        } else {
            const int2 fs = __ldg(&v.face_samples[f]);
            for (int k = fs.x; k < fs.x + fs.y; k++) sample(k);
        }
    }
    float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (area != 0.0f) {
        const float scale = (float)__drcp_rn((double)area);
        e = make_float4(__fadd_rn(0.0f, __fmul_rn(lx, scale)), __fadd_rn(0.0f, __fmul_rn(ly, scale)),
                        __fadd_rn(0.0f, __fmul_rn(lz, scale)), 0.0f);
    }
    const float4 r = __ldg(&v.refl[p]);
    direct[p] = e;
    emit[p] = e;
    shoot[p] = make_float4(__fmul_rn(e.x, r.x), __fmul_rn(e.y, r.y), __fmul_rn(e.z, r.z), 0.0f);
}

// A face's luxel coordinates in double: world to luxel (s, t) and how far a
// box of half sizes h reaches in each.
struct Luxels {
    double ox, oy, oz, sx, sy, sz, tx, ty, tz;
    int w, h, min_s, min_t;
    __device__ __forceinline__ Luxels(const float4 *__restrict__ frames, int f) {
        const float4 o = __ldg(&frames[5 * (int64_t)f]), a = __ldg(&frames[5 * (int64_t)f + 1]),
                     b = __ldg(&frames[5 * (int64_t)f + 2]), c = __ldg(&frames[5 * (int64_t)f + 3]);
        ox = o.x, oy = o.y, oz = o.z;
        sx = a.x, sy = a.y, sz = a.z;
        tx = b.x, ty = b.y, tz = b.z;
        w = __float_as_int(o.w);
        h = __float_as_int(a.w);
        min_s = __float_as_int(b.w);
        min_t = __float_as_int(c.w);
    }
    __device__ __forceinline__ double s(double x, double y, double z) const {
        return (x - ox) * sx + (y - oy) * sy + (z - oz) * sz - (double)min_s;
    }
    __device__ __forceinline__ double t(double x, double y, double z) const {
        return (x - ox) * tx + (y - oy) * ty + (z - oz) * tz - (double)min_t;
    }
    __device__ __forceinline__ double reach_s(double x, double y, double z) const {
        return fabs(sx) * x + fabs(sy) * y + fabs(sz) * z;
    }
    __device__ __forceinline__ double reach_t(double x, double y, double z) const {
        return fabs(tx) * x + fabs(ty) * y + fabs(tz) * z;
    }
};

// How a face's samples lie in its cells: (how far a sample's luxel
// coordinates stray from its cell, s and t; the largest radius; 1 when the
// samples are the cells' in cell order, and all of it is finite).  One warp
// per face.
__global__ void k_face_fit(BounceView v, const int32_t *__restrict__ face_cells, const float4 *__restrict__ frames,
                           const int32_t *__restrict__ cell_sample, float4 *__restrict__ fit) {
    const int f = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (f >= v.nfaces) return;
    const int2 fs = __ldg(&v.face_samples[f]);
    const Luxels lx(frames, f);
    const int base = __ldg(&face_cells[f]), n = __ldg(&face_cells[f + 1]) - base;
    double ds = 0.0, dt = 0.0, r = 0.0;
    bool ok = true;
    int last = fs.x - 1, found = 0;  // the last cell's sample so far, samples found
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int c = c0 + lane, k = c < n ? __ldg(&cell_sample[base + c]) : -1;
        const unsigned have = __ballot_sync(kFull, k >= 0), before = have & ((1u << lane) - 1u);
        const int prev = __shfl_sync(kFull, k, before ? 31 - __clz(before) : 0);
        if (k >= 0) {
            ok = ok && k > (before ? prev : last) && k < fs.x + fs.y;
            const float4 P = __ldg(&v.sample_pos[k]);
            ds = fmax(ds, fabs(lx.s(P.x, P.y, P.z) - (double)(c % lx.w)));
            dt = fmax(dt, fabs(lx.t(P.x, P.y, P.z) - (double)(c / lx.w)));
            const double radius = sqrt((double)__ldg(&v.sample_area[k])) * 0.5;
            r = fmax(r, radius);
            ok = ok && isfinite(P.x) && isfinite(P.y) && isfinite(P.z) && isfinite(radius);
        }
        found += __popc(have);
        if (have) last = __shfl_sync(kFull, k, 31 - __clz(have));
    }
    for (int o = 16; o > 0; o >>= 1) {
        ds = fmax(ds, __shfl_xor_sync(kFull, ds, o));
        dt = fmax(dt, __shfl_xor_sync(kFull, dt, o));
        r = fmax(r, __shfl_xor_sync(kFull, r, o));
    }
    ok = __all_sync(kFull, ok) && found == fs.y && ds < 1e6 && dt < 1e6 && r < 1e6;
    // Rounded up: an upper bound is what is kept.
    if (lane == 0) fit[f] = make_float4(__double2float_ru(ds), __double2float_ru(dt), __double2float_ru(r), ok ? 1.0f : 0.0f);
}

// Each leaf patch's cells in reach, [x, z) by [y, w): those whose sample
// could pass the overlap test, that is, lie in the patch's bounds grown by
// the face's largest radius.  The slack of 1e-3 units and 1e-6 of the
// coordinates covers the test's float roundings (half an ulp is 6e-8 of
// them), that of 0.01 luxels the sums here.  x = -1: the face's samples
// don't lie in cell order or something isn't finite, and the patch looks at
// all of them.
__global__ void k_patch_boxes(BounceView v, const float4 *__restrict__ frames, const float4 *__restrict__ fit,
                              int4 *__restrict__ box) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.npatches) return;
    box[p] = make_int4(-1, 0, 0, 0);
    const float4 mn = __ldg(&v.mins[p]), mx = __ldg(&v.maxs[p]);
    const int f = __float_as_int(mn.w);
    const float4 ft = __ldg(&fit[f]);
    if (ft.w == 0.0f) return;
    const Luxels lx(frames, f);
    const double big = fmax(fmax(fmax(fabs((double)mn.x), fabs((double)mn.y)), fabs((double)mn.z)),
                            fmax(fmax(fabs((double)mx.x), fabs((double)mx.y)), fabs((double)mx.z)));
    const double grow = (double)ft.z + 1e-3 + 1e-6 * big;
    const double cx = 0.5 * ((double)mn.x + mx.x), cy = 0.5 * ((double)mn.y + mx.y), cz = 0.5 * ((double)mn.z + mx.z);
    const double hx = fmax(0.5 * ((double)mx.x - mn.x) + grow, 0.0), hy = fmax(0.5 * ((double)mx.y - mn.y) + grow, 0.0),
                 hz = fmax(0.5 * ((double)mx.z - mn.z) + grow, 0.0);
    const double s = lx.s(cx, cy, cz), t = lx.t(cx, cy, cz);
    const double rs = lx.reach_s(hx, hy, hz) + ft.x + 0.01, rt = lx.reach_t(hx, hy, hz) + ft.y + 0.01;
    if (!(fabs(s) + rs < 1e9 && fabs(t) + rt < 1e9)) return;
    const int s0 = max((int)ceil(s - rs), 0), t0 = max((int)ceil(t - rt), 0);
    box[p] = make_int4(s0, t0, min((int)floor(s + rs) + 1, lx.w), min((int)floor(t + rt) + 1, lx.h));
}

// ---- the parents -------------------------------------------------------------

// The parents' records from their list.
__global__ void k_parent_records(BounceView v, const int32_t *__restrict__ list, int n, int4 *__restrict__ parent,
                                 float2 *__restrict__ share) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p = __ldg(&list[i]);
    const int4 tr = __ldg(&v.tree[p]);
    const float a1 = __ldg(&v.origin[tr.y].w), a2 = __ldg(&v.origin[tr.z].w);
    parent[i] = make_int4(p, tr.y, tr.z, tr.w);
    share[i] = make_float2(__fdiv_rn(a1, __fadd_rn(a1, a2)), __fdiv_rn(a2, __fadd_rn(a1, a2)));
}

// The faces' roots, as the candidate walk reads them.
__global__ void k_roots(BounceView v, float4 *__restrict__ plane, float4 *__restrict__ origin,
                        int4 *__restrict__ tree) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= v.nfaces) return;
    const int root = __ldg(&v.face_range[f].x);
    if (root < 0) {
        tree[f] = make_int4(-1, -1, -1, f);
        // No receiver lies in front of it.
        plane[f] = make_float4(0.0f, 0.0f, 0.0f, FLT_MAX);
        origin[f] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    const int4 tr = __ldg(&v.tree[root]);
    const float4 n = __ldg(&v.normal[root]);
    plane[f] = make_float4(n.x, n.y, n.z, __double2float_rd((double)n.w + 0.01));
    origin[f] = __ldg(&v.origin[root]);
    tree[f] = make_int4(root, tr.y, tr.z, f);
}

// One block per face: its parents level by level, bottom up, so that every
// parent reads final children.  A level is a few loads that wait for one
// another, so what it costs is launches and latency: a launch per level over
// all faces took 93 us a bounce on the 8x8 grid of rooms and 45 on the 3x3
// grid, and a thread per face 1.2 ms and 0.9 ms a pass for the direct light;
// a block per face takes 39 and 16 us (32 to 128 threads: the same; 256: 10
// us more).  OP per parent:
//   kOpDirect   BuildPatchLights' area blend of the children's direct light,
//               then MoveDirectLightToEmission
//   kOpCollect  CollectLight's parents: the blend of the children's light
//               and emission, shot on; nothing from a sky face
//   kOpGuess    the blend of the warm start's guess
enum : int { kOpDirect = 0, kOpCollect = 1, kOpGuess = 2 };
constexpr int kFaceThreads = 64;

__device__ __forceinline__ float4 blend(const float4 &a, const float4 &b, const float2 &s) {
    return make_float4(__fadd_rn(__fmul_rn(a.x, s.x), __fmul_rn(b.x, s.y)),
                       __fadd_rn(__fmul_rn(a.y, s.x), __fmul_rn(b.y, s.y)),
                       __fadd_rn(__fmul_rn(a.z, s.x), __fmul_rn(b.z, s.y)), 0.0f);
}

template <int OP>
__global__ void __launch_bounds__(kFaceThreads)
    k_parents(BounceView v, const int32_t *__restrict__ face_level, const int32_t *__restrict__ level_off,
              const int4 *__restrict__ parent, const float2 *__restrict__ share, float4 *light, float4 *emit,
              float4 *shoot) {
    const int f = blockIdx.x;
    const int h1 = __ldg(&face_level[f + 1]) - 1;
    for (int h = __ldg(&face_level[f]); h < h1; h++) {
        const int end = __ldg(&level_off[h + 1]);
        for (int i = __ldg(&level_off[h]) + threadIdx.x; i < end; i += kFaceThreads) {
            const int4 p = __ldg(&parent[i]);
            const float2 s = __ldg(&share[i]);
            if (OP == kOpCollect && p.w) {
                emit[p.x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                shoot[p.x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                continue;
            }
            const float4 t = blend(light[p.y], light[p.z], s);
            light[p.x] = t;
            if (OP == kOpGuess) continue;
            const float4 e = OP == kOpDirect ? t : blend(emit[p.y], emit[p.z], s), r = __ldg(&v.refl[p.x]);
            emit[p.x] = e;
            shoot[p.x] = make_float4(__fmul_rn(e.x, r.x), __fmul_rn(e.y, r.y), __fmul_rn(e.z, r.z), 0.0f);
        }
        __syncthreads();
    }
}

// ---- transfers ---------------------------------------------------------------

// Enumerator.Run for one receiver: the faces of its cluster's PVS row
// other than its own, each tested with TestPatchToFace, then its patch
// tree walked as TestPatchToPatch recurses (child1's subtree before
// child2's).  Counts, or writes the candidates.
//
// One lane per receiver, but one walk per warp: its receivers share the row
// and lie beside each other, so nearly every node that one of them visits,
// the others do.  A node is popped with the lanes that are to look at it,
// loaded once for all, and its children are pushed with the lanes that
// refine it; what a lane takes still comes in its own walk's order.  The
// row's faces are staged 32 at a time in shared memory.
//
// The comparisons are the reference's, which widens to double, as float
// comparisons that say the same: x > d of a float x and a double d is x > the
// largest float up to d; x / 16 < a is x < 16 a, both products exact.
//
// What bounds it is the issue of the walk's steps, the union of 32 receivers'
// (500 to 1700 nodes on the 3x3 grid of rooms), and for few receivers the
// chain of one warp's, so then a row is cut into segments (row_segments) that
// are warps of their own.  On the 8x8 grid (1 M receivers, 649 M candidates)
// it takes 4.1 ms, a walk by each thread took 6.8; on the 3x3 grid (35 k,
// 10 M) 0.24 ms in 16 segments, 0.40, 0.26 in 4 and 8, 0.59 in one, 0.66 by
// each thread.  Candidates are held back until four make a 16 B store: one by
// one the 8x8 grid takes 6.6 ms, by eight or in rows of 32 by warp 4.2.
constexpr int kHold = 4;

template <bool WRITE>
__global__ void __launch_bounds__(kBounceBlock)
    k_candidates(BounceView v, const float4 *__restrict__ root_plane, const float4 *__restrict__ root_origin,
                 const int4 *__restrict__ root_tree, const int64_t *__restrict__ seg_off,
                 int64_t *__restrict__ counts, int32_t *__restrict__ out, uint32_t *__restrict__ overflow) {
    constexpr int kWarps = kBounceBlock / 32;
    __shared__ float4 s_plane[kWarps][32], s_origin[kWarps][32];
    __shared__ int4 s_tree[kWarps][32];
    __shared__ int2 s_stack[kWarps][kEnumStack];
    __shared__ int s_held[WRITE ? kHold : 1][kBounceBlock];
    const int r = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool live = r < v.nreceivers;
    const int seg = blockIdx.y, nseg = gridDim.y;
    F3 o = {0.0f, 0.0f, 0.0f}, me_n = o;
    float me_d = 0.0f;
    int face = -1, cluster = -1;
    int64_t first = 0;
    if (live) {
        const int p = __ldg(&v.recv[r]);
        const float4 mn = __ldg(&v.mins[p]), mx = __ldg(&v.maxs[p]);
        o = f3(__ldg(&v.origin[p]));
        face = __float_as_int(mn.w);
        cluster = __float_as_int(mx.w);
        me_n = f3(__ldg(&v.face_plane[face]));
        me_d = __double2float_rd((double)__ldg(&v.normal[p].w) + 0.01);
        if (WRITE) first = seg_off[(int64_t)r * nseg + seg];
    }
    int64_t at = first;
    auto take = [&](int s, const float4 &so) {
        if (!(dot3(f3(so), me_n) > me_d)) return;
        if (WRITE) {
            s_held[at & (kHold - 1)][threadIdx.x] = s;
            if ((at & (kHold - 1)) == kHold - 1) {
                if (at - (kHold - 1) >= first)
                    *(int4 *)(out + at - (kHold - 1)) = make_int4(s_held[0][threadIdx.x], s_held[1][threadIdx.x],
                                                                  s_held[2][threadIdx.x], s_held[3][threadIdx.x]);
                else
                    for (int64_t q = first; q <= at; q++) out[q] = s_held[q & (kHold - 1)][threadIdx.x];
            }
        }
        at++;
    };
    // Whether the lane refines the patch (takes its children instead).
    auto refines = [&](const float4 &so, int child1) {
        const F3 d = sub3(o, f3(so));
        return child1 != -1 && dot3(d, d) < 16.0f * so.w;
    };
    unsigned todo = __ballot_sync(kFull, live);
    while (todo) {
        // The lanes of one cluster: all of them but where a warp straddles two.
        const int c = __shfl_sync(kFull, cluster, __ffs(todo) - 1);
        const bool mine = live && cluster == c;
        todo &= ~__ballot_sync(kFull, mine);
        const int row = __ldg(&v.row_off[c]), n = __ldg(&v.row_off[c + 1]) - row;
        const int q0 = row + (int)((int64_t)n * seg / nseg), q1 = row + (int)((int64_t)n * (seg + 1) / nseg);
        for (int q = q0; q < q1; q += 32) {
            const int m = min(32, q1 - q);
            __syncwarp();
            if (lane < m) {
                const int g = __ldg(&v.row_faces[q + lane]);
                s_plane[warp][lane] = __ldg(&root_plane[g]);
                s_origin[warp][lane] = __ldg(&root_origin[g]);
                s_tree[warp][lane] = __ldg(&root_tree[g]);
            }
            __syncwarp();
            for (int k = 0; k < m; k++) {
                const int4 rt = s_tree[warp][k];
                const float4 rp = s_plane[warp][k];
                const bool pass = mine && rt.w != face && dot3(o, f3(rp)) > rp.w;
                if (!__any_sync(kFull, pass)) continue;
                const float4 ro = s_origin[warp][k];
                const bool ref = pass && refines(ro, rt.y);
                if (pass && !ref) take(rt.x, ro);
                unsigned lanes = __ballot_sync(kFull, ref);
                if (!lanes) continue;
                int sp = 2;
                if (lane < 2) s_stack[warp][lane] = make_int2(lane ? rt.y : rt.z, (int)lanes);
                __syncwarp();
                while (sp > 0) {
                    const int2 top = s_stack[warp][--sp];
                    const int4 tr = __ldg(&v.tree[top.x]);
                    const float4 so = __ldg(&v.origin[top.x]);
                    const bool in = ((unsigned)top.y >> lane) & 1u, refine = in && refines(so, tr.y);
                    if (in && !refine) take(top.x, so);
                    lanes = __ballot_sync(kFull, refine);
                    if (!lanes) continue;
                    if (sp + 2 > kEnumStack) {
                        if (lane == 0) atomicOr(overflow, 2u);
                        continue;
                    }
                    if (lane < 2) s_stack[warp][sp + lane] = make_int2(lane ? tr.y : tr.z, (int)lanes);
                    sp += 2;
                    __syncwarp();
                }
            }
        }
    }
    if (!live) return;
    if (!WRITE) counts[(int64_t)r * nseg + seg] = at - first;
    if (WRITE)
        for (int64_t q = max(first, at & ~(int64_t)(kHold - 1)); q < at; q++)
            out[q] = s_held[q & (kHold - 1)][threadIdx.x];
}

// FormFactors.DiffToDiff(o1, n1, o2, n2): delta = normalise(o1 - o2), then
// -(delta . n1) * (delta . n2) / (len * len).
__device__ __forceinline__ float diff_to_diff(F3 o1, F3 n1, F3 o2, F3 n2) {
    float dl;
    const F3 d = normalise3(sub3(o1, o2), dl);
    return __fdiv_rn(__fmul_rn(-dot3(d, n1), dot3(d, n2)), __fmul_rn(dl, dl));
}

// FormFactors.PolyToDiff of a winding of `count` points seen from (o, n).
__device__ float poly_to_diff_pts(const float4 *__restrict__ pts, int count, float area, F3 o, F3 n,
                                  unsigned long long *open) {
    float ff = 0.0f;
    for (int k = 0; k < count; k++) {
        const int k2 = k < count - 1 ? k + 1 : 0;
        float l;
        const F3 v1 = normalise3(sub3(f3(__ldg(&pts[k])), o), l);
        const F3 v2 = normalise3(sub3(f3(__ldg(&pts[k2])), o), l);
        float sin_alpha;
        F3 gamma = normalise3(cross3(v1, v2), sin_alpha);
        if (sin_alpha < -1.0f || sin_alpha > 1.0f) sin_alpha = sin_alpha > 1.0f ? 1.0f : -1.0f;
        gamma = mul3(gamma, asin_cr(sin_alpha, open));
        ff = __fadd_rn(ff, dot3(gamma, n));
    }
    return __fmul_rn(ff, __fdiv_rn(0.5f, area));
}

// PolyToDiff of source s's winding seen from (o, n).
__device__ __forceinline__ float poly_to_diff(const BounceView &v, int s, float area, F3 o, F3 n,
                                              unsigned long long *open) {
    const int2 w = __ldg(&v.wind[s]);
    return poly_to_diff_pts(v.points + w.x, w.y, area, o, n, open);
}

// MakeTransfer for an open pair (receiver p, source s): DiffToDiff(source,
// receiver), the polygon form factor for a near source, trans = area *
// scale > 1e-7; 0 for none.
__device__ __forceinline__ float make_transfer(const BounceView &v, int p, int s, unsigned long long *open) {
    const float4 so = __ldg(&v.origin[s]);
    if (__ldg(&v.tree[s].w) != 0 || !(so.w > 0.0f)) return 0.0f;
    const float4 po = __ldg(&v.origin[p]), pn = __ldg(&v.normal[p]), sn = __ldg(&v.normal[s]);
    float scale = diff_to_diff(f3(so), f3(sn), f3(po), f3(pn));
    if (scale <= 0.0f) return 0.0f;
    const F3 dd = sub3(f3(po), f3(so));
    const float threshold = (float)__dmul_rn(3.141592653589793 * 0.04, (double)dot3(dd, dd));
    if (threshold < so.w) {
        scale = poly_to_diff(v, s, so.w, f3(po), f3(pn), open);
        if (scale <= 0.0f) return 0.0f;
    }
    const float trans = __fmul_rn(so.w, scale);
    return (double)trans > 0.0000001 ? trans : 0.0f;
}

// Where each receiver's transfer rays start their walk.
__global__ void k_starts(BounceView v, DeviceBvh opaque, int32_t *__restrict__ start) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nreceivers) return;
    const int p = __ldg(&v.recv[r]);
    const F3 o = add3(f3(__ldg(&v.origin[p])), f3(__ldg(&v.normal[p])));
    start[r] = start_node(opaque, o.x, o.y, o.z);
}

// One candidate pair: VisMatrix.TransferRay traced (StockExact: every
// triangle blocks, t in (0, len)), then MakeTransfer.  cand_w = the
// transfer, 0 for none, kBlocked for a blocked ray (which k_transfer_count
// counts: an atomic per warp here would be 20 M on one address).  Twelve
// CTAs per SM (40 registers, a few spilled to L1).
constexpr float kBlocked = -1.0f;

template <bool ONE, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 12)
    k_transfer(BounceView v, DeviceScene sc, const int64_t *__restrict__ cand_off, const int32_t *__restrict__ cand_src,
               const int32_t *__restrict__ start_at, float *__restrict__ cand_w, int64_t ncand,
               unsigned long long *open) {
    extern __shared__ int stack_mem[];  // sc.stack_depth() entries per thread
    int *stack = stack_mem + threadIdx.x;
    const int64_t q = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
    // The receiver whose run holds q: one binary search per warp, for its
    // first candidate, then each lane steps forward (a warp's 32
    // candidates seldom span more than one or two receivers).
    const int64_t q0 = (int64_t)blockIdx.x * BLOCK + (threadIdx.x & ~31);
    int r0 = 0;
    if ((threadIdx.x & 31) == 0 && q0 < ncand) {
        int lo = 0, hi = v.nreceivers;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(&cand_off[mid]) <= q0) lo = mid;
            else hi = mid;
        }
        r0 = lo;
    }
    r0 = __shfl_sync(kFull, r0, 0);
    if (q < ncand) {
        int lo = r0;
        while (__ldg(&cand_off[lo + 1]) <= q) lo++;
        const int p = __ldg(&v.recv[lo]);
        const int s = __ldg(&cand_src[q]);
        const float4 po = __ldg(&v.origin[p]), pn = __ldg(&v.normal[p]);
        const float4 so = __ldg(&v.origin[s]), sn = __ldg(&v.normal[s]);
        const F3 start = add3(f3(po), f3(pn)), end = add3(f3(so), f3(sn));
        const F3 delta = sub3(end, start);
        const float len = __fsqrt_rn(dot3(delta, delta));
        const float safe = len == 0.0f ? 1.1920929e-07f : len;
        const RayState ray = make_ray(start.x, start.y, start.z, __fdiv_rn(delta.x, safe), __fdiv_rn(delta.y, safe),
                                      __fdiv_rn(delta.z, safe));
        float t, w = kBlocked;
        int32_t orig;
        uint32_t meta;
        bool blocked;
        trace_ray<ONE, kModeAny, BLOCK, true>(sc, ray, 0.0f, len, -1, ONE ? 0 : __ldg(&start_at[lo]), stack, blocked, t,
                                              orig, meta);
        if (!blocked) {
            // The pair's rows are read again here, not held across the walk:
            // at 40 registers they would be spilled to L1, whose bandwidth
            // bounds the walk (transfer build 53.9 -> 50.2 ms on the 8x8 map).
            int64_t again = q;
            asm volatile("" : "+r"(lo), "+l"(again));
            w = make_transfer(v, __ldg(&v.recv[lo]), __ldg(&cand_src[again]), open);
        }
        cand_w[q] = w;
    }
}

// The groups' warps: one per 32 positions of the longest list of the
// group's receivers.
__global__ void k_group_warps(int nrecv, int ngroups, const int64_t *__restrict__ cand_off, int64_t *__restrict__ warps) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    int64_t n = 0;
    for (int r = g * kGroup; r < min(nrecv, (g + 1) * kGroup); r++) n = max(n, cand_off[r + 1] - cand_off[r]);
    warps[g] = (n + 31) / 32;
}

// Each of those warps' group.
__global__ void k_warp_groups(int ngroups, const int64_t *__restrict__ group_off, int32_t *__restrict__ warp_group) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    for (int64_t w = group_off[g]; w < group_off[g + 1]; w++) warp_group[w] = g;
}

// The same by groups of kGroup receivers, for maps of kGroupedReceivers and
// more.  Neighbouring receivers see much the same sources, in the same order:
// what blocked the ray to a list's j-th source mostly blocks the next
// receiver's.  So a warp takes 32 positions of a group's lists, keeps per
// position the triangle that blocked its last traced ray, and tests each ray
// against that one first; only the others are traced, 32 at a time from a
// queue, so that the walk's lanes stay full.  Any triangle that blocks is
// answer enough, so the answers are the walk's.  On the 8x8 grid of rooms
// (649 M rays, 67 % blocked) the transfer build takes 35.0 ms, ray by ray
// 44.8; with groups of 4 and 8 receivers 39.5 and 36.0; on the 4x4 map (153 M,
// 62 %) 9.2 and 11.0; with 76 k receivers 2.23 and 2.31, with 61 k 1.66 both
// ways, with 36 k 1.07 and 1.03: few receivers make too few warps of 512 rays
// each.  Ten CTAs an SM: twelve 36.4 ms, eight 36.1.
template <bool ONE, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 10)
    k_transfer_groups(BounceView v, DeviceScene sc, const int64_t *__restrict__ cand_off,
                      const int32_t *__restrict__ cand_src, const int32_t *__restrict__ start_at,
                      const int64_t *__restrict__ group_off, const int32_t *__restrict__ warp_group, int64_t nwarps,
                      float *__restrict__ cand_w, unsigned long long *open) {
    extern __shared__ int stack_mem[];  // sc.stack_depth() entries per thread
    __shared__ int64_t s_off[BLOCK / 32][kGroup + 1];  // the receivers' lists at this warp's position
    __shared__ int s_tri[BLOCK / 32][32];              // per position, the triangle that blocked its last ray
    __shared__ uint16_t s_queue[BLOCK / 32][64];       // rays to trace: receiver (of the group) * 32 + position
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int *stack = stack_mem + threadIdx.x;
    int64_t *off = s_off[wib];
    int *tri = s_tri[wib];
    uint16_t *queue = s_queue[wib];
    const int64_t warp = ((int64_t)blockIdx.x * BLOCK + threadIdx.x) >> 5;
    if (warp >= nwarps) return;
    const int group = __ldg(&warp_group[warp]);
    const int r0 = group * kGroup, nr = min(kGroup, v.nreceivers - r0);
    const int chunk = 32 * (int)(warp - __ldg(&group_off[group]));
    if (lane <= nr) off[lane] = __ldg(&cand_off[r0 + lane]);
    tri[lane] = -1;
    __syncwarp();
    // A pair's ray (without the reciprocals where only a triangle is tested).
    auto ray_of = [&](int p, int s, float &len) {
        const float4 po = __ldg(&v.origin[p]), pn = __ldg(&v.normal[p]);
        const float4 so = __ldg(&v.origin[s]), sn = __ldg(&v.normal[s]);
        const F3 start = add3(f3(po), f3(pn)), end = add3(f3(so), f3(sn));
        const F3 delta = sub3(end, start);
        len = __fsqrt_rn(dot3(delta, delta));
        const float safe = len == 0.0f ? 1.1920929e-07f : len;
        return make_ray(start.x, start.y, start.z, __fdiv_rn(delta.x, safe), __fdiv_rn(delta.y, safe),
                        __fdiv_rn(delta.z, safe));
    };
    int n = 0;  // rays in the queue, under 64
    // Traces the queue's last m rays.
    auto trace = [&](int m) {
        __syncwarp();
        if (lane < m) {
            int e = queue[n - m + lane];
            int64_t q = off[e >> 5] + chunk + (e & 31);
            const int r = r0 + (e >> 5);
            float len, t, w = kBlocked;
            const RayState ray = ray_of(__ldg(&v.recv[r]), __ldg(&cand_src[q]), len);
            int32_t orig;
            uint32_t meta;
            int at = -1;
            bool blocked;
            trace_ray<ONE, kModeAny, BLOCK, true>(sc, ray, 0.0f, len, -1, ONE ? 0 : __ldg(&start_at[r]), stack, blocked, t,
                                                  orig, meta, &at);
            // The pair's rows are read again here, not held across the walk.
            e = queue[n - m + lane];
            q = off[e >> 5] + chunk + (e & 31);
            // Of two rays of one position either's triangle will do; an open
            // ray's position is not tested next time.
            tri[e & 31] = at;
            if (!blocked) w = make_transfer(v, __ldg(&v.recv[r0 + (e >> 5)]), __ldg(&cand_src[q]), open);
            cand_w[q] = w;
        }
        n -= m;
        __syncwarp();
    };
    for (int k = 0; k < nr; k++) {
        const int64_t q = off[k] + chunk + lane;
        const bool live = q < off[k + 1];
        if (!__any_sync(kFull, live)) continue;
        bool walk = live;
        const int last = tri[lane];
        if (live && last >= 0) {
            float len, t;
            const RayState ray = ray_of(__ldg(&v.recv[r0 + k]), __ldg(&cand_src[q]), len);
            uint32_t meta;
            int32_t orig;
            if (kd_hit<false>(sc.opaque, last, ray, t, meta, orig, nullptr) && t >= 0.0f && t < len) {
                cand_w[q] = kBlocked;
                walk = false;
            }
        }
        const unsigned rays = __ballot_sync(kFull, walk);
        if (walk) queue[n + __popc(rays & ((1u << lane) - 1u))] = (uint16_t)(32 * k + lane);
        n += __popc(rays);
        if (n >= 32) trace(32);
    }
    if (n) trace(n);
}

// MakeTransfers' count per receiver: accepted pairs, at most MaxPatches;
// and the blocked rays, added to *blocked.
__global__ void k_transfer_count(int nrecv, const int64_t *__restrict__ cand_off, const float *__restrict__ cand_w,
                                 int64_t *__restrict__ counts, unsigned long long *blocked) {
    __shared__ unsigned long long part[kBounceBlock / 32];
    const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const unsigned lane = threadIdx.x & 31;
    int64_t n = 0, shut = 0;
    if (r < nrecv) {
        const int64_t a = cand_off[r], b = cand_off[r + 1];
        for (int64_t base = a; base < b; base += 32) {
            const int64_t q = base + lane;
            const float w = q < b ? cand_w[q] : 0.0f;
            n += __popc(__ballot_sync(kFull, w > 0.0f));
            shut += __popc(__ballot_sync(kFull, w == kBlocked));
        }
        if (lane == 0) counts[r] = n < kMaxTransfersPerReceiver ? n : kMaxTransfersPerReceiver;
    }
    if (lane == 0) part[threadIdx.x >> 5] = (unsigned long long)shut;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sum = 0;
        for (int k = 0; k < kBounceBlock / 32; k++) sum += part[k];
        if (sum) atomicAdd(blocked, sum);
    }
}

// MakeTransfers' writes in candidate order (the first MaxPatches), then
// MakeScales: the float sum in order, total > pi ? 1/total : 1/pi, and the
// weights scaled.
__global__ void k_transfer_write(int nrecv, const int64_t *__restrict__ cand_off, const int32_t *__restrict__ cand_src,
                                 const float *__restrict__ cand_w, const int64_t *__restrict__ tr_off,
                                 int2 *__restrict__ tr) {
    const int r = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const unsigned lane = threadIdx.x & 31;
    if (r >= nrecv) return;
    const int64_t a = cand_off[r], b = cand_off[r + 1];
    const int64_t o0 = tr_off[r], o1 = tr_off[r + 1];
    int64_t made = 0;
    for (int64_t base = a; base < b && o0 + made < o1; base += 32) {
        const int64_t q = base + lane;
        const float w = q < b ? cand_w[q] : 0.0f;
        const unsigned ok = __ballot_sync(kFull, w > 0.0f);
        const int64_t at = o0 + made + __popc(ok & ((1u << lane) - 1u));
        if (w > 0.0f && at < o1) tr[at] = make_int2(cand_src[q], __float_as_int(w));
        made += __popc(ok);
    }
    __syncwarp();
    float scale = 0.0f;
    if (lane == 0 && o1 > o0) {
        float total = 0.0f;
        for (int64_t j = o0; j < o1; j++) total = __fadd_rn(total, __int_as_float(tr[j].y));
        scale = (double)total > 3.141592653589793 ? __fdiv_rn(1.0f, total) : (float)(1.0 / 3.141592653589793);
    }
    scale = __shfl_sync(kFull, scale, 0);
    __syncwarp();
    for (int64_t j = o0 + lane; j < o1; j += 32) {
        const int2 t = tr[j];
        tr[j] = make_int2(t.x, __float_as_int(__fmul_rn(__int_as_float(t.y), scale)));
    }
}

// ---- bounces ---------------------------------------------------------------

// The gather's slices (SELL-32) of the transfer lists: each receiver's key
// and index for the sort by window and count.
__global__ void k_sell_keys(int nrecv, int window, const int64_t *__restrict__ tr_off, uint32_t *__restrict__ key,
                            int32_t *__restrict__ idx) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrecv) return;
    key[r] = ((uint32_t)(r / window) << kCountBits) | (kCountMask - (uint32_t)(tr_off[r + 1] - tr_off[r]));
    idx[r] = r;
}

__device__ __forceinline__ int sell_count(uint32_t key) { return (int)(kCountMask - (key & kCountMask)); }

// Slice s's size: 32 times its first (largest) count.
__global__ void k_sell_width(int nslices, const uint32_t *__restrict__ sorted, int64_t *__restrict__ width) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslices) return;
    width[s] = 32 * (int64_t)sell_count(sorted[32 * s]);
}

// Copies each receiver's transfers into its lane of its slice.
__global__ void k_sell_pack(int nrecv, const int32_t *__restrict__ order, const uint32_t *__restrict__ sorted,
                            const int64_t *__restrict__ sell_off, const int64_t *__restrict__ tr_off,
                            const int2 *__restrict__ tr, int2 *__restrict__ sell) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrecv) return;
    const int r = order[i], n = sell_count(sorted[i]);
    const int2 *src = tr + tr_off[r];
    int2 *dst = sell + sell_off[i >> 5] + (i & 31);
    for (int j = 0; j < n; j++) dst[32 * (int64_t)j] = __ldg(&src[j]);
}

// 32 times each window's largest candidate count, added up: what the slices'
// padding can come to (a slice's padding is at most 32 times its first count
// less its own transfers, and that first count at most the last of the
// slice before).
__global__ void k_sell_pad(int nrecv, int window, const int64_t *__restrict__ cand_off, unsigned long long *pad) {
    __shared__ int largest;
    if (threadIdx.x == 0) largest = 0;
    __syncthreads();
    int m = 0;
    const int r0 = blockIdx.x * window;
    for (int r = r0 + threadIdx.x; r < min(r0 + window, nrecv); r += blockDim.x) {
        const int64_t n = cand_off[r + 1] - cand_off[r];
        m = max(m, (int)(n < kMaxTransfersPerReceiver ? n : kMaxTransfersPerReceiver));
    }
    atomicMax(&largest, m);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(pad, 32ull * (unsigned long long)largest);
}

// The block's part of a bounce's totals: the light the bounce added (the
// sky-free leaves' emission e), in fp64, with two sums that bound how far
// the reference's float sum (CollectLight's, in leaf_desc order) can lie
// from it: the absolute values, and the absolute values each weighted by the
// number of terms from it to the end of that order (left = n - rank).
// Recursive summation's error is at most u * sum_k |partial sum k| <=
// u * sum_i |x_i| (n - rank_i), over 1 - n u.  The blocks add to kSumParts
// parts, so that few meet on one address.
__device__ __forceinline__ void add_totals(const F3 &e, double left, double *__restrict__ sums) {
    __shared__ double part[kSums][kBounceBlock / 32];
    double s[kSums] = {e.x, e.y, e.z, fabs((double)e.x), fabs((double)e.y), fabs((double)e.z)};
    s[6] = s[3] * left, s[7] = s[4] * left, s[8] = s[5] * left;
#pragma unroll
    for (int k = 0; k < kSums; k++)
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_down_sync(kFull, s[k], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < kSums; k++) part[k][warp] = s[k];
    __syncthreads();
    if (threadIdx.x < kSums) {
        double t = 0.0;
        for (int w = 0; w < kBounceBlock / 32; w++) t += part[threadIdx.x][w];
        atomicAdd(&sums[kSums * (blockIdx.x % kSumParts) + threadIdx.x], t);
    }
}

// GatherLight for one receiver (the ordered sum over its transfers of the
// sources' shoot times the weight), then CollectLight's update of that
// leaf: the light added, emitted and shot on, and the bounce's totals.
// Thread i takes the i-th receiver of the slices' order, its transfers from
// its lane of its slice.
//
// Each sum is one chain in the reference's order, so the loads are what a
// thread waits for: it asks for the next eight entries and for this eight's
// sources before it adds.  The entries stream from HBM (8 B a transfer, once
// a bounce); the sources are 16 B from anywhere in the light array, and a
// window of neighbouring receivers, whose lists name much the same sources,
// is what is sorted by count, not the whole map (whose slices then mix
// receivers from everywhere).  With 214 M transfers a bounce (1.7 GB, 0.26
// ms at the copy rate) took 0.66 ms one entry at a time, sorted as a whole,
// with the totals and the parents' levels in launches of their own; 0.53
// with windows of 1024 and those folded in (256 to 2048: the same; the whole
// map: 0.62); 0.41 with eight ahead, of which the gather is 0.36.  Two,
// four, twelve and sixteen ahead: 0.51, 0.51, 0.50 and 0.57.  With 35 k
// receivers, 7 warps an SM, it is latency: 99 us a bounce, then 50.
constexpr int kAhead = 8;

__global__ void __launch_bounds__(kBounceBlock)
    k_gather(BounceView v, const int32_t *__restrict__ order, const uint32_t *__restrict__ sorted,
             const int64_t *__restrict__ sell_off, const int2 *__restrict__ sell, const float4 *__restrict__ shoot_in,
             float4 *__restrict__ total, float4 *__restrict__ emit_out, float4 *__restrict__ shoot_out,
             const int32_t *__restrict__ leaf_rank, int32_t nleaves, double *__restrict__ sums) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    F3 e = {0.0f, 0.0f, 0.0f};
    double left = 0.0;
    if (i < v.nreceivers) {
        const int p = __ldg(&v.recv[__ldg(&order[i])]);
        const int n = sell_count(__ldg(&sorted[i]));
        const int2 *src = sell + __ldg(&sell_off[i >> 5]) + (i & 31);
        float sx = 0.0f, sy = 0.0f, sz = 0.0f;
        int2 t[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; k++)
            if (k < n) t[k] = __ldcs(&src[32 * k]);
        for (int j = 0; j < n; j += kAhead) {
            float4 s[kAhead];
            int2 next[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (j + k < n) s[k] = __ldg(&shoot_in[t[k].x]);
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (j + kAhead + k < n) next[k] = __ldcs(&src[32 * (int64_t)(j + kAhead + k)]);
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (j + k < n) {
                    const float w = __int_as_float(t[k].y);
                    sx = __fadd_rn(sx, __fmul_rn(s[k].x, w));
                    sy = __fadd_rn(sy, __fmul_rn(s[k].y, w));
                    sz = __fadd_rn(sz, __fmul_rn(s[k].z, w));
                }
#pragma unroll
            for (int k = 0; k < kAhead; k++) t[k] = next[k];
        }
        if (__ldg(&v.tree[p].w)) {
            emit_out[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            shoot_out[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            const float4 t = total[p];
            total[p] = make_float4(__fadd_rn(t.x, sx), __fadd_rn(t.y, sy), __fadd_rn(t.z, sz), 0.0f);
            emit_out[p] = make_float4(sx, sy, sz, 0.0f);
            const float4 rf = __ldg(&v.refl[p]);
            shoot_out[p] = make_float4(__fmul_rn(sx, rf.x), __fmul_rn(sy, rf.y), __fmul_rn(sz, rf.z), 0.0f);
            e = {sx, sy, sz};
            left = (double)(nleaves - __ldg(&leaf_rank[p]));
        }
    }
    add_totals(e, left, sums);
}

// CollectLight's own total: the leaves' emission summed in float, in
// descending index order (leaf_desc lists the sky-free leaves that way).
// The sum is one chain of a million dependent, rounded adds, but while it
// stays between two powers of two it is a whole number of ulps u, and adding
// x >= 0 adds rint(x / u) of them, whatever the sum, unless x lies half way
// between two ulps (then the sum's parity decides).  So the leaves are cut
// into chunks:
//   k_exact_sums   each chunk's sum in fp64
//   k_exact_steps  each chunk's whole ulps, for the ulp at which the sums
//                  before it say that it starts
//   k_exact_walk   from chunk to chunk: a chunk whose start has that ulp,
//                  that leaves it unchanged and that has no half way case
//                  is one integer add; any other is added up value by value
// A sum over 1 M leaves passes about twenty powers of two, so nearly every
// chunk is one add: 0.5 ms, 5.0 as one chain of adds fed by a block.
struct ExactStep {
    long long ulps;
    int32_t exponent;  // the biased exponent of the chunk's start
    int32_t kind;      // kByValue, kByUlps, or kNothing: every value is zero
};
enum : int32_t { kByValue = 0, kByUlps = 1, kNothing = 2 };
constexpr int kExactBlock = 128;

__device__ __forceinline__ float channel(const float4 &v, int c) { return c == 0 ? v.x : c == 1 ? v.y : v.z; }

// The block's sum of x; every thread has it.
template <typename T>
__device__ __forceinline__ T block_sum(T x, T *part) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
    __syncthreads();
    T t = part[0];
    for (int w = 1; w < kExactBlock / 32; w++) t += part[w];
    return t;
}

__global__ void __launch_bounds__(kExactBlock) k_exact_sums(const int32_t *__restrict__ leaf_desc, int32_t n, int per,
                                                            int nchunks, const float4 *__restrict__ emit,
                                                            double *__restrict__ sums) {
    __shared__ double part[kExactBlock / 32];
    double s[3] = {0.0, 0.0, 0.0};
    const int64_t first = (int64_t)blockIdx.x * per, end = first + per < n ? first + per : n;
    for (int64_t i = first + threadIdx.x; i < end; i += kExactBlock) {
        const float4 v = __ldg(&emit[__ldg(&leaf_desc[i])]);
        for (int c = 0; c < 3; c++) s[c] += (double)channel(v, c);
    }
    for (int c = 0; c < 3; c++) {
        const double t = block_sum(s[c], part);
        if (threadIdx.x == 0) sums[(int64_t)c * nchunks + blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kExactBlock) k_exact_steps(const int32_t *__restrict__ leaf_desc, int32_t n, int per,
                                                             int nchunks, const float4 *__restrict__ emit,
                                                             const double *__restrict__ sums,
                                                             ExactStep *__restrict__ steps) {
    __shared__ double part[kExactBlock / 32];
    __shared__ long long ipart[kExactBlock / 32];
    const int64_t first = (int64_t)blockIdx.x * per, end = first + per < n ? first + per : n;
    for (int c = 0; c < 3; c++) {
        double before = 0.0;
        for (int k = threadIdx.x; k < (int)blockIdx.x; k += kExactBlock) before += __ldg(&sums[(int64_t)c * nchunks + k]);
        const float start = (float)block_sum(before, part);
        const int e = (int)(__float_as_uint(start) >> 23);
        // 2^(150 - e), one over the ulp.
        const double per_ulp = __longlong_as_double((long long)(1023 + 150 - e) << 52);
        long long ulps = 0;
        bool whole = e > 0 && e < 255, zero = true;
        for (int64_t i = first + threadIdx.x; i < end; i += kExactBlock) {
            const float x = channel(__ldg(&emit[__ldg(&leaf_desc[i])]), c);
            zero = zero && x == 0.0f;
            const double q = (double)x * per_ulp;
            whole = whole && x >= 0.0f && q < 16777216.0 && q - floor(q) != 0.5;
            if (whole) ulps += __double2ll_rn(q);
        }
        ulps = block_sum(ulps, ipart);
        whole = __syncthreads_and(whole);
        zero = __syncthreads_and(zero);
        if (threadIdx.x == 0)
            steps[(int64_t)c * nchunks + blockIdx.x] = {ulps, e, zero ? kNothing : whole ? kByUlps : kByValue};
    }
}

// One warp per channel.
__global__ void __launch_bounds__(96) k_exact_walk(const int32_t *__restrict__ leaf_desc, int32_t n, int per, int nchunks,
                                                   const float4 *__restrict__ emit, const ExactStep *__restrict__ steps,
                                                   float *__restrict__ out) {
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto value = [&](int64_t i, int64_t end) {
        return i < end ? channel(__ldg(&emit[__ldg(&leaf_desc[i])]), c) : 0.0f;
    };
    float s = 0.0f;
    for (int base = 0; base < nchunks; base += 32) {
        const int m = min(32, nchunks - base);
        ExactStep mine = {0, 0, kNothing};
        if (lane < m) mine = steps[(int64_t)c * nchunks + base + lane];
        for (int j = 0; j < m; j++) {
            const int kind = __shfl_sync(kFull, mine.kind, j);
            const int e = __shfl_sync(kFull, mine.exponent, j);
            const long long ulps = __shfl_sync(kFull, mine.ulps, j);
            if (kind == kNothing) continue;
            const uint32_t bits = __float_as_uint(s);
            const long long k = (long long)((bits & 0x7FFFFFu) | 0x800000u) + ulps;
            if (kind == kByUlps && (int)(bits >> 23) == e && k < 0x1000000) {
                s = __uint_as_float(((uint32_t)e << 23) | ((uint32_t)k & 0x7FFFFFu));
                continue;
            }
            const int64_t first = (int64_t)(base + j) * per, end = first + per < n ? first + per : n;
            float next = value(first + lane, end);
            for (int64_t i = first; i < end; i += 32) {
                const float v = next;
                next = value(i + 32 + lane, end);
                if (i + 32 <= end) {
#pragma unroll
                    for (int l = 0; l < 32; l++) s = __fadd_rn(s, __shfl_sync(kFull, v, l));
                } else {
                    for (int l = 0; l < (int)(end - i); l++) s = __fadd_rn(s, __shfl_sync(kFull, v, l));
                }
            }
        }
    }
    if (lane == 0) out[c] = s;
}

// ---- the learned warm start --------------------------------------------------

// Per receiver, the network's 32 inputs (BF16): the shading normal, log2 of
// the area over 16, the reflectivity, log1p of the direct and of the
// first-bounce light over 8, log2(1 + d) over 16 of the distances d to the
// eight nearest point and spot lights (1 when there are fewer), zeros.
__global__ void k_features(BounceView v, const float4 *__restrict__ direct, const float4 *__restrict__ first,
                           const float4 *__restrict__ lights, int32_t nlights, uint16_t *__restrict__ x) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nreceivers) return;
    const int p = __ldg(&v.recv[r]);
    const float4 o = __ldg(&v.origin[p]), nrm = __ldg(&v.normal[p]), rf = __ldg(&v.refl[p]);
    const float4 d = direct[p], b1 = first[p];
    float f[kFeatures];
    f[0] = nrm.x, f[1] = nrm.y, f[2] = nrm.z;
    f[3] = log2f(fmaxf(o.w, 1e-6f)) / 16.0f;
    f[4] = rf.x, f[5] = rf.y, f[6] = rf.z;
    f[7] = log1pf(fmaxf(d.x, 0.0f)) / 8.0f, f[8] = log1pf(fmaxf(d.y, 0.0f)) / 8.0f, f[9] = log1pf(fmaxf(d.z, 0.0f)) / 8.0f;
    f[10] = log1pf(fmaxf(b1.x, 0.0f)) / 8.0f, f[11] = log1pf(fmaxf(b1.y, 0.0f)) / 8.0f;
    f[12] = log1pf(fmaxf(b1.z, 0.0f)) / 8.0f;
    float best[8];
    for (int k = 0; k < 8; k++) best[k] = INFINITY;
    for (int l = 0; l < nlights; l++) {
        const float4 a = __ldg(&lights[5 * l]);
        const int type = __float_as_int(a.w);
        if (type != 1 && type != 2) continue;
        const float dx = a.x - o.x, dy = a.y - o.y, dz = a.z - o.z;
        float q = dx * dx + dy * dy + dz * dz;
        for (int k = 0; k < 8; k++) {
            if (q < best[k]) {
                const float tmp = best[k];
                best[k] = q;
                q = tmp;
            }
        }
    }
    for (int k = 0; k < 8; k++) f[13 + k] = isinf(best[k]) ? 1.0f : log2f(1.0f + sqrtf(best[k])) / 16.0f;
    for (int k = 21; k < kFeatures; k++) f[k] = 0.0f;
    for (int k = 0; k < kFeatures; k++) x[(int64_t)r * kFeatures + k] = __bfloat16_as_ushort(__float2bfloat16_rn(f[k]));
}

// The network's guess as light per patch: expm1 of its output, at least
// zero, on the non-sky receivers (everything else zero).
__global__ void k_guess(BounceView v, const float *__restrict__ y, float4 *__restrict__ guess) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nreceivers) return;
    const int p = __ldg(&v.recv[r]);
    float4 gv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!__ldg(&v.tree[p].w)) {
        gv.x = fmaxf(expm1f(y[3 * (int64_t)r]), 0.0f);
        gv.y = fmaxf(expm1f(y[3 * (int64_t)r + 1]), 0.0f);
        gv.z = fmaxf(expm1f(y[3 * (int64_t)r + 2]), 0.0f);
    }
    guess[p] = gv;
}

// The first warm step for each receiver (in count order, its transfers
// from its slice lane): A = the transfers' gather of the guess's shot
// light, then light = B1 + A (the Jacobi step from the guess), emission =
// light - guess (the change, which later bounces carry on).
__device__ __forceinline__ F3 warm_combine(const BounceView &v, int i, const int32_t *__restrict__ order,
                                           const uint32_t *__restrict__ sorted, const int64_t *__restrict__ sell_off,
                                           const int2 *__restrict__ sell, const float4 *__restrict__ guess,
                                           const float4 *__restrict__ first, float4 *__restrict__ total,
                                           float4 *__restrict__ emit_out, float4 *__restrict__ shoot_out, int &p) {
    p = __ldg(&v.recv[__ldg(&order[i])]);
    const int n = sell_count(__ldg(&sorted[i]));
    const int2 *src = sell + __ldg(&sell_off[i >> 5]) + (i & 31);
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    for (int j = 0; j < n; j++) {
        const int2 t = __ldg(&src[32 * (int64_t)j]);
        const float w = __int_as_float(t.y);
        const float4 gs = guess[t.x], rf = __ldg(&v.refl[t.x]);
        sx += gs.x * rf.x * w;
        sy += gs.y * rf.y * w;
        sz += gs.z * rf.z * w;
    }
    if (__ldg(&v.tree[p].w)) {
        emit_out[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        shoot_out[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        p = -1;
        return {0.0f, 0.0f, 0.0f};
    }
    const float4 b1 = first[p], gv = guess[p];
    const float4 t = make_float4(b1.x + sx, b1.y + sy, b1.z + sz, 0.0f);
    total[p] = t;
    const float4 d = make_float4(t.x - gv.x, t.y - gv.y, t.z - gv.z, 0.0f);
    emit_out[p] = d;
    const float4 rf = __ldg(&v.refl[p]);
    shoot_out[p] = make_float4(d.x * rf.x, d.y * rf.y, d.z * rf.z, 0.0f);
    return f3(d);
}

__global__ void __launch_bounds__(kBounceBlock)
    k_warm_combine(BounceView v, const int32_t *__restrict__ order, const uint32_t *__restrict__ sorted,
                   const int64_t *__restrict__ sell_off, const int2 *__restrict__ sell, const float4 *__restrict__ guess,
                   const float4 *__restrict__ first, float4 *__restrict__ total, float4 *__restrict__ emit_out,
                   float4 *__restrict__ shoot_out, const int32_t *__restrict__ leaf_rank, int32_t nleaves,
                   double *__restrict__ sums) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    F3 e = {0.0f, 0.0f, 0.0f};
    int p = -1;
    if (i < v.nreceivers) e = warm_combine(v, i, order, sorted, sell_off, sell, guess, first, total, emit_out, shoot_out, p);
    add_totals(e, p >= 0 ? (double)(nleaves - __ldg(&leaf_rank[p])) : 0.0, sums);
}

unsigned blocks(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

}  // namespace

void BounceBuffers::release() {
    void *ptrs[] = {origin, normal, mins, maxs, refl, tree, wind, points, face_range, face_samples, face_plane,
                    recv, start, row_off, row_faces, sample_area, cand_off, seg_off, group_off, warp_group, cand_src, cand_w, tr_off, tr, scan_tmp,
                    direct, total, emit[0], emit[1], shoot[0], shoot[1], sums, exact, exact_sums, exact_steps, counters, leaf_desc,
                    face_level, level_off, parent_list, parent, share, patch_box, root_plane, root_origin, root_tree, leaf_rank,
                    sell_key, sell_idx, sell_sorted, sell_order, sell_off, sell, sort_tmp,
                    first, guess, feat, pred,
                    pr_off, pr_patch, pr_box, pr_coord, prad_light, prad_weight};
    for (void *q : ptrs) dev_free(q);
    for (cudaGraphExec_t &g : bounce_graph)
        if (g) cudaGraphExecDestroy(g);
    // The pinned stop-rule sums stay for the next upload (freeing pinned
    // memory can stall); free_pinned() frees them.
    double *parts_h = h_parts;
    float *exact_h = h_exact;
    *this = BounceBuffers();
    h_parts = parts_h;
    h_exact = exact_h;
}

void BounceBuffers::free_pinned() {
    cudaFreeHost(h_parts);
    cudaFreeHost(h_exact);
    h_parts = nullptr;
    h_exact = nullptr;
}

template <int OP>
static cudaError_t launch_parents(const BounceBuffers &b, float4 *light, float4 *emit, float4 *shoot,
                                  cudaStream_t stream) {
    if (b.nparents == 0) return cudaSuccess;
    k_parents<OP><<<b.nfaces, kFaceThreads, 0, stream>>>(
        b.view, b.face_level, b.level_off, b.parent, b.share, light, emit, shoot);
    return cudaGetLastError();
}

cudaError_t launch_bounce_tables(const BounceBuffers &b, const FinalView &fv, float4 *face_fit, cudaStream_t stream) {
    if (b.nfaces)
        k_face_fit<<<blocks((int64_t)b.nfaces * 32, kBounceBlock), kBounceBlock, 0, stream>>>(
            b.view, fv.face_cells, fv.frames, fv.cell_sample, face_fit);
    if (b.nfaces)
        k_roots<<<blocks(b.nfaces, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, b.root_plane, b.root_origin,
                                                                             b.root_tree);
    if (b.npatches)
        k_patch_boxes<<<blocks(b.npatches, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, fv.frames, face_fit,
                                                                                     b.patch_box);
    if (b.nparents)
        k_parent_records<<<blocks(b.nparents, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, b.parent_list, b.nparents,
                                                                                        b.parent, b.share);
    return cudaGetLastError();
}

cudaError_t launch_warp_groups(const BounceBuffers &b, cudaStream_t stream) {
    if (b.grouped()) k_warp_groups<<<blocks(b.ngroups(), 128), 128, 0, stream>>>(b.ngroups(), b.group_off, b.warp_group);
    return cudaGetLastError();
}

cudaError_t launch_sell_pad(const BounceBuffers &b, unsigned long long *d_pad, cudaStream_t stream) {
    if (b.nreceivers == 0) return cudaSuccess;
    k_sell_pad<<<blocks(b.nreceivers, b.sell_window), 256, 0, stream>>>(b.nreceivers, b.sell_window, b.cand_off, d_pad);
    return cudaGetLastError();
}

cudaError_t sell_sort(BounceBuffers &b, int32_t window, void *tmp, size_t &bytes, cudaStream_t stream) {
    const int nwindows = (int)blocks(b.nreceivers, window);
    int bits = kCountBits;
    while (bits < 32 && ((int64_t)nwindows - 1) >> (bits - kCountBits)) bits++;
    return cub::DeviceRadixSort::SortPairs(tmp, bytes, b.sell_key, b.sell_sorted, b.sell_idx, b.sell_order, b.nreceivers,
                                           0, bits, stream);
}

cudaError_t launch_patch_light(const BounceBuffers &b, const FinalView &fv, const float4 *sample_light,
                               cudaStream_t stream) {
    if (b.npatches == 0) return cudaSuccess;
    k_patch_samples<<<blocks(b.npatches, kBounceBlock), kBounceBlock, 0, stream>>>(
        b.view, b.patch_box, fv.face_cells, fv.frames, fv.cell_sample, sample_light, b.direct, b.total, b.emit[0],
        b.shoot[0]);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_parents<kOpDirect>(b, b.direct, b.emit[0], b.shoot[0], stream);
}

// The transfer build.  count_only: the candidate counts and offsets alone
// (at upload: they size the buffers, and they depend only on the patch
// tree and the PVS rows, so they stay valid until the next upload).
// Otherwise, with those offsets, the candidates written, their rays and
// form factors, and the transfer lists; counters[1..2] are added to.
cudaError_t launch_transfers(BounceBuffers &b, const DeviceScene &scene, uint32_t *overflow, cudaStream_t stream,
                             bool count_only) {
    const int R = b.nreceivers;
    if (R == 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    size_t tmp = 0;
    if (count_only) {
        // Candidate counts into cand_off[1..R], then the exclusive scan.
        k_candidates<false><<<dim3(blocks(R, kBounceBlock), b.segments), kBounceBlock, 0, stream>>>(
            b.view, b.root_plane, b.root_origin, b.root_tree, nullptr, b.seg_off + 1, nullptr, overflow);
        e = cudaMemsetAsync(b.seg_off, 0, sizeof(int64_t), stream);
        if (e != cudaSuccess) return e;
        tmp = b.scan_tmp_bytes;
        e = cub::DeviceScan::InclusiveSum(b.scan_tmp, tmp, b.seg_off + 1, b.seg_off + 1, (int64_t)R * b.segments, stream);
        if (e == cudaSuccess)
            e = cudaMemcpy2DAsync(b.cand_off, sizeof(int64_t), b.seg_off, sizeof(int64_t) * (size_t)b.segments,
                                  sizeof(int64_t), (size_t)R + 1, cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess || !b.grouped()) return e != cudaSuccess ? e : cudaGetLastError();
        // The transfer rays' warps by group.
        k_group_warps<<<blocks(b.ngroups(), kBounceBlock), kBounceBlock, 0, stream>>>(R, b.ngroups(), b.cand_off,
                                                                                     b.group_off + 1);
        e = cudaMemsetAsync(b.group_off, 0, sizeof(int64_t), stream);
        if (e != cudaSuccess) return e;
        tmp = b.scan_tmp_bytes;
        e = cub::DeviceScan::InclusiveSum(b.scan_tmp, tmp, b.group_off + 1, b.group_off + 1, b.ngroups(), stream);
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    k_candidates<true><<<dim3(blocks(R, kBounceBlock), b.segments), kBounceBlock, 0, stream>>>(
        b.view, b.root_plane, b.root_origin, b.root_tree, b.seg_off, nullptr, b.cand_src, overflow);
    if (!scene.one_copy) k_starts<<<blocks(R, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, scene.opaque, b.start);
    const size_t stack = sizeof(int) * scene.stack_depth() * kBlock;
    by_copies(scene, [&](auto one) {
        constexpr bool kOne = decltype(one)::value;
        if (!b.grouped() && b.ncand > 0)
            k_transfer<kOne, kBlock><<<blocks(b.ncand, kBlock), kBlock, stack, stream>>>(
                b.view, scene, b.cand_off, b.cand_src, b.start, b.cand_w, b.ncand, &b.counters[2]);
        if (b.transfer_warps > 0)
            k_transfer_groups<kOne, kBlock><<<blocks(32 * b.transfer_warps, kBlock), kBlock, stack, stream>>>(
                b.view, scene, b.cand_off, b.cand_src, b.start, b.group_off, b.warp_group, b.transfer_warps, b.cand_w,
                &b.counters[2]);
    });
    k_transfer_count<<<blocks((int64_t)R * 32, kBounceBlock), kBounceBlock, 0, stream>>>(
        R, b.cand_off, b.cand_w, b.tr_off + 1, &b.counters[1]);
    e = cudaMemsetAsync(b.tr_off, 0, sizeof(int64_t), stream);
    if (e != cudaSuccess) return e;
    tmp = b.scan_tmp_bytes;
    e = cub::DeviceScan::InclusiveSum(b.scan_tmp, tmp, b.tr_off + 1, b.tr_off + 1, R, stream);
    if (e != cudaSuccess) return e;
    if (!b.tr) return cudaGetLastError();
    k_transfer_write<<<blocks((int64_t)R * 32, kBounceBlock), kBounceBlock, 0, stream>>>(
        R, b.cand_off, b.cand_src, b.cand_w, b.tr_off, b.tr);
    e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_sell(b, b.sell_window, stream);
}

// The gather's slices (SELL-32) from the transfer lists tr_off / tr.
cudaError_t launch_sell(BounceBuffers &b, int32_t window, cudaStream_t stream) {
    const int R = b.nreceivers;
    if (R == 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    size_t tmp = 0;
    const int nslices = (R + 31) / 32;
    k_sell_keys<<<blocks(R, kBounceBlock), kBounceBlock, 0, stream>>>(R, window, b.tr_off, b.sell_key, b.sell_idx);
    tmp = b.sort_tmp_bytes;
    e = sell_sort(b, window, b.sort_tmp, tmp, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.sell_off, 0, sizeof(int64_t), stream);
    if (e != cudaSuccess) return e;
    k_sell_width<<<blocks(nslices, kBounceBlock), kBounceBlock, 0, stream>>>(nslices, b.sell_sorted, b.sell_off + 1);
    tmp = b.scan_tmp_bytes;
    e = cub::DeviceScan::InclusiveSum(b.scan_tmp, tmp, b.sell_off + 1, b.sell_off + 1, nslices, stream);
    if (e != cudaSuccess) return e;
    k_sell_pack<<<blocks(R, kBounceBlock), kBounceBlock, 0, stream>>>(R, b.sell_order, b.sell_sorted, b.sell_off,
                                                                      b.tr_off, b.tr, b.sell);
    return cudaGetLastError();
}

// Bounce number `bounce` (0-based): reads shoot[bounce & 1], writes the
// other half, then the fp64 totals.
cudaError_t launch_gather(BounceBuffers &b, int bounce, cudaStream_t stream) {
    const int in = bounce & 1, out = in ^ 1;
    cudaError_t e = cudaMemsetAsync(b.sums, 0, kSumParts * kSums * sizeof(double), stream);
    if (e != cudaSuccess) return e;
    if (b.nreceivers)
        k_gather<<<blocks(b.nreceivers, kBounceBlock), kBounceBlock, 0, stream>>>(
            b.view, b.sell_order, b.sell_sorted, b.sell_off, b.sell, b.shoot[in], b.total, b.emit[out], b.shoot[out],
            b.leaf_rank, b.nleaves, b.sums);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_parents<kOpCollect>(b, b.total, b.emit[out], b.shoot[out], stream);
    b.last_buffer = out;
    return e;
}

cudaError_t launch_features(BounceBuffers &b, const DeviceWorld &w, cudaStream_t stream) {
    if (!b.nreceivers) return cudaSuccess;
    k_features<<<blocks(b.nreceivers, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, b.direct, b.first, w.lights,
                                                                                w.nlights, b.feat);
    return cudaGetLastError();
}

// The warm start after bounce 0 (which left B1 in b.first): the guess from
// the network, blended to the parents, the first warm step into the other
// emit/shoot half, the parents' light and emission, and the totals.
cudaError_t launch_warm_start(BounceBuffers &b, const DeviceWorld &w, const vrad_mlp &m, cudaStream_t stream) {
    if (!b.nreceivers) return cudaSuccess;
    cudaError_t e = launch_features(b, w, stream);
    if (e == cudaSuccess) e = mlp_forward(m, b.feat, b.nreceivers, b.pred, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.guess, 0, sizeof(float4) * (size_t)b.npatches, stream);
    if (e != cudaSuccess) return e;
    k_guess<<<blocks(b.nreceivers, kBounceBlock), kBounceBlock, 0, stream>>>(b.view, b.pred, b.guess);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_parents<kOpGuess>(b, b.guess, nullptr, nullptr, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(b.sums, 0, kSumParts * kSums * sizeof(double), stream);
    if (e != cudaSuccess) return e;
    // Bounce 0 wrote half 1; the warm step writes half 0, as bounce 1 would.
    k_warm_combine<<<blocks(b.nreceivers, kBounceBlock), kBounceBlock, 0, stream>>>(
        b.view, b.sell_order, b.sell_sorted, b.sell_off, b.sell, b.guess, b.first, b.total, b.emit[0], b.shoot[0],
        b.leaf_rank, b.nleaves, b.sums);
    e = cudaGetLastError();
    b.last_buffer = 0;
    return e != cudaSuccess ? e : launch_parents<kOpCollect>(b, b.total, b.emit[0], b.shoot[0], stream);
}

cudaError_t launch_bounce_graph(BounceBuffers &b, int bounce, cudaStream_t capture, cudaStream_t stream) {
    const int k = bounce & 1;
    if (!b.bounce_graph[k]) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(capture, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return e;
        cudaError_t inside = launch_gather(b, bounce, capture);
        if (inside == cudaSuccess)
            inside = cudaMemcpyAsync(b.h_parts, b.sums, kSumParts * kSums * sizeof(double), cudaMemcpyDeviceToHost,
                                     capture);
        e = cudaStreamEndCapture(capture, &g);
        if (e == cudaSuccess) e = inside;
        if (e == cudaSuccess) e = cudaGraphInstantiate(&b.bounce_graph[k], g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            b.bounce_graph[k] = nullptr;
            return e;
        }
    }
    b.last_buffer = k ^ 1;
    return cudaGraphLaunch(b.bounce_graph[k], stream);
}

cudaError_t alloc_exact(BounceBuffers &b) {
    // Chunks of 512 leaves, or larger ones so that there are 4096 at most (a
    // chunk's block adds up the sums before it).
    b.exact_per = (int32_t)std::max<int64_t>(512, ((int64_t)b.nleaves + 4095) / 4096);
    b.exact_chunks = (int32_t)(((int64_t)b.nleaves + b.exact_per - 1) / b.exact_per);
    const size_t n = 3 * (size_t)std::max(b.exact_chunks, 1);
    cudaError_t e = dev_alloc(&b.exact, 3 * sizeof(float));
    if (e == cudaSuccess) e = dev_alloc(&b.exact_sums, n * sizeof(double));
    if (e == cudaSuccess) e = dev_alloc(&b.exact_steps, n * sizeof(ExactStep));
    return e;
}

cudaError_t launch_exact_total(BounceBuffers &b, int bounce, cudaStream_t stream) {
    const float4 *emit = b.emit[(bounce & 1) ^ 1];
    ExactStep *steps = (ExactStep *)b.exact_steps;
    const int nchunks = b.exact_chunks;
    if (nchunks) {
        k_exact_sums<<<nchunks, kExactBlock, 0, stream>>>(b.leaf_desc, b.nleaves, b.exact_per, nchunks, emit,
                                                          b.exact_sums);
        k_exact_steps<<<nchunks, kExactBlock, 0, stream>>>(b.leaf_desc, b.nleaves, b.exact_per, nchunks, emit,
                                                           b.exact_sums, steps);
    }
    k_exact_walk<<<1, 96, 0, stream>>>(b.leaf_desc, b.nleaves, b.exact_per, nchunks, emit, steps, b.exact);
    return cudaGetLastError();
}

}  // namespace vrad

// ---- form factors on their own (inspection) ----------------------------------
//
// The transfer build's DiffToDiff and PolyToDiff, evaluated for caller-given
// cases by the same device functions k_transfer calls, so the reference's
// known-answer cases (Tests/MapTools/Rad/Bounce/FormFactorsTests.cs) run on
// the device's own arithmetic.

namespace {

__global__ void k_ff_diff(const float *__restrict__ c, int64_t n, float *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *q = c + 12 * i;
    out[i] = vrad::diff_to_diff({q[0], q[1], q[2]}, {q[3], q[4], q[5]}, {q[6], q[7], q[8]}, {q[9], q[10], q[11]});
}

__global__ void k_ff_poly(const float4 *__restrict__ pts, const int32_t *__restrict__ first,
                          const float *__restrict__ c, int64_t n, float *__restrict__ out,
                          unsigned long long *open) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *q = c + 7 * i;
    out[i] = vrad::poly_to_diff_pts(pts + first[i], first[i + 1] - first[i], q[0], {q[1], q[2], q[3]},
                                    {q[4], q[5], q[6]}, open);
}

// Copies `bytes` from host to a fresh device block (the inspection calls'
// own small temporaries).
cudaError_t upload_tmp(void **d, const void *h, size_t bytes, cudaStream_t s) {
    cudaError_t e = cudaMalloc(d, bytes ? bytes : 16);
    if (e == cudaSuccess && bytes) e = cudaMemcpyAsync(*d, h, bytes, cudaMemcpyHostToDevice, s);
    return e;
}

}  // namespace

extern "C" int32_t vrad_form_factor_diff(vrad_ctx *ctx, const float *cases, int64_t n, float *out) {
    if (!ctx || n < 0 || (n && (!cases || !out))) return vrad_fail(ctx, VRAD_ERR_ARG, "invalid form factor cases");
    if (n == 0) return VRAD_OK;
    std::lock_guard<std::mutex> g(ctx->mu);
    void *dc = nullptr, *dout = nullptr;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess) e = upload_tmp(&dc, cases, sizeof(float) * 12 * (size_t)n, ctx->stream);
    if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(float) * (size_t)n);
    if (e == cudaSuccess) {
        k_ff_diff<<<(unsigned)((n + 127) / 128), 128, 0, ctx->stream>>>(static_cast<const float *>(dc), n,
                                                                      static_cast<float *>(dout));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = vrad::wait_stream(ctx->stream);
    cudaFree(dc);
    cudaFree(dout);
    return e == cudaSuccess ? VRAD_OK : vrad_cuda_fail(ctx, e, "form factors");
}

extern "C" int32_t vrad_form_factor_poly(vrad_ctx *ctx, const float *points, const int32_t *first,
                                         const float *cases, int64_t n, float *out) {
    if (!ctx || n < 0 || (n && (!points || !first || !cases || !out)))
        return vrad_fail(ctx, VRAD_ERR_ARG, "invalid form factor cases");
    if (n == 0) return VRAD_OK;
    for (int64_t i = 0; i < n; i++)
        if (first[i] < 0 || first[i + 1] < first[i] + 3)
            return vrad_fail(ctx, VRAD_ERR_ARG, "winding %lld has fewer than three points", (long long)i);
    const int64_t np = first[n];
    std::vector<float4> pts((size_t)np);
    for (int64_t k = 0; k < np; k++) pts[(size_t)k] = make_float4(points[3 * k], points[3 * k + 1], points[3 * k + 2], 0.0f);
    std::lock_guard<std::mutex> g(ctx->mu);
    void *dp = nullptr, *df = nullptr, *dc = nullptr, *dout = nullptr, *dopen = nullptr;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess) e = upload_tmp(&dp, pts.data(), sizeof(float4) * (size_t)np, ctx->stream);
    if (e == cudaSuccess) e = upload_tmp(&df, first, sizeof(int32_t) * (size_t)(n + 1), ctx->stream);
    if (e == cudaSuccess) e = upload_tmp(&dc, cases, sizeof(float) * 7 * (size_t)n, ctx->stream);
    if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(float) * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&dopen, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemsetAsync(dopen, 0, sizeof(unsigned long long), ctx->stream);
    if (e == cudaSuccess) {
        k_ff_poly<<<(unsigned)((n + 127) / 128), 128, 0, ctx->stream>>>(
            static_cast<const float4 *>(dp), static_cast<const int32_t *>(df), static_cast<const float *>(dc), n,
            static_cast<float *>(dout), static_cast<unsigned long long *>(dopen));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = vrad::wait_stream(ctx->stream);
    for (void *q : {dp, df, dc, dout, dopen}) cudaFree(q);
    return e == cudaSuccess ? VRAD_OK : vrad_cuda_fail(ctx, e, "form factors");
}
