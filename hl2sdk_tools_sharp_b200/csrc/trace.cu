// trace.cu -- ray traversal kernels: any-hit visibility, closest hit, and
// sky-passing visibility, over the BVH built in scene.cu.
//
// Per-triangle arithmetic is the reference's KdRayTracer.IntersectTriangle
// (MapTools/Tracing/KdRayTracer.cs:1194-1267) operation for operation, each
// an explicitly rounded intrinsic, so an accepted/rejected decision and a
// hit distance are the CPU's bits.  What the traversal adds is only WHICH
// triangles get tested: every triangle whose padded box the segment meets,
// which includes every triangle the predicate can accept (the pad is far
// above the rounding of the box test and of the predicate's hit point).
//
// Work distribution: one ray per thread, 128-thread CTAs scheduled by the
// hardware (no shared work counter, so launches on different streams never
// interfere); a warp's 32 visibility bits are one 32-bit word written with
// a single store after a ballot.  The traversal stack lives in shared
// memory, one column per thread.

#include <cfloat>

#include "scene.cuh"
#include "traverse.cuh"

namespace vrad {

namespace {

// A ray of `rays` with the direction's reciprocals.
__device__ __forceinline__ RayState load_ray(const vrad_ray *__restrict__ ray, float &reach) {
    const float *f = reinterpret_cast<const float *>(ray);
    reach = __ldg(f + 6);
    return make_ray(__ldg(f + 0), __ldg(f + 1), __ldg(f + 2), __ldg(f + 3), __ldg(f + 4), __ldg(f + 5));
}

// A warp whose rays lie in more octants walks octant 0's copy of the nodes as
// a large scene's rays do (walk_one): the copies of six or eight octants at
// once leave L1 little to keep.  Rays in random directions, 2 M of them
// through soups of 1 k, 3 k and 10 k triangles, any hit: 0.60, 0.80 and 1.06
// ms by octants, 0.51, 0.73 and 1.03 so (one copy alone had 0.52, 0.75 and
// 1.03); warps of neighbouring rays, which seldom see more than four octants
// (a target straight ahead), take as long as before, 4.2 M closest hits on the
// 8x8 room grid 300 us against 299.  A call of its own, so that the walk by
// octants keeps its registers.
//
// Not for a batch that leaves the chip part idle, whose time is its longest
// ray's: by octants that has fewer instructions a node.  1 k triangles, by
// octants and so: 1,024 rays 31.4 and 35.4 us, 32,768 36.6 and 39.5, 65,536
// 41.7 and 40.6, 131,072 53.6 and 49.6.
constexpr int kTogether = 4;
constexpr int64_t kApartRays = 65536;

template <int MODE>
__device__ __noinline__ int4 trace_apart(const DeviceScene &s, const vrad_ray *ray, const TraceParams &p, int *stack) {
    float reach, best_t;
    const RayState r = load_ray(ray, reach);
    bool hit;
    int32_t best_orig;
    uint32_t best_meta;
    trace_ray<true, MODE>(s, r, p.tmin, reach, p.skip_id, 0, stack, hit, best_t, best_orig, best_meta);
    return make_int4(hit ? 1 : 0, __float_as_int(best_t), best_orig, 0);
}

// APART: the batch is large enough for trace_apart.
template <bool ONE, bool APART, int MODE>
__global__ void __launch_bounds__(kBlock) k_trace(const __grid_constant__ DeviceScene s,
                                                  const vrad_ray *__restrict__ rays, int64_t n,
                                                  const __grid_constant__ TraceParams p, uint32_t *__restrict__ bits,
                                                  vrad_hit *__restrict__ hits) {
    extern __shared__ int stack_mem[];  // sc.stack_depth() entries per thread
    int *stack = stack_mem + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    if (i - lane >= n) return;  // whole warp past the end
    bool hit = false;
    float best_t = 0.0f, reach = 1.0f;
    int32_t best_orig = -1;
    uint32_t best_meta = 0;
    const unsigned live = __ballot_sync(kFull, i < n);
    if (i < n) {
        const RayState r = load_ray(rays + i, reach);
        if (ONE) {
            trace_ray<true, MODE>(s, r, p.tmin, reach, p.skip_id, 0, stack, hit, best_t, best_orig, best_meta);
        } else if (APART && octants_of(live, r) > kTogether) {
            const int4 h = trace_apart<MODE>(s, rays + i, p, stack);
            hit = h.x != 0;
            best_t = __int_as_float(h.y);
            best_orig = h.z;
        } else {
            trace_ray<false, MODE>(s, r, p.tmin, reach, p.skip_id, 0, stack, hit, best_t, best_orig, best_meta);
        }
    }
    if (MODE == kModeClosest) {
        if (i < n) {
            vrad_hit h;
            if (hit) {
                h.surface = __ldg(&s.tri_id[best_orig]);
                h.fraction = reach == 1.0f ? best_t : __fdiv_rn(best_t, reach);
            } else {
                h.surface = -1;
                h.fraction = 1.0f;
            }
            hits[i] = h;
        }
    } else {
        const uint32_t word = __ballot_sync(kFull, hit);
        if (lane == 0) bits[i >> 5] = word;
    }
}

}  // namespace

cudaError_t launch_trace(const DeviceScene &scene, const vrad_ray *d_rays, int64_t n,
                         const TraceParams &p, uint32_t *d_bits, vrad_hit *d_hits,
                         cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const int64_t grid = (n + kBlock - 1) / kBlock;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    const size_t smem = sizeof(int) * (size_t)scene.stack_depth() * kBlock;
    auto launch = [&](auto one, auto apart) {
        constexpr bool kOne = decltype(one)::value, kApart = decltype(apart)::value;
        switch (p.mode) {
            case kModeAny:
                k_trace<kOne, kApart, kModeAny><<<(unsigned)grid, kBlock, smem, stream>>>(scene, d_rays, n, p, d_bits, d_hits);
                break;
            case kModeClosest:
                k_trace<kOne, kApart, kModeClosest><<<(unsigned)grid, kBlock, smem, stream>>>(scene, d_rays, n, p, d_bits,
                                                                                            d_hits);
                break;
            default:
                k_trace<kOne, kApart, kModeSkyPass><<<(unsigned)grid, kBlock, smem, stream>>>(scene, d_rays, n, p, d_bits,
                                                                                            d_hits);
                break;
        }
    };
    if (scene.one_copy) launch(std::true_type{}, std::false_type{});
    else if (n > kApartRays) launch(std::false_type{}, std::true_type{});
    else launch(std::false_type{}, std::false_type{});
    return cudaGetLastError();
}

static_assert(VRAD_STATIC_MAX_RAYS <= kApartRays, "the allocation-free entry launches no kernel that is not loaded here");

cudaError_t load_visibility_kernels() {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, k_trace<false, false, kModeAny>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_trace<false, false, kModeSkyPass>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_trace<true, false, kModeAny>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_trace<true, false, kModeSkyPass>);
    return e;
}

}  // namespace vrad
