// ambient.cu -- the leaf ambient sample on the device: at each position the
// 162 rays into the map through the BSP surface walk, each hit's lightmap
// colour blended by the cone, projected onto the six sides of the cube.
//
// Reference behaviour restated (muflub/hl2sdk_tools_sharp, MapTools/Rad/Ambient):
//   AmbientSampler.ComputeRayCube (AmbientSampler.cs:211-227): ray i runs
//     from the position to position + anorm[i] x RayLength (32768 x 1.74);
//     its delta is end - start, in float; only light style 0 is kept;
//   RayAmbientLighting.Accumulate (RayAmbientLighting.cs:89-134): the cone's
//     radius at the hit, |delta| x tan(7.275 deg) x fraction, remapped from
//     [20, 40] to [0, 1] is the face average's weight (1 for a sky hit, which
//     has no luxel), the rest the luxel's;
//   AddFaceAverage (:196-226): a sky face gives the sky ambient; a lit face
//     each style-0 slot's decoded, tinted average (AmbientScene.cs:280-300);
//   AddFacePointSample (:241-291): the luxel (truncated, clamped to the
//     lightmap), each slot's RGBE decoded by the (float)(2^(e-128) / 255)
//     table (StockLightColor.cs:69-78, 262-271), tinted by reflectivity or,
//     on a sky face, replaced by the sky ambient;
//   AmbientCube.Project (AmbientCube.cs:80-103): per side, the rays whose
//     direction has a positive cosine with the side, weighted by it, summed
//     in table order, times 1 / (sum of the weights).
// Every float operation is an explicitly rounded intrinsic in the
// reference's order, so a cube is the reference's bits.
//
// Work distribution.  One ray per thread.  The walk is divergent (an
// average ray takes 18 nodes and 15 face tests, some take hundreds), so
// what counts is that a warp's rays go the same way.  Samples come in
// groups of 32, 162 warps a group: where the group's points lie close
// together (kCompact), a warp takes one direction from all 32; otherwise 32
// directions, grouped by octant, from one point.  The lanes' walks fill
// 0.41 of the warp's steps the first way on dm_lockdown's leaves against
// 0.25 in table order, 0.16 when the points lie apart; 0.28 by octant.
// Each ray writes its colour to a chunk scratch (12 B), planes of one
// channel of one direction, so that neighbouring samples lie together; and
// k_ambient_project runs one warp per side of 32 samples, summing their 162
// colours in table order.

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "ambient.cuh"
#include "bsp_walk.cuh"
#include "context.cuh"
#include "device_pool.h"

namespace vrad {

void AmbientBuffers::release() {
    for (void *p : {(void *)light, (void *)faces, (void *)directions, (void *)by_octant, (void *)facing, (void *)power2n, (void *)rad, (void *)flags})
        dev_free(p);
    light = nullptr;
    faces = nullptr;
    by_octant = nullptr;
    facing = nullptr;
    directions = power2n = rad = nullptr;
    flags = nullptr;
    rad_samples = 0;
    ready = false;
    view = AmbientView{};
}

namespace {

constexpr int kRayBlock = 128;
constexpr int kProjectBlock = 32 * kAmbientSides * 3;
constexpr int64_t kChunkSamples = 32768;  // at most 63.7 MB of ray colours
// A group's points are close together within this many units along each
// axis: 100 k samples of dm_lockdown 3.90 ms at 256, 3.57 at 512, 3.38 at
// 1024, the largest that was tried, 5.61 when no group is.
constexpr float kCompact = 1024.0f;
// At most this many samples take four rays a warp: 100 samples 111 us
// against 152 with 32, 300 samples 146 against 160, 768 samples 228 against
// 184.  The two cross somewhere between the last two; the line lies below.
constexpr int64_t kFewSamples = 256;
constexpr float kRayLength = 32768.0f * 1.74f;
constexpr uint32_t kFlagStack = 1, kFlagBadAverage = 2, kFlagOutsideLump = 4;

__device__ __forceinline__ void add_scaled(float &x, float &y, float &z, float cx, float cy, float cz, float s) {
    x = __fadd_rn(x, __fmul_rn(cx, s));
    y = __fadd_rn(y, __fmul_rn(cy, s));
    z = __fadd_rn(z, __fmul_rn(cz, s));
}

// The warp's range (largest minus smallest) of v; NaN counts as a large one.
__device__ __forceinline__ float warp_range(float v) {
    // Floats as integers in the floats' order.
    auto key = [](float f) {
        const uint32_t u = __float_as_uint(f);
        return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
    };
    auto value = [](uint32_t k) { return __uint_as_float(k & 0x80000000u ? k ^ 0x80000000u : ~k); };
    const uint32_t k = key(v);
    return value(__reduce_max_sync(0xffffffffu, k)) - value(__reduce_min_sync(0xffffffffu, k));
}

__global__ void __launch_bounds__(kRayBlock) k_ambient_rays(DeviceBsp g, AmbientView a,
                                                            const float *__restrict__ positions, int64_t nsamples,
                                                            float *__restrict__ rad, int64_t pitch, int lanes,
                                                            uint32_t *flags) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * kRayBlock + threadIdx.x) >> 5;
    const int per_group = kAmbientDirs * 32 / lanes;
    const int64_t group = warp / per_group;
    const int w = (int)(warp - group * per_group);
    const int64_t s0 = 32 * group;
    if (s0 >= nsamples) return;  // whole warps
    const int m = nsamples - s0 < 32 ? (int)(nsamples - s0) : 32;  // the group's samples
    const float *p = positions + 3 * (s0 + (lane < m ? lane : m - 1));
    float sx = __ldg(p), sy = __ldg(p + 1), sz = __ldg(p + 2);
    const bool compact = warp_range(sx) <= kCompact && warp_range(sy) <= kCompact && warp_range(sz) <= kCompact;
    int k, i;  // the sample within the group, the direction
    bool live = lane < lanes;  // the walk takes whole warps
    float ax, ay, az;
    if (compact) {
        const int part = 32 / lanes;
        k = w % part * lanes + lane;
        i = w / part;
        ax = __ldg(a.directions + 3 * i);
        ay = __ldg(a.directions + 3 * i + 1);
        az = __ldg(a.directions + 3 * i + 2);
    } else {
        const int j = lanes * w + lane;
        k = j / kAmbientDirs;
        const float4 d = __ldg(&a.by_octant[j % kAmbientDirs]);
        ax = d.x;
        ay = d.y;
        az = d.z;
        i = __float_as_int(d.w);
    }
    live = live && k < m;
    const int64_t s = s0 + (live ? k : 0);
    sx = __ldg(positions + 3 * s);
    sy = __ldg(positions + 3 * s + 1);
    sz = __ldg(positions + 3 * s + 2);
    bspwalk::Walk c;
    c.ox = sx;
    c.oy = sy;
    c.oz = sz;
    c.dx = __fsub_rn(__fadd_rn(sx, __fmul_rn(ax, kRayLength)), sx);
    c.dy = __fsub_rn(__fadd_rn(sy, __fmul_rn(ay, kRayLength)), sy);
    c.dz = __fsub_rn(__fadd_rn(sz, __fmul_rn(az, kRayLength)), sz);
    c.hit_frac = 1.0f;
    c.min_frac = 0.0f;
    c.surface = -1;
    c.has_luxel = false;
    c.luxel_s = c.luxel_t = 0.0f;
    float rx = 0.0f, ry = 0.0f, rz = 0.0f;  // light style 0
    const bool ok = bspwalk::walk(g, c, live);
    if (!live) return;
    if (!ok) {
        atomicOr(flags, kFlagStack);
    } else if (c.surface >= 0) {
        const vrad_ambient_face &F = a.faces[c.surface];
        const int32_t fflags = F.flags, nstyles = F.nstyles;
        const uint32_t styles = F.styles;
        // RemapValClamped(|delta| tan(theta) fraction, 20, 40, 0, 1).
        const float len = __fsqrt_rn(bspwalk::dot3(c.dx, c.dy, c.dz, c.dx, c.dy, c.dz));
        const float dist = __fmul_rn(__fmul_rn(len, a.tan_theta), c.hit_frac);
        float cv = __fdiv_rn(__fsub_rn(dist, 20.0f), __fsub_rn(40.0f, 20.0f));
        if (cv < 0.0f) cv = 0.0f;
        else if (cv > 1.0f) cv = 1.0f;
        float scale_avg = __fadd_rn(0.0f, __fmul_rn(__fsub_rn(1.0f, 0.0f), cv));
        if (!c.has_luxel) scale_avg = 1.0f;
        const float scale_sample = __fsub_rn(1.0f, scale_avg);
        if (scale_avg != 0.0f) {
            if (fflags & VRAD_AMBIENT_SKY) {
                if (a.has_sky) add_scaled(rx, ry, rz, a.sky[0], a.sky[1], a.sky[2], scale_avg);
            } else if (fflags & VRAD_AMBIENT_BAD_AVERAGE) {
                atomicOr(flags, kFlagBadAverage);
            } else {
                for (int m = 0; m < nstyles; m++)
                    if (((styles >> (8 * m)) & 0xFF) == 0)
                        add_scaled(rx, ry, rz, F.averages[m][0], F.averages[m][1], F.averages[m][2], scale_avg);
            }
        }
        if (scale_sample != 0.0f && F.lightofs != -1) {
            if (F.smax < 1 || F.tmax < 1) {
                atomicOr(flags, kFlagOutsideLump);
            } else {
                int ds = __float2int_rz(c.luxel_s), dt = __float2int_rz(c.luxel_t);
                ds = ds < 0 ? 0 : (ds > F.smax - 1 ? F.smax - 1 : ds);
                dt = dt < 0 ? 0 : (dt > F.tmax - 1 ? F.tmax - 1 : dt);
                const int32_t index = dt * F.smax + ds;
                const uint32_t last = (uint32_t)(int32_t)(a.light_bytes - 4);
                for (int m = 0; m < nstyles; m++) {
                    // int arithmetic that wraps, as the reference's does
                    const uint32_t ofs =
                        (uint32_t)F.lightofs + ((uint32_t)index + (uint32_t)m * (uint32_t)F.stride) * 4u;
                    if (a.light_bytes < 4 || ofs > last) {
                        atomicOr(flags, kFlagOutsideLump);
                        break;
                    }
                    const uint8_t *p = a.light + ofs;
                    const float e = __ldg(a.power2n + ((int)(int8_t)__ldg(p + 3) + 128));
                    float cx = __fmul_rn((float)__ldg(p), e), cy = __fmul_rn((float)__ldg(p + 1), e),
                          cz = __fmul_rn((float)__ldg(p + 2), e);
                    if (fflags & VRAD_AMBIENT_SKY) {
                        if (a.has_sky) {
                            cx = a.sky[0];
                            cy = a.sky[1];
                            cz = a.sky[2];
                        }
                    } else {
                        cx = __fmul_rn(cx, F.reflectivity[0]);
                        cy = __fmul_rn(cy, F.reflectivity[1]);
                        cz = __fmul_rn(cz, F.reflectivity[2]);
                    }
                    if (((styles >> (8 * m)) & 0xFF) == 0) add_scaled(rx, ry, rz, cx, cy, cz, scale_sample);
                }
            }
        }
    }
    float *o = rad + 3 * (int64_t)i * pitch + s;
    o[0] = rx;
    o[pitch] = ry;
    o[2 * pitch] = rz;
}

// One thread per (sample, side, channel), a warp 32 samples: the ordered sum
// over the directions that face the side, eight loads ahead of the adds.
__global__ void __launch_bounds__(kProjectBlock) k_ambient_project(const float *__restrict__ rad, int64_t pitch,
                                                                   int64_t nsamples, AmbientView a,
                                                                   float *__restrict__ cubes) {
    const int64_t s = 32 * (int64_t)blockIdx.x + (threadIdx.x & 31);
    const int j = (threadIdx.x >> 5) / 3, ch = (threadIdx.x >> 5) % 3;
    if (s >= nsamples) return;
    const float2 *f = a.facing + kAmbientDirs * j;
    const float *r = rad + ch * pitch + s;
    const int n = a.nfacing[j];
    float x = 0.0f;
    int q = 0;
    for (; q + 8 <= n; q += 8) {
        float c[8], v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 d = __ldg(&f[q + k]);
            c[k] = d.y;
            v[k] = __ldg(r + 3 * (int64_t)__float_as_int(d.x) * pitch);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) x = __fadd_rn(x, __fmul_rn(v[k], c[k]));
    }
    for (; q < n; q++) {
        const float2 d = __ldg(&f[q]);
        x = __fadd_rn(x, __fmul_rn(__ldg(r + 3 * (int64_t)__float_as_int(d.x) * pitch), d.y));
    }
    cubes[3 * (kAmbientSides * s + j) + ch] = __fmul_rn(x, a.inv[j]);
}

// Orders a caller's stream s after the context's stream (which every
// earlier call's kernels joined), so that calls on different streams take
// the chunk scratch in turn.  Not while s is being captured.
cudaError_t after_context(vrad_ctx *ctx, cudaStream_t s) {
    if (s == ctx->stream) return cudaSuccess;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &cap);
    if (e != cudaSuccess || cap != cudaStreamCaptureStatusNone) return e;
    e = cudaEventRecord(ctx->join, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ctx->join, 0);
    return e;
}

// The cubes of n device positions into device cubes, chunk by chunk.
int32_t cubes_on(vrad_ctx *ctx, const float *d_pos, int64_t n, float *d_cubes, cudaStream_t s) {
    if (!ctx->bsp.ready) return vrad_fail(ctx, VRAD_ERR_NO_SCENE, "no BSP uploaded");
    AmbientBuffers &A = ctx->ambient;
    if (!A.ready) return vrad_fail(ctx, VRAD_ERR_NO_SCENE, "no ambient lighting uploaded");
    if (A.view.nfaces != ctx->bsp.nsurfaces)
        return vrad_fail(ctx, VRAD_ERR_ARG, "the ambient lighting has %d faces, the BSP %d", A.view.nfaces,
                         ctx->bsp.nsurfaces);
    // Chunks of one size, whole groups of 32.
    const int64_t chunks = (n + kChunkSamples - 1) / kChunkSamples;
    const int64_t chunk = ((n + chunks - 1) / chunks + 31) / 32 * 32;
    cudaError_t e = after_context(ctx, s);
    if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "ordering the caller's stream");
    if (A.rad_samples < chunk) {
        e = wait_stream(s);  // the old scratch may still be in use
        if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "ambient scratch");
        dev_free(A.rad);
        A.rad = nullptr;
        A.rad_samples = 0;
        e = dev_alloc(&A.rad, sizeof(float) * 3 * kAmbientDirs * (size_t)chunk);
        if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "ambient ray scratch");
        A.rad_samples = chunk;
    }
    // Few samples leave the chip idle and take as long as their slowest
    // warp: four rays a warp, whose other lanes help with the long lists.
    const int lanes = n <= kFewSamples ? 4 : 32;
    for (int64_t b = 0; b < n && e == cudaSuccess; b += chunk) {
        const int64_t m = (n - b) < chunk ? (n - b) : chunk;
        const int64_t groups = (m + 31) / 32, threads = 32 * groups * (kAmbientDirs * 32 / lanes);
        k_ambient_rays<<<(unsigned)((threads + kRayBlock - 1) / kRayBlock), kRayBlock, 0, s>>>(
            ctx->bsp.view, A.view, d_pos + 3 * b, m, A.rad, A.rad_samples, lanes, A.flags);
        k_ambient_project<<<(unsigned)groups, kProjectBlock, 0, s>>>(A.rad, A.rad_samples, m, A.view,
                                                                    d_cubes + 3 * kAmbientSides * b);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? VRAD_OK : vrad_cuda_fail(ctx, e, "ambient cube launch");
}

int32_t read_flags(vrad_ctx *ctx) {
    uint32_t f = 0;
    cudaError_t e = cudaMemcpyAsync(&f, ctx->ambient.flags, sizeof f, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = wait_stream(ctx->stream);
    if (e == cudaSuccess && f) e = cudaMemsetAsync(ctx->ambient.flags, 0, sizeof f, ctx->stream);
    if (e == cudaSuccess && f) e = wait_stream(ctx->stream);
    if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "ambient status");
    if (f & kFlagStack)
        return vrad_fail(ctx, VRAD_ERR_CUDA, "the BSP walk went deeper than %d pending splits", bspwalk::kStack);
    if (f & kFlagBadAverage)
        return vrad_fail(ctx, VRAD_ERR_ARG, "a ray hit a face with light styles whose averages lie outside the lump");
    if (f & kFlagOutsideLump) return vrad_fail(ctx, VRAD_ERR_ARG, "a ray hit a luxel that lies outside the lump");
    return VRAD_OK;
}

}  // namespace
}  // namespace vrad

extern "C" int32_t vrad_ambient_upload(vrad_ctx *ctx, const vrad_ambient_lighting *L) {
    if (!ctx) return vrad_fail(nullptr, VRAD_ERR_ARG, "null context");
    if (!L || L->nfaces < 0 || (L->nfaces && !L->faces) || L->lighting_bytes < 0 ||
        L->lighting_bytes > 0x7fffffffLL || (L->lighting_bytes && !L->lighting) || !L->directions ||
        L->ndirections != vrad::kAmbientDirs || std::isnan(L->tan_theta))
        return vrad_fail(ctx, VRAD_ERR_ARG, "invalid ambient lighting");
    for (int32_t f = 0; f < L->nfaces; f++)
        if (L->faces[f].nstyles < 0 || L->faces[f].nstyles > 4)
            return vrad_fail(ctx, VRAD_ERR_ARG, "face %d has %d style slots", f, L->faces[f].nstyles);
    // StockLightColor's Power2N: (float)(2^(k - 128) / 255) in double, rounded once.
    float p2n[256];
    for (int k = 0; k < 256; k++) p2n[k] = (float)(std::ldexp(1.0, k - 128) / 255.0);
    // The directions octant by octant, in an order that changes one axis's
    // sign at a time.
    std::vector<float4> by_octant;
    for (const int oct : {0, 1, 3, 2, 6, 7, 5, 4})
        for (int i = 0; i < vrad::kAmbientDirs; i++) {
            const float *d = L->directions + 3 * i;
            if (((std::signbit(d[0]) ? 1 : 0) | (std::signbit(d[1]) ? 2 : 0) | (std::signbit(d[2]) ? 4 : 0)) != oct) continue;
            float4 v = make_float4(d[0], d[1], d[2], 0.0f);
            std::memcpy(&v.w, &i, sizeof i);
            by_octant.push_back(v);
        }
    // Per side (+x, -x, +y, -y, +z, -z) the directions with a positive cosine
    // and the weights' ordered float sum (host code rounds every operation).
    std::vector<float2> facing((size_t)vrad::kAmbientSides * vrad::kAmbientDirs);
    int32_t nfacing[vrad::kAmbientSides] = {};
    float inv[vrad::kAmbientSides];
    for (int j = 0; j < vrad::kAmbientSides; j++) {
        float t = 0.0f;
        for (int i = 0; i < vrad::kAmbientDirs; i++) {
            const float *d = L->directions + 3 * i, e = j & 1 ? -1.0f : 1.0f;
            const float c = (d[0] * (j / 2 == 0 ? e : 0.0f) + d[1] * (j / 2 == 1 ? e : 0.0f)) + d[2] * (j / 2 == 2 ? e : 0.0f);
            if (!(c > 0.0f)) continue;
            float2 v = make_float2(0.0f, c);
            std::memcpy(&v.x, &i, sizeof i);
            facing[(size_t)(vrad::kAmbientDirs * j + nfacing[j]++)] = v;
            t = t + c;
        }
        inv[j] = 1.0f / t;
    }
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess) e = vrad::quiesce(ctx);
    vrad::AmbientBuffers &A = ctx->ambient;
    A.release();
    auto up = [&](auto **dst, const void *src, size_t bytes) {
        cudaError_t r = vrad::dev_alloc(dst, bytes ? bytes : 16);
        if (r == cudaSuccess && bytes) r = cudaMemcpyAsync(*dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream);
        return r;
    };
    if (e == cudaSuccess) e = up(&A.light, L->lighting, (size_t)L->lighting_bytes);
    if (e == cudaSuccess) e = up(&A.faces, L->faces, sizeof(vrad_ambient_face) * (size_t)L->nfaces);
    if (e == cudaSuccess) e = up(&A.directions, L->directions, sizeof(float) * 3 * vrad::kAmbientDirs);
    if (e == cudaSuccess) e = up(&A.by_octant, by_octant.data(), sizeof(float4) * by_octant.size());
    if (e == cudaSuccess) e = up(&A.facing, facing.data(), sizeof(float2) * facing.size());
    if (e == cudaSuccess) e = up(&A.power2n, p2n, sizeof p2n);
    if (e == cudaSuccess) e = vrad::dev_alloc(&A.flags, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemsetAsync(A.flags, 0, sizeof(uint32_t), ctx->stream);
    if (e == cudaSuccess) e = vrad::wait_stream(ctx->stream);  // p2n dies at return
    if (e != cudaSuccess) {
        A.release();
        return vrad_cuda_fail(ctx, e, "ambient upload");
    }
    A.view = vrad::AmbientView{A.light, L->lighting_bytes, A.faces, L->nfaces, A.directions, A.by_octant, A.facing, {},
                               {}, A.power2n, L->tan_theta, L->has_sky_ambient ? 1 : 0,
                               {L->sky_ambient[0], L->sky_ambient[1], L->sky_ambient[2]}};
    for (int j = 0; j < vrad::kAmbientSides; j++) {
        A.view.nfacing[j] = nfacing[j];
        A.view.inv[j] = inv[j];
    }
    A.ready = true;
    return VRAD_OK;
}

extern "C" int32_t vrad_ambient_cubes_device(vrad_ctx *ctx, const float *d_positions, int64_t n, float *d_cubes,
                                             void *stream) {
    if (!ctx) return vrad_fail(nullptr, VRAD_ERR_ARG, "null context");
    if (n < 0 || (n && (!d_positions || !d_cubes))) return vrad_fail(ctx, VRAD_ERR_ARG, "invalid positions or cubes");
    if (n == 0) return VRAD_OK;
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "cudaSetDevice");
    const int32_t rc = vrad::cubes_on(ctx, d_positions, n, d_cubes, (cudaStream_t)stream);
    e = vrad::join_stream(ctx, (cudaStream_t)stream);
    return rc != VRAD_OK || e == cudaSuccess ? rc : vrad_cuda_fail(ctx, e, "joining the caller's stream");
}

extern "C" int32_t vrad_ambient_status(vrad_ctx *ctx) {
    if (!ctx) return vrad_fail(nullptr, VRAD_ERR_ARG, "null context");
    std::lock_guard<std::mutex> g(ctx->mu);
    if (!ctx->ambient.ready) return vrad_fail(ctx, VRAD_ERR_NO_SCENE, "no ambient lighting uploaded");
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return vrad_cuda_fail(ctx, e, "cudaSetDevice");
    return vrad::read_flags(ctx);
}

extern "C" int32_t vrad_ambient_cubes(vrad_ctx *ctx, const float *positions, int64_t n, float *cubes) {
    if (!ctx) return vrad_fail(nullptr, VRAD_ERR_ARG, "null context");
    if (n < 0 || (n && (!positions || !cubes))) return vrad_fail(ctx, VRAD_ERR_ARG, "invalid positions or cubes");
    if (n == 0) return VRAD_OK;
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaError_t e = cudaSetDevice(ctx->device);
    float *d_pos = nullptr, *d_cubes = nullptr;
    if (e == cudaSuccess) e = vrad::dev_alloc(&d_pos, sizeof(float) * 3 * (size_t)n);
    if (e == cudaSuccess) e = vrad::dev_alloc(&d_cubes, sizeof(float) * 3 * vrad::kAmbientSides * (size_t)n);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_pos, positions, sizeof(float) * 3 * (size_t)n, cudaMemcpyHostToDevice, ctx->stream);
    int32_t rc = e == cudaSuccess ? vrad::cubes_on(ctx, d_pos, n, d_cubes, ctx->stream)
                                  : vrad_cuda_fail(ctx, e, "ambient set-up");
    if (rc == VRAD_OK) {
        e = cudaMemcpyAsync(cubes, d_cubes, sizeof(float) * 3 * vrad::kAmbientSides * (size_t)n,
                            cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = vrad::wait_stream(ctx->stream);
        rc = e == cudaSuccess ? vrad::read_flags(ctx) : vrad_cuda_fail(ctx, e, "ambient cubes");
    }
    vrad::dev_free(d_pos);
    vrad::dev_free(d_cubes);
    return rc;
}
