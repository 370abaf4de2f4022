// mlp.cu -- the learned warm start's training on the tensor cores: the
// gradient (forward, backward and weight gradients in one kernel) and Adam.
//
// Every matrix product is mma.sync.m16n8k16 with BF16 operands and FP32
// accumulators.  The forward keeps a warp's 16 rows in registers through
// all three layers: the accumulator fragments of one layer are, packed to
// BF16, the A fragments of the next (the m16n8 C layout of two adjacent
// n-tiles is the m16k16 A layout); the backward does the same for the
// activation gradients.  The weight gradients are P^T Q over a tile's rows,
// both operands read transposed from the row-major tiles in shared memory
// (ldmatrix.trans), and the tiles' products and the bias gradients are FP32
// sums.  Master weights and Adam's moments are FP32; the BF16
// operand copies are refreshed after every step.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <vector>

#include "context.cuh"
#include "mlp.cuh"

namespace vrad {

namespace {

constexpr int kMlpWarps = 8;
constexpr int kMlpThreads = 32 * kMlpWarps;
constexpr int kTileRows = 16 * kMlpWarps;  // rows per CTA iteration

__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t ld32(const uint16_t *p) { return *reinterpret_cast<const uint32_t *>(p); }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Four 8 x 8 matrices of b16; lanes 8 i .. 8 i + 7 give matrix i's rows.
__device__ __forceinline__ void ldsm4(uint32_t r[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t r[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ldsm2_t(uint32_t r[2], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(addr)
                 : "memory");
}

// Row strides in shared memory (b16): eight more than the row, so that the
// eight rows of an ldmatrix fall into different banks.
constexpr int kSx = kMlpIn + 8, kSh = kMlpHidden + 8;

struct __align__(16) GradSmem {
    uint16_t w1t[kMlpHidden * kSx];   // [128][32], output-major
    uint16_t w2t[kMlpHidden * kSh];   // [128][128], output-major
    uint16_t w3t[kMlpOutPad * kSh];   // [8][128], output-major
    uint16_t w2[kMlpHidden * kSh];    // [128][128], input-major
    uint16_t w3[kMlpHidden * kMlpOutPad];  // [128][8], input-major
    uint16_t x[kTileRows * kSx];      // the tile's inputs
    uint16_t h1[kTileRows * kSh];     // first hidden layer
    uint16_t h2[kTileRows * kSh];     // second hidden layer, then dz1
    uint16_t dz[kTileRows * kSh];     // dz2
    uint16_t dy[kTileRows * kMlpOutPad];
    float b1[kMlpHidden], b2[kMlpHidden], b3[kMlpOutPad];
    float b3part[kMlpWarps][kMlpOutPad];
};
static_assert(kMlpThreads == 2 * kMlpHidden, "a thread per hidden bias");
static_assert(sizeof(GradSmem) <= 227 * 1024, "one CTA's shared memory");

// acc[16 n-tiles] += A (16 x 16 KT) B, B from wt[n][k] with row stride S.
template <int KT, int S>
__device__ __forceinline__ void product(float acc[16][4], const uint32_t a[][4], const uint16_t *wt, int lane) {
    const uint32_t at = smem_u32(wt + (lane & 7) * S + 8 * (lane >> 3));
    // The sixteen accumulators' chains side by side.
#pragma unroll
    for (int kp = 0; kp < KT / 2; kp++)
#pragma unroll
        for (int j = 0; j < 16; j++) {
            uint32_t b[4];  // the n-tile's B fragments of two k-tiles
            ldsm4(b, at + 2 * (8 * j * S + 32 * kp));
            mma16816(acc[j], a[2 * kp], b);
            mma16816(acc[j], a[2 * kp + 1], b + 2);
        }
}

__device__ __forceinline__ void set_bias(float acc[16][4], const float *bias, int t) {
#pragma unroll
    for (int j = 0; j < 16; j++) {
        acc[j][0] = acc[j][2] = bias[8 * j + 2 * t];
        acc[j][1] = acc[j][3] = bias[8 * j + 2 * t + 1];
    }
}

// The accumulators as the next product's A fragments.
__device__ __forceinline__ void pack(const float acc[16][4], uint32_t a[8][4]) {
#pragma unroll
    for (int kt = 0; kt < 8; kt++) {
        a[kt][0] = pack2(acc[2 * kt][0], acc[2 * kt][1]);
        a[kt][1] = pack2(acc[2 * kt][2], acc[2 * kt][3]);
        a[kt][2] = pack2(acc[2 * kt + 1][0], acc[2 * kt + 1][1]);
        a[kt][3] = pack2(acc[2 * kt + 1][2], acc[2 * kt + 1][3]);
    }
}

// ReLU, then pack; m = which of the 64 packed activations are above zero.
__device__ __forceinline__ void relu_pack(float acc[16][4], uint32_t a[8][4], uint32_t m[2]) {
#pragma unroll
    for (int j = 0; j < 16; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[j][q] = acc[j][q] > 0.0f ? acc[j][q] : 0.0f;
    pack(acc, a);
    m[0] = m[1] = 0;
#pragma unroll
    for (int kt = 0; kt < 8; kt++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int bit = 8 * (kt & 3) + 2 * q;
            if (bf_lo(a[kt][q]) > 0.0f) m[kt >> 2] |= 1u << bit;
            if (bf_hi(a[kt][q]) > 0.0f) m[kt >> 2] |= 2u << bit;
        }
}

// Zero where the activation was not above zero, then pack.
__device__ __forceinline__ void mask_pack(float acc[16][4], const uint32_t m[2], uint32_t a[8][4]) {
#pragma unroll
    for (int kt = 0; kt < 8; kt++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int bit = 8 * (kt & 3) + 2 * q, j = 2 * kt + (q >> 1), e = 2 * (q & 1);
            if (!((m[kt >> 2] >> bit) & 1u)) acc[j][e] = 0.0f;
            if (!((m[kt >> 2] >> bit) & 2u)) acc[j][e + 1] = 0.0f;
        }
    pack(acc, a);
}

// A warp's 16 x 128 tile from its A fragments into shared memory rows.
__device__ __forceinline__ void store_tile(uint16_t *rows, const uint32_t a[8][4], int g, int t) {
    uint16_t *p = rows + g * kSh + 2 * t;
#pragma unroll
    for (int kt = 0; kt < 8; kt++) {
        *reinterpret_cast<uint32_t *>(p + 16 * kt) = a[kt][0];
        *reinterpret_cast<uint32_t *>(p + 8 * kSh + 16 * kt) = a[kt][1];
        *reinterpret_cast<uint32_t *>(p + 16 * kt + 8) = a[kt][2];
        *reinterpret_cast<uint32_t *>(p + 8 * kSh + 16 * kt + 8) = a[kt][3];
    }
}

__device__ __forceinline__ void add4(float to[4], const float from[4]) {
#pragma unroll
    for (int q = 0; q < 4; q++) to[q] += from[q];
}

// Adds a tile's column sums to c: the thread's two columns, 2 (tid & 63) and
// the next, over its quarter of the rows.
__device__ __forceinline__ void add_columns(float c[2], const uint16_t *rows, int tid) {
    constexpr int kRows = kTileRows / (kMlpThreads / 64);
    const uint16_t *p = rows + (tid >> 6) * kRows * kSh + 2 * (tid & 63);
    float lo = 0.0f, hi = 0.0f;
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const uint32_t v = ld32(p + r * kSh);
        lo += bf_lo(v);
        hi += bf_hi(v);
    }
    c[0] += lo;
    c[1] += hi;
}

// Adds a weight gradient's m16n8 tile at row m0, column n0 of grad.
__device__ __forceinline__ void add_tile(float *grad, int stride, int ncols, int m0, int n0, const float c[4], int g,
                                         int t) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int col = n0 + 2 * t + (q & 1);
        if (col < ncols) atomicAdd(&grad[(m0 + g + 8 * (q >> 1)) * stride + col], c[q]);
    }
}

// The mean squared error's gradient over n rows: m.grad += it, m.loss += the
// loss.  A CTA of 8 warps takes tiles of 128 rows, 16 rows a warp for the
// layers:
//   forward, h1 and h2 into shared memory; dy = 2 (y - target) / 3n;
//   dz2 = (dy W3^T) * [h2 > 0], dz1 = (dz2 W2^T) * [h1 > 0];
// then the products over the tile's rows, split by output rows among the
// warps: dW3 = h2^T dy, dW2 = h1^T dz2, dW1 = x^T dz1; and the bias gradients,
// the columns' sums.  What is summed over tiles is summed by FP32 adds, in
// registers: the tensor cores' accumulators cut off what the sum's last place
// does not hold, and over the tiles of a CTA that adds up (a million rows,
// against 64 bits: dW3 off by 2.4e-5 accumulated there, by 2.9e-7 so; 65,536
// rows 6.9e-7 and 3.9e-7).
// A minibatch is a few hundred tiles, so what counts is one tile's time and
// what it sends to memory: nothing but x and the targets in, and one atomic
// add per parameter and CTA out.  A tile takes 8.2 us, near the rate of
// mma.sync on this chip (sixteen warps, two to a row group, take as long), and
// what is around the tiles, the weights in and the gradients out, 16 us for
// one CTA and 24 for 148: 128 rows 24 us, 18,944 (a tile a CTA) 32, 32,768 35,
// 151,552 (eight) 90.  As five kernels with the activations and their
// gradients in HBM, shared memory operands read with up to eight-way bank
// conflicts and transposed by 2-byte stores, 32,768 rows took 145 us.
__global__ void __launch_bounds__(kMlpThreads, 1) k_mlp_gradient(vrad_mlp m, const uint16_t *__restrict__ x,
                                                                 const float *__restrict__ target, int64_t n, float inv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GradSmem &s = *reinterpret_cast<GradSmem *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // The weights, eight at a time.
    auto copy = [&](uint16_t *dst, const uint16_t *src, int rows, int cols, int stride) {
        for (int i = tid; i < rows * cols / 8; i += kMlpThreads) {
            const int r = i / (cols / 8), c = 8 * (i % (cols / 8));
            *reinterpret_cast<uint4 *>(dst + r * stride + c) = *reinterpret_cast<const uint4 *>(src + r * cols + c);
        }
    };
    copy(s.w1t, m.w1t, kMlpHidden, kMlpIn, kSx);
    copy(s.w2t, m.w2t, kMlpHidden, kMlpHidden, kSh);
    copy(s.w3t, m.w3t, kMlpOutPad, kMlpHidden, kSh);
    copy(s.w2, m.w2, kMlpHidden, kMlpHidden, kSh);
    copy(s.w3, m.w3, kMlpHidden, kMlpOutPad, kMlpOutPad);
    for (int i = tid; i < kMlpHidden; i += kMlpThreads) {
        s.b1[i] = m.master[kOffB1 + i];
        s.b2[i] = m.master[kOffB2 + i];
    }
    if (tid < kMlpOutPad) s.b3[tid] = tid < kMlpOut ? m.master[kOffB3 + tid] : 0.0f;
    __syncthreads();

    float g2[16][4] = {}, g1[4][4] = {}, g3[4] = {}, gb2[2] = {}, gb1[2] = {}, gb3[2] = {};
    float loss = 0.0f;
    uint16_t *xs = s.x + 16 * warp * kSx, *h1 = s.h1 + 16 * warp * kSh, *h2 = s.h2 + 16 * warp * kSh,
             *dz = s.dz + 16 * warp * kSh, *dy = s.dy + 16 * warp * kMlpOutPad;
    for (int64_t tile = blockIdx.x; tile * kTileRows < n; tile += gridDim.x) {
        const int64_t ra = tile * kTileRows + 16 * warp + g, rb = ra + 8;
        float acc[16][4];
        uint32_t a[8][4], m1[2], m2[2];
#pragma unroll
        for (int kt = 0; kt < 2; kt++) {
            a[kt][0] = ra < n ? ld32(x + ra * kMlpIn + 16 * kt + 2 * t) : 0u;
            a[kt][1] = rb < n ? ld32(x + rb * kMlpIn + 16 * kt + 2 * t) : 0u;
            a[kt][2] = ra < n ? ld32(x + ra * kMlpIn + 16 * kt + 8 + 2 * t) : 0u;
            a[kt][3] = rb < n ? ld32(x + rb * kMlpIn + 16 * kt + 8 + 2 * t) : 0u;
        }
        // This row pair's targets, loaded ahead of the layers.
        float want[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = 2 * t + (q & 1);
            const int64_t r = q < 2 ? ra : rb;
            want[q] = c < kMlpOut && r < n ? __ldg(&target[r * kMlpOut + c]) : 0.0f;
        }
#pragma unroll
        for (int kt = 0; kt < 2; kt++) {
            *reinterpret_cast<uint32_t *>(xs + g * kSx + 16 * kt + 2 * t) = a[kt][0];
            *reinterpret_cast<uint32_t *>(xs + (g + 8) * kSx + 16 * kt + 2 * t) = a[kt][1];
            *reinterpret_cast<uint32_t *>(xs + g * kSx + 16 * kt + 8 + 2 * t) = a[kt][2];
            *reinterpret_cast<uint32_t *>(xs + (g + 8) * kSx + 16 * kt + 8 + 2 * t) = a[kt][3];
        }
        set_bias(acc, s.b1, t);
        product<2, kSx>(acc, a, s.w1t, lane);
        relu_pack(acc, a, m1);
        store_tile(h1, a, g, t);
        set_bias(acc, s.b2, t);
        product<8, kSh>(acc, a, s.w2t, lane);
        relu_pack(acc, a, m2);
        store_tile(h2, a, g, t);
        float out[4] = {s.b3[2 * t], s.b3[2 * t + 1], s.b3[2 * t], s.b3[2 * t + 1]};
#pragma unroll
        for (int kp = 0; kp < 4; kp++) {
            uint32_t b[4];
            ldsm4(b, smem_u32(s.w3t + (lane & 7) * kSh + 8 * (lane >> 3) + 32 * kp));
            mma16816(out, a[2 * kp], b);
            mma16816(out, a[2 * kp + 1], b + 2);
        }
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (2 * t + (q & 1) < kMlpOut && (q < 2 ? ra : rb) < n) {
                const float e = out[q] - want[q];
                loss += e * e;
                d[q] = 2.0f * e * inv;
            }
        const uint32_t ady[4] = {pack2(d[0], d[1]), pack2(d[2], d[3]), 0u, 0u};
        *reinterpret_cast<uint32_t *>(dy + g * kMlpOutPad + 2 * t) = ady[0];
        *reinterpret_cast<uint32_t *>(dy + (g + 8) * kMlpOutPad + 2 * t) = ady[1];
        gb3[0] += bf_lo(ady[0]) + bf_lo(ady[1]);
        gb3[1] += bf_hi(ady[0]) + bf_hi(ady[1]);
        // dh2 = dy (16 x 8, k padded to 16 with zeros) W3^T.
#pragma unroll
        for (int j = 0; j < 16; j++) {
            acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
            const uint32_t b[2] = {ld32(s.w3 + (8 * j + g) * kMlpOutPad + 2 * t), 0u};
            mma16816(acc[j], ady, b);
        }
        mask_pack(acc, m2, a);
        store_tile(dz, a, g, t);
        // dh1 = dz2 W2^T.
#pragma unroll
        for (int j = 0; j < 16; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
        product<8, kSh>(acc, a, s.w2, lane);
        mask_pack(acc, m1, a);
        __syncthreads();  // every warp's x, h1, h2, dy, dz2
        // dW3 and dW2: this warp's 16 input rows.  A (m16 k16) of P^T from
        // P's rows k: matrices (m, k) = (0, 0), (8, 0), (0, 8), (8, 8).
        const int ka = (lane & 7) + 8 * (lane >> 4), ma = 16 * warp + 8 * ((lane >> 3) & 1);
        // B (k16 n8) of two n-tiles: (k, n) = (0, 0), (8, 0), (0, 8), (8, 8).
        const int kb = (lane & 7) + 8 * ((lane >> 3) & 1), nb = 8 * (lane >> 4);
#pragma unroll
        for (int j = 0; j < 16; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
        float one[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int kt = 0; kt < 8; kt++) {
            uint32_t p[4], q[4];
            ldsm4_t(p, smem_u32(s.h2 + (16 * kt + ka) * kSh + ma));
            ldsm2_t(q, smem_u32(s.dy + (16 * kt + (lane & 15)) * kMlpOutPad));
            mma16816(one, p, q);
            ldsm4_t(p, smem_u32(s.h1 + (16 * kt + ka) * kSh + ma));
#pragma unroll
            for (int j = 0; j < 8; j++) {
                ldsm4_t(q, smem_u32(s.dz + (16 * kt + kb) * kSh + 16 * j + nb));
                mma16816(acc[2 * j], p, q);
                mma16816(acc[2 * j + 1], p, q + 2);
            }
        }
#pragma unroll
        for (int j = 0; j < 16; j++) add4(g2[j], acc[j]);
        add4(g3, one);
        add_columns(gb2, s.dz, tid);
        __syncthreads();  // h2 is read
        store_tile(h2, a, g, t);  // dz1
        __syncthreads();
        // dW1: input rows 16 (warp & 1) .., columns 32 (warp >> 1) ...
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
        for (int kt = 0; kt < 8; kt++) {
            uint32_t p[4], q[4];
            ldsm4_t(p, smem_u32(s.x + (16 * kt + ka) * kSx + 16 * (warp & 1) + 8 * ((lane >> 3) & 1)));
#pragma unroll
            for (int j = 0; j < 2; j++) {
                ldsm4_t(q, smem_u32(s.h2 + (16 * kt + kb) * kSh + 32 * (warp >> 1) + 16 * j + nb));
                mma16816(acc[2 * j], p, q);
                mma16816(acc[2 * j + 1], p, q + 2);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) add4(g1[j], acc[j]);
        add_columns(gb1, s.h2, tid);
        __syncthreads();  // x and dz1 are read
    }
    // The CTA's sums.
#pragma unroll
    for (int j = 0; j < 16; j++) add_tile(m.grad + kOffW2, kMlpHidden, kMlpHidden, 16 * warp, 8 * j, g2[j], g, t);
#pragma unroll
    for (int j = 0; j < 4; j++)
        add_tile(m.grad, kMlpHidden, kMlpHidden, 16 * (warp & 1), 32 * (warp >> 1) + 8 * j, g1[j], g, t);
    add_tile(m.grad + kOffW3, kMlpOut, kMlpOut, 16 * warp, 0, g3, g, t);
    // The bias gradients' parts first within the CTA: row quarters, warps.
    float(*part)[2 * kMlpHidden + 2] = reinterpret_cast<float(*)[2 * kMlpHidden + 2]>(s.dz);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int col = 2 * (tid & 63) + q;
        part[tid >> 6][col] = gb1[q];
        part[tid >> 6][kMlpHidden + col] = gb2[q];
        for (int o = 16; o > 2; o >>= 1) gb3[q] += __shfl_xor_sync(0xffffffffu, gb3[q], o);  // the rows g
        if (g == 0) s.b3part[warp][2 * t + q] = gb3[q];
    }
    __syncthreads();
    const float b = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
    atomicAdd(&m.grad[tid < kMlpHidden ? kOffB1 + tid : kOffB2 + tid - kMlpHidden], b);
    if (tid < kMlpOut) {
        float b3 = 0.0f;
        for (int w = 0; w < kMlpWarps; w++) b3 += s.b3part[w][tid];
        atomicAdd(&m.grad[kOffB3 + tid], b3);
    }
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) atomicAdd(m.loss, loss * inv);
}

// The BF16 operand copies of the master weights.
__global__ void k_mlp_refresh(vrad_mlp m) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kW1) {
        const int k = i / kMlpHidden, c = i % kMlpHidden;
        m.w1t[c * kMlpIn + k] = __bfloat16_as_ushort(__float2bfloat16_rn(m.master[i]));
    }
    if (i < kW2) {
        const int k = i / kMlpHidden, c = i % kMlpHidden;
        const uint16_t v = __bfloat16_as_ushort(__float2bfloat16_rn(m.master[kOffW2 + i]));
        m.w2t[c * kMlpHidden + k] = v;
        m.w2[k * kMlpHidden + c] = v;
    }
    if (i < kMlpHidden * kMlpOutPad) {
        const int k = i / kMlpOutPad, c = i % kMlpOutPad;
        const uint16_t v = c < kMlpOut ? __bfloat16_as_ushort(__float2bfloat16_rn(m.master[kOffW3 + k * kMlpOut + c]))
                                       : (uint16_t)0;
        m.w3t[c * kMlpHidden + k] = v;
        m.w3[k * kMlpOutPad + c] = v;
    }
}

// Adam (beta1 0.9, beta2 0.999, epsilon 1e-8) on the master weights.
__global__ void k_mlp_adam(vrad_mlp m, float lr, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kMlpParams) return;
    const float gr = m.grad[i];
    const float mm = 0.9f * m.adam_m[i] + 0.1f * gr;
    const float vv = 0.999f * m.adam_v[i] + 0.001f * gr * gr;
    m.adam_m[i] = mm;
    m.adam_v[i] = vv;
    m.master[i] -= lr * (mm / c1) / (sqrtf(vv / c2) + 1e-8f);
}

// The MSE gradient into m.grad (and the loss into m.loss, which lies just
// behind it), on `s`.
cudaError_t gradient(vrad_mlp &m, const uint16_t *x, const float *target, int64_t n, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(m.grad, 0, sizeof(float) * (kMlpParams + 1), s);
    if (e != cudaSuccess || n == 0) return e;
    const int64_t tiles = (n + kTileRows - 1) / kTileRows;
    k_mlp_gradient<<<(unsigned)(tiles < m.sms ? tiles : m.sms), kMlpThreads, sizeof(GradSmem), s>>>(
        m, x, target, n, 1.0f / (3.0f * (float)n));
    return cudaGetLastError();
}

bool smem_ready[64];
std::mutex smem_mu;

cudaError_t allow_smem(int device) {
    std::lock_guard<std::mutex> g(smem_mu);
    if (device >= 0 && device < 64 && smem_ready[device]) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(k_mlp_gradient, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem));
    if (e == cudaSuccess && device >= 0 && device < 64) smem_ready[device] = true;
    return e;
}

}  // namespace

cudaError_t mlp_forward(const vrad_mlp &m, const uint16_t *x, int64_t n, float *y, cudaStream_t s) {
    return mlp_forward_tc(m, x, n, y, s);
}

}  // namespace vrad

namespace {

// The pinned blocks that carry a gradient to the host.  A call of
// vrad_mlp_gradient_device takes one and gives it back: pinning one takes 1
// to 2.5 ms where the driver maps new memory for it, several times what
// creating a network takes, and a network that is only run forward or trained
// needs none.  At most kSpareBlocks (85 KB each) are kept.
constexpr int kSpareBlocks = 8;
std::mutex spare_mu;
float *spare_blocks[kSpareBlocks];
int nspare = 0;

cudaError_t take_block(float **out) {
    {
        std::lock_guard<std::mutex> g(spare_mu);
        if (nspare > 0) {
            *out = spare_blocks[--nspare];
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(out, sizeof(float) * (vrad::kMlpParams + 1), cudaHostAllocPortable);
}

void give_block(float *p) {
    if (!p) return;
    {
        std::lock_guard<std::mutex> g(spare_mu);
        if (nspare < kSpareBlocks) {
            spare_blocks[nspare++] = p;
            return;
        }
    }
    cudaFreeHost(p);
}

void release_mlp(vrad_mlp *m) {
    for (void *p : {(void *)m->master, (void *)m->adam_m, (void *)m->adam_v, (void *)m->grad, (void *)m->w1t,
                    (void *)m->w2t, (void *)m->w3t, (void *)m->w2, (void *)m->w3, (void *)m->flags})
        cudaFree(p);
    delete m;
}

cudaError_t refresh(vrad_mlp *m, cudaStream_t s) {
    vrad::k_mlp_refresh<<<(vrad::kW2 + 255) / 256, 256, 0, s>>>(*m);
    return cudaGetLastError();
}

}  // namespace

extern "C" int32_t vrad_mlp_create(vrad_ctx *ctx, uint64_t seed, vrad_mlp **out) {
    using namespace vrad;
    if (!ctx || !out) return vrad_fail(ctx, VRAD_ERR_ARG, "null argument");
    *out = nullptr;
    cudaError_t e = cudaSetDevice(ctx->device);
    vrad_mlp *m = new vrad_mlp();
    m->device = ctx->device;
    for (float **p : {&m->master, &m->adam_m, &m->adam_v, &m->grad})
        if (e == cudaSuccess) e = cudaMalloc(p, sizeof(float) * (kMlpParams + 1));
    for (uint16_t **p : {&m->w1t, &m->w2t, &m->w3t, &m->w2, &m->w3})
        if (e == cudaSuccess) e = cudaMalloc(p, sizeof(uint16_t) * kW2);
    m->loss = m->grad ? m->grad + kMlpParams : nullptr;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (e == cudaSuccess) e = cudaMalloc(&m->flags, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(m->flags, 0, sizeof(uint32_t));
    if (e == cudaSuccess) e = allow_smem(ctx->device);
    // He initialisation from a seeded generator; biases zero.
    std::vector<float> w((size_t)kMlpParams, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fan_in, int count) {
        std::normal_distribution<double> nd(0.0, std::sqrt(2.0 / fan_in));
        for (int i = 0; i < count; i++) w[(size_t)(off + i)] = (float)nd(rng);
    };
    fill(0, kMlpIn, kW1);
    fill(kOffW2, kMlpHidden, kW2);
    fill(kOffW3, kMlpHidden, kW3);
    if (e == cudaSuccess) e = cudaMemcpy(m->master, w.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->adam_m, 0, sizeof(float) * kMlpParams);
    if (e == cudaSuccess) e = cudaMemset(m->adam_v, 0, sizeof(float) * kMlpParams);
    if (e == cudaSuccess) e = cudaMemset(m->w3t, 0, sizeof(uint16_t) * kW2);
    if (e == cudaSuccess) e = refresh(m, nullptr);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        release_mlp(m);
        return vrad_cuda_fail(ctx, e, "network creation");
    }
    *out = m;
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_destroy(vrad_mlp *m) {
    if (!m) return VRAD_OK;
    cudaSetDevice(m->device);
    cudaDeviceSynchronize();
    release_mlp(m);
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_params(vrad_mlp *m, float *get, const float *set) {
    if (!m) return vrad_fail(nullptr, VRAD_ERR_ARG, "null network");
    cudaError_t e = cudaSetDevice(m->device);
    if (e == cudaSuccess && set) e = cudaMemcpy(m->master, set, sizeof(float) * vrad::kMlpParams, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && set) e = refresh(m, nullptr);
    if (e == cudaSuccess && get) e = cudaMemcpy(get, m->master, sizeof(float) * vrad::kMlpParams, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "network parameters");
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_forward_device(vrad_mlp *m, const uint16_t *x, int64_t n, float *y, void *stream) {
    if (!m || n < 0 || (n && (!x || !y))) return vrad_fail(nullptr, VRAD_ERR_ARG, "invalid network forward");
    if (((uintptr_t)x & 3) || ((uintptr_t)y & 3)) return vrad_fail(nullptr, VRAD_ERR_ARG, "x and y must be 4-byte aligned");
    cudaError_t e = cudaSetDevice(m->device);
    if (e == cudaSuccess) e = vrad::mlp_forward(*m, x, n, y, (cudaStream_t)stream);
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "network forward");
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_gradient_device(vrad_mlp *m, const uint16_t *x, const float *target, int64_t n,
                                            float *grad, float *loss, void *stream) {
    if (!m || n < 0 || (n && (!x || !target))) return vrad_fail(nullptr, VRAD_ERR_ARG, "invalid network gradient");
    cudaError_t e = cudaSetDevice(m->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (e == cudaSuccess) e = vrad::gradient(*m, x, target, n, s);
    // Gradient and loss in one copy, through pinned memory.
    float *host = nullptr;
    if (e == cudaSuccess) e = take_block(&host);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(host, m->grad, sizeof(float) * (vrad::kMlpParams + 1), cudaMemcpyDeviceToHost, s);
    // No copy may be in flight into a block that goes back.
    const cudaError_t done = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = done;
    if (e == cudaSuccess && grad) std::memcpy(grad, host, sizeof(float) * vrad::kMlpParams);
    if (e == cudaSuccess && loss) *loss = host[vrad::kMlpParams];
    give_block(host);
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "network gradient");
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_train_step_device(vrad_mlp *m, const uint16_t *x, const float *target, int64_t n, float lr,
                                              void *stream) {
    if (!m || n <= 0 || !x || !target || !(lr > 0.0f)) return vrad_fail(nullptr, VRAD_ERR_ARG, "invalid training step");
    cudaError_t e = cudaSetDevice(m->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (e == cudaSuccess) e = vrad::gradient(*m, x, target, n, s);
    if (e == cudaSuccess) {
        m->step++;
        const float c1 = 1.0f - (float)std::pow(0.9, (double)m->step), c2 = 1.0f - (float)std::pow(0.999, (double)m->step);
        vrad::k_mlp_adam<<<(vrad::kMlpParams + 255) / 256, 256, 0, s>>>(*m, lr, c1, c2);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = refresh(m, s);
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "training step");
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_loss(vrad_mlp *m, float *loss) {
    if (!m || !loss) return vrad_fail(nullptr, VRAD_ERR_ARG, "null argument");
    cudaError_t e = cudaSetDevice(m->device);
    if (e == cudaSuccess) e = cudaMemcpy(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "network loss");
    return VRAD_OK;
}

extern "C" int32_t vrad_mlp_status(vrad_mlp *m) {
    if (!m) return vrad_fail(nullptr, VRAD_ERR_ARG, "null network");
    uint32_t f = 0;
    cudaError_t e = cudaSetDevice(m->device);
    if (e == cudaSuccess) e = cudaMemcpy(&f, m->flags, sizeof f, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && f) e = cudaMemset(m->flags, 0, sizeof f);
    if (e != cudaSuccess) return vrad_cuda_fail(nullptr, e, "network status");
    if (f) return vrad_fail(nullptr, VRAD_ERR_TIMEOUT, "a network forward's tensor-core wait ran out");
    return VRAD_OK;
}
