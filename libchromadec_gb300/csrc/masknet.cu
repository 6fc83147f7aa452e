// masknet.cu -- the learned chroma mask of the Transform-PAL 3D learned form:
// a small 3D convolutional network over one tile's spectrum that predicts,
// for each bin the filter can keep, the fraction of it that is chroma, in
// place of the fixed mirror threshold of TransformPal3D::applyFilter
// (src/decoders/palcolour/transform_pal_3d.cpp:249-333). The reference has no
// learned PAL path; its NTSC nnTransform3D decoder is the precedent for a
// per-bin mask on a 3D tile spectrum (src/decoders/nntransform3d/
// nntransform3d_pipeline_cuda.cu:160-244, 544-567).
//
// Domain of one tile: the 1,280 bins kz 0..7, ky 0..31 (periodic axes of the
// DFT) and q = kx - 2 in 0..4 (zero outside), voxel v = (q * 8 + kz) * 32 + ky.
// Network: input channels f(b) = ln(1 + |X_b|) / 16 and f at b's mirror about
// the carrier, ((10 - kz) mod 8, (40 - ky) mod 32, 4 - q); three 3x3x3
// convolutions of 16 channels with bias and ReLU; a 1x1x1 sigmoid head giving
// p(b). BF16 weights, features and activations, FP32 accumulation. A tile
// whose mean |p - 1/2| is below the confidence limit falls back to the
// threshold decisions.
//
// Kernels:
//  * mn_tc_forward_kernel<TRAIN> (the default forward pass): each
//    convolution as implicit GEMMs on the tensor cores (tcgen05, BF16
//    operands, FP32 accumulators in tensor memory), warp-specialised and
//    persistent over tiles; described where it is defined.
//  * mn_tc_half_kernel: the same on features that repeat along (kz + 4, ky +
//    16), as those the walk computes do: what the engine's decode runs.
// The CUDA-core kernels (one CTA of 256 threads per tile, persistent over
// tiles; thread t owns the (kz, ky) column t and computes its 5 q x 16
// channels):
//  * mn_forward_kernel<TRAIN>: features -> p (+ fallback flags), the
//    cross-check of the tensor-core pass; the training variant also keeps
//    each layer's activations for the backward pass.
// Training:
//  * mn_backward_kernel: dL/dz of the head for L = sum |p X - C|^2 / sum |X|^2,
//    the head, then per layer the weight and input gradients as tensor-core
//    contractions; described where it is defined. Each CTA writes its own
//    slice of a partial-gradient buffer; mn_adam_kernel reduces the slices and
//    takes one Adam step on the FP32 master weights.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/chromadec_gb300.h"
#include "error_state.h"
#include "masknet.h"
#include "tcgen05_ptx.cuh"

namespace chdg {
namespace mn {

constexpr int kThreads = 256;
constexpr int NQ = 5, NZY = 256, NV = 1280, NC = 16, NCIN = 2;
constexpr int CS = 1282;   // channel stride of shared activations (bf16), bank-skewed
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + 27 * NCIN * NC, OFF_W2 = OFF_B1 + NC, OFF_B2 = OFF_W2 + 27 * NC * NC,
              OFF_W3 = OFF_B2 + NC, OFF_B3 = OFF_W3 + 27 * NC * NC, OFF_WH = OFF_B3 + NC, OFF_BH = OFF_WH + NC;
constexpr int NPARAM = OFF_BH + 1;
constexpr int NPARAM_PAD = (NPARAM + 3) & ~3;
static_assert(NPARAM == CHDG_MASKNET_PARAMS, "parameter count");
static_assert(OFF_W2 % 4 == 0 && OFF_W3 % 4 == 0, "float4 weight rows");

__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Accumulate a 3x3x3 convolution of CI input channels into acc[q][co] for
// the thread's column (z, y). in(ci, v) reads input channel ci at voxel v;
// wrow(t, ci) points at the 16 output-channel weights of tap t, input ci
// (stride `wstride` floats between them).
template <int CI, typename In, typename WRow>
__device__ __forceinline__ void conv_acc(const In &in, const WRow &wrow, int z, int y, float (&acc)[NQ][NC])
{
#pragma unroll 1
    for (int dz = -1; dz <= 1; dz++) {
#pragma unroll 1
        for (int dy = -1; dy <= 1; dy++) {
            const int zy = (((z + dz) & 7) << 5) | ((y + dy) & 31);
            const int tb = (dz + 1) * 9 + (dy + 1) * 3;
#pragma unroll 2
            for (int ci = 0; ci < CI; ci++) {
                float xin[NQ + 2];
                xin[0] = 0.f;
                xin[NQ + 1] = 0.f;
#pragma unroll
                for (int q = 0; q < NQ; q++) xin[q + 1] = in(ci, q * NZY + zy);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    float w[NC];
                    wrow(tb + j, ci, w);
#pragma unroll
                    for (int q = 0; q < NQ; q++) {
                        const float xv = xin[q + j];
#pragma unroll
                        for (int co = 0; co < NC; co++) acc[q][co] = __fmaf_rn(xv, w[co], acc[q][co]);
                    }
                }
            }
        }
    }
}

// Weight rows of a layer's W[27][CI][16] in shared memory (forward)
template <int CI>
struct WFwd {
    const float *W;
    __device__ __forceinline__ void operator()(int t, int ci, float (&w)[NC]) const
    {
        const float4 *p = reinterpret_cast<const float4 *>(W + (t * CI + ci) * NC);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 v = p[k];
            w[4 * k] = v.x, w[4 * k + 1] = v.y, w[4 * k + 2] = v.z, w[4 * k + 3] = v.w;
        }
    }
};

struct InBf16 {
    const __nv_bfloat16 *a;   // [16][CS]
    __device__ __forceinline__ float operator()(int c, int v) const { return __bfloat162float(a[c * CS + v]); }
};

struct InF32 {
    const float *a;   // [CI][NV]
    __device__ __forceinline__ float operator()(int c, int v) const { return a[c * NV + v]; }
};

__device__ __forceinline__ void acc_init(float (&acc)[NQ][NC], const float *bias)
{
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int co = 0; co < NC; co++) acc[q][co] = bias ? bias[co] : 0.f;
}

// ReLU, round to bf16 and store channel co of the thread's voxels
__device__ __forceinline__ void acc_store_relu(const float (&acc)[NQ][NC], __nv_bfloat16 *out, int zy)
{
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int co = 0; co < NC; co++) out[co * CS + q * NZY + zy] = __float2bfloat16_rn(fmaxf(acc[q][co], 0.f));
}

// Inputs: the tile's features and their mirror, as two FP32 channels
__device__ __forceinline__ void load_input(const uint16_t *feat_tile, float *x0, int zy)
{
    const int z = zy >> 5, y = zy & 31;
    const int mzy = (((10 - z) & 7) << 5) | ((40 - y) & 31);
    const __nv_bfloat16 *f = reinterpret_cast<const __nv_bfloat16 *>(feat_tile);
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        x0[q * NZY + zy] = __bfloat162float(f[q * NZY + zy]);
        x0[NV + q * NZY + zy] = __bfloat162float(f[(4 - q) * NZY + mzy]);
    }
}

// Activations kept for the backward pass: [tile][channel half][voxel][8]
// bf16, the backward pass's shared layout.
__device__ __forceinline__ size_t act_at(long long tile, int c, int v)
{
    return ((size_t)tile * 2 + (c >> 3)) * (NV * 8) + (size_t)v * 8 + (c & 7);
}

__device__ __forceinline__ void copy_act_out(const __nv_bfloat16 *s, __nv_bfloat16 *g, long long tile, int zy)
{
    // [16][CS] shared -> the thread's column
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int q = 0; q < NQ; q++) g[act_at(tile, c, q * NZY + zy)] = s[c * CS + q * NZY + zy];
}

__device__ __forceinline__ float block_sum(float v, float *red)
{
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) v += __shfl_xor_sync(0xffffffffu, v, h);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) s += red[w];
    return s;
}

constexpr size_t kFwdSmem = sizeof(float) * (NPARAM_PAD + 2 * NV) + 2 * sizeof(__nv_bfloat16) * NC * CS;

// params: the network's weights as used (weights bf16-rounded, biases FP32).
// TRAIN: also write A1, A2, A3 (act_at) for the backward pass.
template <bool TRAIN>
__global__ void __launch_bounds__(kThreads, 1)
    mn_forward_kernel(const float *params, const uint16_t *feat, long long ntiles, float conf_limit, float *p_out,
                      uint8_t *fallback, __nv_bfloat16 *a1g, __nv_bfloat16 *a2g, __nv_bfloat16 *a3g)
{
    extern __shared__ float4 smem4[];
    float *wsm = reinterpret_cast<float *>(smem4);
    float *x0 = wsm + NPARAM_PAD;
    __nv_bfloat16 *act0 = reinterpret_cast<__nv_bfloat16 *>(x0 + 2 * NV);
    __nv_bfloat16 *act1 = act0 + NC * CS;
    __shared__ float red[kThreads / 32];
    for (int i = threadIdx.x; i < NPARAM; i += kThreads) wsm[i] = params[i];
    const int zy = threadIdx.x, z = zy >> 5, y = zy & 31;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        __syncthreads();   // the previous tile is done with x0 and the activations
        load_input(feat + tile * NV, x0, zy);
        __syncthreads();
        float acc[NQ][NC];
        acc_init(acc, wsm + OFF_B1);
        conv_acc<NCIN>(InF32{x0}, WFwd<NCIN>{wsm + OFF_W1}, z, y, acc);
        acc_store_relu(acc, act0, zy);
        __syncthreads();
        acc_init(acc, wsm + OFF_B2);
        conv_acc<NC>(InBf16{act0}, WFwd<NC>{wsm + OFF_W2}, z, y, acc);
        acc_store_relu(acc, act1, zy);
        __syncthreads();
        acc_init(acc, wsm + OFF_B3);
        conv_acc<NC>(InBf16{act1}, WFwd<NC>{wsm + OFF_W3}, z, y, acc);
        if (TRAIN) {
            copy_act_out(act0, a1g, tile, zy);
            copy_act_out(act1, a2g, tile, zy);
        }
        float conf = 0.f;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            float zh = wsm[OFF_BH];
#pragma unroll
            for (int co = 0; co < NC; co++) {
                const float a = bfr(fmaxf(acc[q][co], 0.f));
                if (TRAIN) a3g[act_at(tile, co, q * NZY + zy)] = __float2bfloat16_rn(a);
                zh = __fmaf_rn(a, wsm[OFF_WH + co], zh);
            }
            const float p = 1.0f / (1.0f + expf(-zh));
            p_out[tile * NV + q * NZY + zy] = p;
            conf += fabsf(p - 0.5f);
        }
        const float s = block_sum(conf, red);
        if (threadIdx.x == 0 && fallback != nullptr) fallback[tile] = (s * (1.0f / NV) < conf_limit) ? 1 : 0;
    }
}

// sum of a = |X|^2 over the batch (ac: [tile][NV] of (a, c))
__global__ void mn_sum_kernel(const float2 *ac, long long n, double *out)
{
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        s += (double)ac[i].x;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) s += __shfl_xor_sync(0xffffffffu, s, h);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// ---------------------------------------------------------------------------
// Backward pass
// ---------------------------------------------------------------------------
// One CTA of 9 warps a tile, two CTAs a SM. Activations and pre-activation
// gradients are bf16 (the gradients rounded once, as they enter the next
// contraction) in shared memory as [channel half][voxel][8], 16 bytes a row:
// ldmatrix reads any 8 voxels, so a tap's shift is only another row address,
// and the same rows serve both contractions of a layer:
//  * weight gradient g[tap][ci][co] = sum_v in[ci][v + tap] d[co][v]: M = ci,
//    N = co, K = 16 voxels along ky, both operands transposed by ldmatrix.
//    Warp w owns the (dz, dy) of that index and its three dq taps; per (kz, ky
//    half) it loads the five q rows of each operand once for 13 pairs.
//  * input gradient dA[v][ci] = sum_tap,co d[v - tap][co] W[tap][ci][co]: M = 16
//    voxels along ky, N = ci, K = co; a (kz, ky half) is one unit of work, its
//    five q accumulated together. The result is rounded to bf16, and a few
//    bright bins carry most of a gradient, so a value near a rounding boundary
//    that falls on the other side moves the gradient by up to 1e-4 of it:
//    values nearer to a boundary than several times what the order of summing
//    changes are summed again one product after another, in the order (dz, dy,
//    co, dq), so that gradients do not depend on the tensor cores' order and can be
//    held against a plain restatement (to 1e-7 of their norm where the
//    activations are exact). The margin is an estimate (from the products'
//    2-norm), not a proof.
// Both contractions are m16n8k16 mma.sync on registers. For the weight gradient
// (M and N 16 a tap, operands that shift by single rows) a tcgen05 tile would
// leave its accumulator almost empty. The input gradient could fold its taps
// into N as the forward pass does; it has not been tried, as its operand would
// need a second copy of the gradients beside the one that the weight gradient
// reads. FP32 accumulation; the weight
// gradient's tensor-core sums are five products long and then added in FP32.
//
// 256 tiles: 622 us on the CUDA cores (thread (ci, co) walking the voxels, two
// rounds of 152 CTAs) -> 133 us, of which the values summed again are about
// half; the whole step 764 -> 225 us.
constexpr int kBwdThreads = 288;
constexpr int kActBytes = 2 * NV * 16;
constexpr float kNoMargin = __builtin_nanf("");
constexpr int kNearCap = 2048;              // values to sum again that are listed; more are summed at once
constexpr size_t kBwdSmem = 2 * kActBytes + sizeof(float) * (2 * NV + 9 * 20 + 32) + sizeof(uint16_t) * kNearCap + 16;
constexpr int kWFragBytes = 27 * 32 * 16;   // a layer's weights as B fragments of the input gradient

__device__ __forceinline__ void ldsm4(uint32_t a, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t a, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t a, uint32_t &r0, uint32_t &r1)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void load_act(uint32_t dst, const __nv_bfloat16 *g)
{
    const char *src = reinterpret_cast<const char *>(g);
    for (int i = threadIdx.x; i < kActBytes / 16; i += kBwdThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// first: store, else add (the CTA's own slice)
__device__ __forceinline__ void put_grad(float *g, float v, bool first) { *g = first ? v : *g + v; }

// Weight gradient of a 16-channel layer: `in` and `d` in shared memory.
__device__ __forceinline__ void wgrad16(uint32_t in, uint32_t d, float *gw, bool first)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dz = warp / 3 - 1, dy = warp % 3 - 1;
    // lane's row and channel half of the four 8x8 matrices of an operand
    const int mi = lane >> 3;
    const int ra = (lane & 7) + (mi >> 1) * 8, ha = mi & 1;   // A: (half 0, rows 0-7), (1, 0-7), (0, 8-15), (1, 8-15)
    const int rb = (lane & 7) + (mi & 1) * 8, hb = mi >> 1;   // B: (0, 0-7), (0, 8-15), (1, 0-7), (1, 8-15)
    float acc[3][2][4] = {};
#pragma unroll 1
    for (int u = 0; u < 16; u++) {
        const int kz = u >> 1, blk = u & 1;
        const int va = (((kz + dz) & 7) << 5) | ((16 * blk + ra + dy) & 31), vb = (kz << 5) | (16 * blk + rb);
        const uint32_t pa = in + (ha * NV + va) * 16, pb = d + (hb * NV + vb) * 16;
        uint32_t A[NQ][4], B[NQ][4];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            ldsm4t(pa + q * NZY * 16, A[q]);
            ldsm4t(pb + q * NZY * 16, B[q]);
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            float c[2][4] = {};
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const int qi = q + j - 1;
                if (qi < 0 || qi >= NQ) continue;
                mma16816(c[0], A[qi][0], A[qi][1], A[qi][2], A[qi][3], B[q][0], B[q][1]);
                mma16816(c[1], A[qi][0], A[qi][1], A[qi][2], A[qi][3], B[q][2], B[q][3]);
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[j][n][i] += c[n][i];
        }
    }
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++)
                put_grad(gw + ((warp * 3 + j) * NC + g + 8 * (i >> 1)) * NC + 8 * n + 2 * tq + (i & 1), acc[j][n][i], first);
}

// One input-gradient value, voxel and channel id = 16 v + ci, as one chain of
// FP32 FMAs; W: the layer's weights.
__device__ __noinline__ float dgrad_one(const __nv_bfloat16 *d, const float *W, int id)
{
    const int v = id >> 4, ci = id & 15, q = v >> 8, z = (v >> 5) & 7, y = v & 31;
    float acc = 0.f;
#pragma unroll 1
    for (int zy = 0; zy < 9; zy++) {
        const int at = (((z + zy / 3 - 1) & 7) << 5) | ((y + zy % 3 - 1) & 31);
#pragma unroll
        for (int h = 0; h < 2; h++) {   // eight co at a time
            uint4 x[3];
            float4 w[3][2];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int qi = q + j - 1;
                x[j] = qi >= 0 && qi < NQ ? reinterpret_cast<const uint4 *>(d)[h * NV + qi * NZY + at] : make_uint4(0, 0, 0, 0);
                const float4 *row = reinterpret_cast<const float4 *>(W + ((26 - (zy * 3 + j)) * NC + ci) * NC + 8 * h);
                w[j][0] = __ldg(row);
                w[j][1] = __ldg(row + 1);
            }
#pragma unroll
            for (int c = 0; c < 8; c++)
#pragma unroll
                for (int j = 0; j < 3; j++)
                    acc = __fmaf_rn(__bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(&x[j])[c]),
                                    reinterpret_cast<const float *>(&w[j])[c], acc);
        }
    }
    return acc;
}

// Values near a rounding boundary: reach[v] = the 2-norm of the 27 x 16
// gradients the value is a sum of, wmax[ci] the layer's largest |W|, near the list and its count.
// Where either is zero it holds a NaN, so that no value counts as near: the sum
// is zero in any order. (Tiles without energy consist of such values; all of
// them summed again, one lane at a time, took 304 tiles 1.79 ms, now 0.22 ms.)
struct DgradNear {
    const float *reach, *wmax;
    uint16_t *list;
    int *count;
};

// Input gradient of a 16-channel layer from `d`, masked by the activations in
// `act` (> 0) and rounded to bf16 in their place.
__device__ __forceinline__ void dgrad16(const __nv_bfloat16 *dbuf, uint32_t d, __nv_bfloat16 *act, const uint4 *wfrag,
                                        const float *W0, const DgradNear &N)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mi = lane >> 3, r = (lane & 7) + (mi & 1) * 8, h = mi >> 1;
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll 1
    for (int u = warp; u < 16; u += 9) {
        const int kz = u >> 1, blk = u & 1;
        float acc[NQ][2][4] = {};
#pragma unroll 1
        for (int zy = 0; zy < 9; zy++) {
            const int dz = zy / 3 - 1, dy = zy % 3 - 1;
            const int v = (((kz - dz) & 7) << 5) | ((16 * blk + r - dy) & 31);
            const uint32_t pa = d + (h * NV + v) * 16;
            uint32_t A[NQ][4];
            uint4 W[3];
#pragma unroll
            for (int q = 0; q < NQ; q++) ldsm4(pa + q * NZY * 16, A[q]);
#pragma unroll
            for (int j = 0; j < 3; j++) W[j] = __ldg(wfrag + (zy * 3 + j) * 32 + lane);
#pragma unroll
            for (int j = 0; j < 3; j++)
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    const int qd = q - (j - 1);
                    if (qd < 0 || qd >= NQ) continue;
                    mma16816(acc[q][0], A[qd][0], A[qd][1], A[qd][2], A[qd][3], W[j].x, W[j].y);
                    mma16816(acc[q][1], A[qd][0], A[qd][1], A[qd][2], A[qd][3], W[j].z, W[j].w);
                }
        }
#pragma unroll
        for (int q = 0; q < NQ; q++)
#pragma unroll
            for (int i = 0; i < 2; i++) {   // rows g, g + 8
                const int v = ((q * 8 + kz) << 5) | (16 * blk + g + 8 * i);
                const float reach = N.reach[v];
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    __nv_bfloat162 *at = reinterpret_cast<__nv_bfloat162 *>(act + (n * NV + v) * 8 + 2 * tq);
                    const float2 a = __bfloat1622float2(*at);
                    float o[2] = {0.f, 0.f};
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        if (!((k ? a.y : a.x) > 0.f)) continue;
                        float x = acc[q][n][2 * i + k];
                        // distance to the midpoint of two bf16 values, in
                        // units of 2^(exponent - 23), against 2^-18 of a bound of
                        // the products' 2-norm: each of the 432 sums is rounded
                        // by at most 2^-25 of a partial sum of about that norm;
                        // errors of either sign add up to about 2^-20.6 of it, so
                        // this is several times the error of either order
                        // (all of one sign they would reach 2^-16)
                        const uint32_t bits = __float_as_uint(x);
                        const int ci = 8 * n + 2 * tq + k;
                        const float dist = (float)abs((int)(bits & 0xFFFFu) - 0x8000);
                        if (dist * __uint_as_float(bits & 0x7F800000u) <= 32.0f * N.wmax[ci] * reach) {
                            const int slot = atomicAdd(N.count, 1);
                            if (slot < kNearCap) N.list[slot] = (uint16_t)(v * 16 + ci);
                            else x = dgrad_one(dbuf, W0, v * 16 + ci);
                        }
                        o[k] = x;
                    }
                    __nv_bfloat162 w;
                    w.x = __float2bfloat16_rn(o[0]);
                    w.y = __float2bfloat16_rn(o[1]);
                    *at = w;
                }
            }
    }
}

// sum over the voxels of each channel of a gradient buffer -> red[warp][8] for
// the channel half warp / 4 (8 warps)
__device__ __forceinline__ void channel_sums(const __nv_bfloat16 *buf, float *red)
{
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t >= 256) return;
    const int h = t >> 7;
    float s[8] = {};
    for (int v = t & 127; v < NV; v += 128) {
        const uint4 raw = reinterpret_cast<const uint4 *>(buf)[h * NV + v];
        const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16 *>(&raw);
#pragma unroll
        for (int c = 0; c < 8; c++) s[c] += __bfloat162float(a[c]);
    }
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], m);
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 8; c++) red[warp * 20 + c] = s[c];
}

__global__ void __launch_bounds__(kBwdThreads, 2)
    mn_backward_kernel(const float *params, const uint8_t *wfrag, const uint16_t *feat, const __nv_bfloat16 *a1g,
                       const __nv_bfloat16 *a2g, const __nv_bfloat16 *a3g, const float *pg, const float2 *acg,
                       const double *S, long long ntiles, float *gpart, double *loss)
{
    extern __shared__ __align__(128) uint8_t bsm[];
    __nv_bfloat16 *bufA = reinterpret_cast<__nv_bfloat16 *>(bsm), *bufB = bufA + 2 * NV * 8;
    float *dzs = reinterpret_cast<float *>(bsm + 2 * kActBytes);   // [NV]
    float *reach = dzs + NV;                                       // [NV]
    float *red = reach + NV;                                       // [9][20]
    float *wmax = red + 9 * 20;                                    // [2 layers][16]
    int *near_count = reinterpret_cast<int *>(wmax + 32);
    uint16_t *near_list = reinterpret_cast<uint16_t *>(near_count + 4);
    const uint32_t sA = (uint32_t)__cvta_generic_to_shared(bufA), sB = (uint32_t)__cvta_generic_to_shared(bufB);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    float *gp = gpart + (size_t)blockIdx.x * NPARAM;
    const float inv = (float)(1.0 / *S);
    double l = 0.0;
    const uint4 *w2 = reinterpret_cast<const uint4 *>(wfrag), *w3 = w2 + kWFragBytes / 16;
    // the largest |weight| of layers 2 and 3 per input channel
    if (t < 32) wmax[t] = 0.f;
    __syncthreads();
    {
        const int pair = t / 9, layer = pair >> 4, ci = pair & 15;
        const float *W = params + (layer == 0 ? OFF_W2 : OFF_W3);
        float m = 0.f;
        for (int k = 0; k < 48; k++) {
            const int e = (t % 9) * 48 + k;   // (tap, co)
            m = fmaxf(m, fabsf(W[((e >> 4) * NC + ci) * NC + (e & 15)]));
        }
        atomicMax(reinterpret_cast<int *>(wmax + pair), __float_as_int(m));
    }
    __syncthreads();
    if (t < 32 && wmax[t] == 0.f) wmax[t] = kNoMargin;
    // Input gradient of layer L (1: layer 2, 2: layer 3) from d into act, and
    // its channel sums, the previous layer's bias gradient, into gp + off.
    auto input_gradient = [&](int L, const __nv_bfloat16 *dbuf, uint32_t d, __nv_bfloat16 *act, int off, bool first) {
        const float *W = params + (L == 1 ? OFF_W2 : OFF_W3);
        for (int v = t; v < NV; v += kBwdThreads) {
            float s = 0.f;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint4 raw = reinterpret_cast<const uint4 *>(dbuf)[h * NV + v];
                const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16 *>(&raw);
#pragma unroll
                for (int c = 0; c < 8; c++) s = __fmaf_rn(__bfloat162float(a[c]), __bfloat162float(a[c]), s);
            }
            dzs[v] = s;
        }
        if (t == 0) *near_count = 0;
        __syncthreads();
        for (int v = t; v < NV; v += kBwdThreads) {
            const int q = v >> 8, z = (v >> 5) & 7, y = v & 31;
            float s = 0.f;
            for (int zy = 0; zy < 9; zy++) {
                const int at = (((z + zy / 3 - 1) & 7) << 5) | ((y + zy % 3 - 1) & 31);
                for (int qi = max(q - 1, 0); qi <= min(q + 1, NQ - 1); qi++) s += dzs[qi * NZY + at];
            }
            reach[v] = s > 0.f ? sqrtf(s) : kNoMargin;
        }
        __syncthreads();
        const DgradNear N = {reach, wmax + 16 * (L - 1), near_list, near_count};
        dgrad16(dbuf, d, act, L == 1 ? w2 : w3, W, N);
        __syncthreads();
        const int n = min(*near_count, kNearCap);
        for (int i = t; i < n; i += kBwdThreads) {
            const int id = near_list[i];
            act[((id & 15) >> 3) * NV * 8 + (id >> 4) * 8 + (id & 7)] = __float2bfloat16_rn(dgrad_one(dbuf, W, id));
        }
        __syncthreads();
        channel_sums(act, red);
        __syncthreads();
        if (t < NC) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < 4; w++) s += red[(4 * (t >> 3) + w) * 20 + (t & 7)];
            put_grad(gp + off + t, s, first);
        }
    };
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const bool first = tile == blockIdx.x;
        __syncthreads();   // the previous tile is done with the buffers
        // dz = dL/dz_head = 2 (p a - c) / S * p (1 - p); loss partial sums
        for (int v = t; v < NV; v += kBwdThreads) {
            const float pv = pg[tile * NV + v];
            const float2 ac = acg[tile * NV + v];
            const float dp = 2.0f * (pv * ac.x - ac.y) * inv;
            dzs[v] = dp * pv * (1.0f - pv);
            l += (double)((pv * pv * ac.x - 2.0f * pv * ac.y) * inv);
        }
        load_act(sB, a3g + tile * NC * NV);
        __syncthreads();
        // head: d wh[c] = sum_v dz[v] A3[c][v], d bh = sum_v dz[v];
        // dZ3 = bf16(dz wh[c] (A3 > 0)) and its sums (layer 3's bias gradient)
        if (t < 256) {
            const int h = t >> 7;
            float sw[8] = {}, sb[8] = {}, sz = 0.f, wh[8];
#pragma unroll
            for (int c = 0; c < 8; c++) wh[c] = params[OFF_WH + 8 * h + c];
            for (int v = t & 127; v < NV; v += 128) {
                const float dz = dzs[v];
                const uint4 raw = reinterpret_cast<const uint4 *>(bufB)[h * NV + v];
                const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16 *>(&raw);
                __align__(16) __nv_bfloat16 o[8];
                sz += dz;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float av = __bfloat162float(a[c]);
                    sw[c] = __fmaf_rn(dz, av, sw[c]);
                    o[c] = __float2bfloat16_rn(av > 0.f ? dz * wh[c] : 0.f);
                    sb[c] += __bfloat162float(o[c]);
                }
                reinterpret_cast<uint4 *>(bufA)[h * NV + v] = *reinterpret_cast<const uint4 *>(o);
            }
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) {
                sz += __shfl_xor_sync(0xffffffffu, sz, m);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    sw[c] += __shfl_xor_sync(0xffffffffu, sw[c], m);
                    sb[c] += __shfl_xor_sync(0xffffffffu, sb[c], m);
                }
            }
            if (lane == 0) {
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    red[warp * 20 + c] = sw[c];
                    red[warp * 20 + 8 + c] = sb[c];
                }
                red[warp * 20 + 16] = sz;
            }
        }
        __syncthreads();
        if (t < 33) {
            const int h = (t & 15) >> 3, i = t < 32 ? (t >> 4) * 8 + (t & 7) : 16;
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < 4; w++) s += red[(4 * (t < 32 ? h : 0) + w) * 20 + i];
            put_grad(gp + (t < 16 ? OFF_WH + t : t < 32 ? OFF_B3 + t - 16 : OFF_BH), s, first);
        }
        load_act(sB, a2g + tile * NC * NV);
        __syncthreads();
        // layer 3: weight gradient, then dA2 -> dZ2 in place of A2
        wgrad16(sB, sA, gp + OFF_W3, first);
        __syncthreads();
        input_gradient(2, bufA, sA, bufB, OFF_B2, first);
        __syncthreads();   // dZ3 has been read, dZ2 is complete
        load_act(sA, a1g + tile * NC * NV);
        __syncthreads();
        // layer 2
        wgrad16(sA, sB, gp + OFF_W2, first);
        __syncthreads();
        input_gradient(1, bufB, sB, bufA, OFF_B1, first);
        // layer 1: the two input channels at q - 1, q, q + 1 as six rows of M,
        // so only the (dz, dy) taps remain
        {
            const __nv_bfloat16 *f = reinterpret_cast<const __nv_bfloat16 *>(feat + tile * NV);
            __syncthreads();   // dZ2 has been read
            for (int v = t; v < NV; v += kBwdThreads) {
                const int q = v >> 8, zy = v & 255, z = zy >> 5, y = zy & 31;
                const int mzy = (((10 - z) & 7) << 5) | ((40 - y) & 31);
                __align__(16) __nv_bfloat16 x[8];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const int qi = q + j - 1;
                    const bool in = qi >= 0 && qi < NQ;
                    x[2 * j] = in ? f[qi * NZY + zy] : __float2bfloat16_rn(0.f);
                    x[2 * j + 1] = in ? f[(4 - qi) * NZY + mzy] : __float2bfloat16_rn(0.f);
                }
                x[6] = x[7] = __float2bfloat16_rn(0.f);
                reinterpret_cast<uint4 *>(bufB)[v] = *reinterpret_cast<const uint4 *>(x);
            }
            __syncthreads();
            const int dz = warp / 3 - 1, dy = warp % 3 - 1;
            const int mi = lane >> 3, ra = (lane & 7) + (mi & 1) * 8;
            float acc[2][4] = {};
#pragma unroll 1
            for (int u = 0; u < 16; u++) {
                const int kz = u >> 1, blk = u & 1;
                const uint32_t pa = sB + ((((kz + dz) & 7) << 5) | ((16 * blk + ra + dy) & 31)) * 16;
                const uint32_t pb = sA + ((mi >> 1) * NV + ((kz << 5) | (16 * blk + ra))) * 16;
                float c[2][4] = {};
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    uint32_t a0, a2, B[4];
                    ldsm2t(pa + q * NZY * 16, a0, a2);
                    ldsm4t(pb + q * NZY * 16, B);
                    mma16816(c[0], a0, 0u, a2, 0u, B[0], B[1]);
                    mma16816(c[1], a0, 0u, a2, 0u, B[2], B[3]);
                }
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    acc[n][0] += c[n][0];
                    acc[n][1] += c[n][1];
                }
            }
            const int g = lane >> 2, tq = lane & 3;
            if (g < 6)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int i = 0; i < 2; i++)
                        put_grad(gp + OFF_W1 + ((warp * 3 + (g >> 1)) * NCIN + (g & 1)) * NC + 8 * n + 2 * tq + i, acc[n][i], first);
        }
    }
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) l += __shfl_xor_sync(0xffffffffu, l, h);
    if (lane == 0) atomicAdd(loss, l);
}

// One Adam step: g = sum over the partial slices; the FP32 master weights
// move, and `used` gets the values the kernels compute with (weights rounded
// to bf16, biases as they are). A block takes 32 parameters, eight warps an
// eighth of the slices each: one thread a parameter summed the slices one
// after another on 58 blocks (101 us at 152 slices).
__global__ void __launch_bounds__(256)
    mn_adam_kernel(float *master, float *used, float *m, float *v, const float *gpart, int nslices, float lr, float b1,
                   float b2, float eps, float c1, float c2, float *grad_out)
{
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < NPARAM)
#pragma unroll 8
        for (int k = grp; k < nslices; k += 8) s += gpart[(size_t)k * NPARAM + i];
    part[grp][lane] = s;
    __syncthreads();
    if (grp != 0 || i >= NPARAM) return;
    float g = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) g += part[k][lane];
    if (grad_out) grad_out[i] = g;
    if (lr == 0.f) return;
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float w = master[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    master[i] = w;
    const bool bias = (i >= OFF_B1 && i < OFF_W2) || (i >= OFF_B2 && i < OFF_W3) || (i >= OFF_B3 && i < OFF_WH) ||
                      i == OFF_BH;
    used[i] = bias ? w : bfr(w);
}

// Training pairs per bin: (|X|^2, Re(C conj X)) from the composite's and the
// true chroma's spectra
__global__ void mn_pairs_kernel(const float2 *x, const float2 *c, long long n, float2 *ac)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float2 a = x[i], b = c[i];
        ac[i] = make_float2(a.x * a.x + a.y * a.y, b.x * a.x + b.y * a.y);
    }
}

__global__ void mn_round_kernel(const float *master, float *used)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    const bool bias = (i >= OFF_B1 && i < OFF_W2) || (i >= OFF_B2 && i < OFF_W3) || (i >= OFF_B3 && i < OFF_WH) ||
                      i == OFF_BH;
    used[i] = bias ? master[i] : bfr(master[i]);
}

// ---------------------------------------------------------------------------
// Tensor-core forward pass (tcgen05): each convolution as implicit GEMMs
// ---------------------------------------------------------------------------
// Rows m = ky * 8 + kz (kz fastest: each ky is one 8-row core-matrix group;
// 256 rows, two M blocks of 128), K = (q', ci) of the layer's input, N =
// (q, dz, co): the kz taps are outputs, D_dz(ky, kz) = sum over (dy, q', ci)
// of x(ky + dy - 1, kz) W[dz][dy][q' - q], and the epilogue forms
// y(ky, kz) = sum_dz D_dz(ky, kz + dz - 1) with shuffles inside the 8 lanes
// of each ky (the kz axis is periodic, as the lanes are). A ky tap is an
// offset of whole groups into the one A operand (a periodic halo group on
// both sides). The kx taps fold into N and K: output block q takes input
// block q' through W[.][.][q' - q] for |q' - q| <= 1, so in layers 2 and 3
// the MMAs of one K chunk (input q', its 16 channels) write only the 96 or
// 144 columns of the outputs q = q' - 1 .. q' + 1 (N is ordered q, dz, co).
// Layer 1 (K = 16: the five q' of the two input channels, zero-padded) takes
// the full N = 240. Each M block has its own 240 accumulator columns.
//
// Schedule: the M blocks take turns. A layer's block-0 MMAs, then its block-1
// MMAs, which run while the epilogue empties block 0; block 1's epilogue then
// runs while the next layer's block-0 MMAs go, chunk by chunk as it releases
// them. Block 0's epilogue writes the next layer's input while block 1's MMAs
// still read this layer's: the two row groups both touch (ky = 15, and the
// halo copy of ky = 0) go to a stash that block 1's epilogue moves into place.
//
// Roles (one CTA per SM, persistent over tiles):
//  * warps 0-7, the epilogue, all on one M block at a time: warp w reads
//    tensor-memory lanes 32 (w & 3) .. and the channel half w >> 2 of each
//    output. Per output block q = 0..4 of a layer: read its columns, zero them
//    for the next layer (whose banded MMAs all accumulate), add the dz partial
//    sums, the bias and ReLU, round to bf16 and write K chunk q of the next
//    layer's input; block 1's step q releases the next layer's chunk q. The
//    last layer: the sigmoid head over all 16 channels, warps 0-3 taking
//    output blocks q = 0..2 and warps 4-7 q = 3..4; after block 0's head,
//    warps 4-7 write the next tile's input.
//  * warp 8, one thread: issues the MMAs.
//  * warp 9, one thread: the TMA bulk copies -- the weight pieces of each
//    tile (each used by both M blocks) through a ring of slots, and each next
//    tile's features into one of two stages.
// All waits are bounded; a wait that runs out raises the error flag and the
// CTA leaves after its copies and MMAs in flight have completed.
constexpr int kEpiWarps = 8;
constexpr int kTcThreads = 32 * (kEpiWarps + 2);
constexpr int kGroupsA = 34;                       // 32 ky groups + one halo group on each side
constexpr int A_BYTES = kGroupsA * 8 * 160;         // a layer's input, K up to 80
constexpr int NCOL = 3 * 80;                       // accumulator columns of one M block: (q, dz, co)
constexpr int kSlots = 8;                          // weight-piece ring (a layer's 5 pieces stay for both blocks)
constexpr int SLOT_BYTES = 3 * 144 * 32;           // the largest piece: three ky taps x 144 rows x K 16
constexpr int FEAT_BYTES = NV * 2;
constexpr int kPieces = 10;                        // streamed weight pieces of one tile (layers 2 and 3)
constexpr int W1_BYTES = 3 * NCOL * 32;            // layer 1's weights, resident
constexpr int STASH_BYTES = 2 * 8 * 160;           // row groups 16 and 33 of the next layer's input
constexpr int IN_BYTES = kGroupsA * 8 * 32;         // layer 1's input, K = 16
// shared memory: layers 2 and 3's input [34 groups][8 rows][K 80] and layer
// 1's [34][8][K 16], both canonical (apart, so a tile's input can be written
// while the previous layers' operands are read), the ring, two feature
// stages, the stash, the barriers
constexpr int SM_A = 0;
constexpr int SM_IN = A_BYTES;
constexpr int SM_W1 = SM_IN + IN_BYTES;
constexpr int SM_SLOT = SM_W1 + W1_BYTES;
constexpr int SM_FEAT = SM_SLOT + kSlots * SLOT_BYTES;
constexpr int SM_STASH = SM_FEAT + 2 * FEAT_BYTES;
constexpr int SM_BAR = SM_STASH + STASH_BYTES;
// barriers: an M block's MMAs of a layer done (2); a release of the MMAs (5:
// chunk q of the next layer's input written, and for layer 1 the input (0)
// and block 1's columns read (1)); slot full (kSlots); slot free (kSlots);
// feature stage full (2) and free (2); the final drain of the MMAs; layer
// 1's weights landed
constexpr int B_FULL = 0, B_READY = 2, B_SFULL = B_READY + 5, B_SFREE = B_SFULL + kSlots, B_FFULL = B_SFREE + kSlots,
              B_FFREE = B_FFULL + 2, B_DRAIN = B_FFREE + 2, B_W1 = B_DRAIN + 1, NBAR = B_W1 + 1;
constexpr int SM_TSLOT = SM_BAR + 8 * NBAR;
constexpr int SM_FLAG = SM_TSLOT + 4;
constexpr int kTcSmem = SM_FLAG + 12;
static_assert(kTcSmem + 1024 <= 227 * 1024, "shared memory of one CTA");
static_assert(SM_IN % 16 == 0 && SM_W1 % 16 == 0 && SM_SLOT % 16 == 0 && SLOT_BYTES % 16 == 0 &&
                  SM_FEAT % 16 == 0 && SM_STASH % 16 == 0 && SM_BAR % 8 == 0,
              "copy alignment");

// the band of output blocks of input block (K chunk) ks in layers 2 and 3
__host__ __device__ constexpr int band_lo(int ks) { return ks > 0 ? ks - 1 : 0; }
__host__ __device__ constexpr int band_q(int ks) { return (ks < 4 ? ks + 1 : 4) - band_lo(ks) + 1; }
__host__ __device__ constexpr int band_off(int ks)
{
    int o = 0;
    for (int k = 0; k < ks; k++) o += 3 * 48 * band_q(k) * 32;
    return o;
}
// weight images in global memory, in the order the MMAs take them: layer 1
// [dy][240 rows (q, dz, co)][K 16]; layers 2 and 3 [chunk ks][dy][48 x
// band_q(ks) rows][K 16]; each ky tap's image canonical (8-row groups 256
// bytes apart)
constexpr int IMG_L1 = 0;
constexpr int IMG_L2 = IMG_L1 + 3 * NCOL * 32;
constexpr int IMG_L3 = IMG_L2 + band_off(5);
constexpr int IMG_BYTES = IMG_L3 + band_off(5);
static_assert(band_off(5) == 3 * 48 * 13 * 32, "band sizes");
static_assert(NCOL * 32 <= SLOT_BYTES, "pieces fit a slot");

// Streamed piece p of a tile's weights: source offset and bytes. Pieces
// 0-4: layer 2's chunks; 5-9: layer 3's. Layer 1's weights stay in shared
// memory.
__device__ __forceinline__ void weight_piece(int p, int &off, int &bytes)
{
    const int ks = p % 5;
    off = (p < 5 ? IMG_L2 : IMG_L3) + band_off(ks);
    bytes = 3 * 48 * band_q(ks) * 32;
}

// The weight images, and behind them the backward pass's B fragments of
// layers 2 and 3: [tap][lane] of (n 0 k-low, n 0 k-high, n 1 ..., n 1 ...).
__global__ void mn_build_images_kernel(const float *used, uint8_t *img)
{
    const int n1 = 3 * NCOL * 16, n2 = 3 * 48 * 13 * 16, n3 = 27 * 32 * 8;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n1 + 2 * n2 + 2 * n3; idx += gridDim.x * blockDim.x) {
        if (idx >= n1 + 2 * n2) {
            const int e = idx - n1 - 2 * n2, layer = e / n3, r = e % n3;
            const int part = r & 1, reg = (r >> 1) & 3, lane = (r >> 3) & 31, tap = r >> 8;
            const int ci = 8 * (reg >> 1) + (lane >> 2), co = 8 * (reg & 1) + 2 * (lane & 3) + part;
            reinterpret_cast<__nv_bfloat16 *>(img + IMG_BYTES)[e] =
                __float2bfloat16_rn(used[(layer == 0 ? OFF_W2 : OFF_W3) + (tap * NC + ci) * NC + co]);
            continue;
        }
        const int k = idx & 15;
        float v = 0.f;
        uint32_t off;
        if (idx < n1) {
            const int n = (idx >> 4) % NCOL, dy = (idx >> 4) / NCOL;
            const int q = n / 48, dz = (n % 48) >> 4, co = n & 15;
            if (k < 5 * NCIN) {
                const int dq = k / NCIN - q, ci = k % NCIN;
                if (dq >= -1 && dq <= 1) v = used[OFF_W1 + (((dz * 3 + dy) * 3 + dq + 1) * NCIN + ci) * NC + co];
            }
            off = IMG_L1 + dy * NCOL * 32 + tpal::tc::elem_off(n, k, 2, 32);
        } else {
            const int r = idx - n1, layer = r < n2 ? 1 : 2, rr = (r % n2) >> 4;
            int ks = 0;
            while (rr >= band_off(ks + 1) / 32) ks++;
            const int nb = 48 * band_q(ks), within = rr - band_off(ks) / 32, dy = within / nb, n = within % nb;
            const int q = band_lo(ks) + n / 48, dz = (n % 48) >> 4, co = n & 15, dq = ks - q;   // |dq| <= 1
            v = used[(layer == 1 ? OFF_W2 : OFF_W3) + (((dz * 3 + dy) * 3 + dq + 1) * NC + k) * NC + co];
            off = (layer == 1 ? IMG_L2 : IMG_L3) + band_off(ks) + dy * nb * 32 + tpal::tc::elem_off(n, k, 2, 32);
        }
        *reinterpret_cast<__nv_bfloat16 *>(img + off) = __float2bfloat16_rn(v);
    }
}

// One 16-byte chunk c of input row (ky, kz) of a layer whose rows hold KB
// bytes: row kz of group ky + 1; groups 0 and 33 repeat ky = 31 and ky = 0
// (the periodic halo).
__device__ __forceinline__ void put_row(uint8_t *A, int KB, int ky, int kz, int c, uint4 v)
{
    const int grp = 8 * KB;
    uint8_t *base = A + c * 128 + kz * 16;
    *reinterpret_cast<uint4 *>(base + (ky + 1) * grp) = v;
    if (ky == 31) *reinterpret_cast<uint4 *>(base) = v;
    if (ky == 0) *reinterpret_cast<uint4 *>(base + (kGroupsA - 1) * grp) = v;
}

// OR of a predicate over an epilogue's 256 threads (named barrier id).
__device__ __forceinline__ bool epi_or(bool v, int id = 1)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\tbar.red.or.pred p, %3, %2, q;\n\t"
                 "selp.b32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(r)
                 : "r"((uint32_t)v), "r"(32 * kEpiWarps), "r"(id)
                 : "memory");
    return r != 0;
}

struct TcShared {
    uint8_t *A, *in, *w1, *slots, *stage;
    uint64_t *bars;
    volatile int *abort_flag;
};

// Descriptor arithmetic: the start address is bits 0-13 of a shared-memory
// descriptor in 16-byte units, so moving an operand by a byte offset that
// keeps it inside shared memory (below 256 KB) adds offset / 16.
__device__ __forceinline__ uint64_t desc_at(uint64_t d, uint32_t bytes) { return d + (bytes >> 4); }

// Layer 1, ky tap DY of one M block from its weight piece: K = 16, N = 240;
// tap 0 starts the block's sum. ab: A at the block's first row group.
template <int DY>
__device__ __forceinline__ void mma_layer1(uint32_t d, uint64_t ab, uint64_t bslot)
{
    tpal::tc::mma<1>(d, desc_at(ab, DY * 256), bslot, tpal::tc::idesc(1, 128, NCOL), DY > 0 ? 1u : 0u);
}

// Layers 2 and 3, K chunk KS (input block q' = KS) of one M block: three ky
// taps into the band's 96 or 144 columns; every MMA accumulates.
template <int KS>
__device__ __forceinline__ void mma_band(uint32_t d, uint64_t ab, uint64_t bslot)
{
    constexpr int nb = 48 * band_q(KS);
    constexpr uint32_t id = tpal::tc::idesc(1, 128, nb);
#pragma unroll
    for (int dy = 0; dy < 3; dy++)
        tpal::tc::mma<1>(d + 48 * band_lo(KS), desc_at(ab, dy * 1280 + KS * 256), desc_at(bslot, dy * nb * 32), id,
                         1u);
}

__device__ __forceinline__ void mma_band_any(int ks, uint32_t d, uint64_t ab, uint64_t bslot)
{
    switch (ks) {
    case 0: mma_band<0>(d, ab, bslot); break;
    case 1: mma_band<1>(d, ab, bslot); break;
    case 2: mma_band<2>(d, ab, bslot); break;
    case 3: mma_band<3>(d, ab, bslot); break;
    default: mma_band<4>(d, ab, bslot); break;
    }
}

// The MMA warp's thread. Per tile and layer: block 0's MMAs (each chunk once
// released), then block 1's with the same weight pieces, whose slots are then
// freed.
__device__ bool tc_mma_role(const TcShared &S, uint32_t tmem, long long first, long long step, long long ntiles)
{
    using namespace tpal::tc;
    uint64_t *full = S.bars + B_FULL, *ready = S.bars + B_READY, *sfull = S.bars + B_SFULL,
             *sfree = S.bars + B_SFREE;
    // operand descriptors at the bases: A with 8-row groups 256 bytes apart
    // (layer 1) or 1280 (layers 2 and 3), the weight slots 256; block 1's A
    // starts 16 row groups in
    const uint64_t a1 = sdesc(smem_addr(S.in), 256), a2 = sdesc(smem_addr(S.A), 1280),
                   b0 = sdesc(smem_addr(S.slots), 256);
    const uint64_t a1b[2] = {a1, desc_at(a1, 16 * 256)}, a2b[2] = {a2, desc_at(a2, 16 * 1280)};
    uint32_t rbits = 0;   // parity of each release barrier's next phase
    long long sc = 0;     // weight pieces taken
    bool ok = true;
    auto take_ready = [&](int q) {
        if (!bar_wait(ready + q, (rbits >> q) & 1)) return false;
        rbits ^= 1u << q;
        fence_after();
        return true;
    };
    // the weight piece p's slot, once its copy has landed
    auto take_slot = [&](long long p) {
        if (!bar_wait(sfull + (int)(p % kSlots), (uint32_t)((p / kSlots) & 1))) return false;
        fence_after();
        return true;
    };
    auto slot_desc = [&](long long p) { return desc_at(b0, (int)(p % kSlots) * SLOT_BYTES); };
    // layer 1's weights, copied once
    const uint64_t w1 = sdesc(smem_addr(S.w1), 256);
    if (ntiles > first) {
        ok = bar_wait(S.bars + B_W1, 0);
        fence_after();
    }
    for (long long tile = first; tile < ntiles && ok && !*S.abort_flag; tile += step) {
        // layer 1: block 0 once the tile's input is written and the previous
        // tile's head has read block 0's columns, block 1 once it has read
        // block 1's
        ok = take_ready(0);
        if (ok) {
            mma_layer1<0>(tmem, a1b[0], w1);
            mma_layer1<1>(tmem, a1b[0], desc_at(w1, NCOL * 32));
            mma_layer1<2>(tmem, a1b[0], desc_at(w1, 2 * NCOL * 32));
        }
        mma_commit(full + 0);
        if (ok) ok = take_ready(1);
        if (ok) {
            mma_layer1<0>(tmem + 256, a1b[1], w1);
            mma_layer1<1>(tmem + 256, a1b[1], desc_at(w1, NCOL * 32));
            mma_layer1<2>(tmem + 256, a1b[1], desc_at(w1, 2 * NCOL * 32));
        }
        mma_commit(full + 1);
        // layers 2 and 3: block 0's chunk ks once block 1's epilogue of the
        // previous layer released it (the weight piece is taken first: it
        // landed long before, so that wait overlaps the epilogue step that
        // releases the chunk); block 1's chunks need nothing more
        for (int L = 1; L < 3 && ok; L++) {
            const long long p = sc;
            for (int ks = 0; ks < 5 && ok; ks++) {
                ok = take_slot(p + ks) && take_ready(ks);
                if (ok) mma_band_any(ks, tmem, a2b[0], slot_desc(p + ks));
            }
            mma_commit(full + 0);
            if (ok) {
                for (int ks = 0; ks < 5; ks++) {
                    mma_band_any(ks, tmem + 256, a2b[1], slot_desc(p + ks));
                    mma_commit(sfree + (int)((p + ks) % kSlots));
                }
            }
            mma_commit(full + 1);
            sc += 5;
        }
    }
    if (!ok) *S.abort_flag = 1;
    // every MMA issued has completed before the tensor memory is released
    mma_commit(S.bars + B_DRAIN);
    return bar_wait(S.bars + B_DRAIN, 0) && ok;
}

// The copy warp's thread: weight pieces through the ring, features of the
// next tile into the other stage.
__device__ bool tc_copy_role(const TcShared &S, const uint8_t *img, const uint16_t *feat, long long first,
                             long long step, long long ntiles)
{
    using namespace tpal::tc;
    uint64_t *sfull = S.bars + B_SFULL, *sfree = S.bars + B_SFREE, *ffull = S.bars + B_FFULL,
             *ffree = S.bars + B_FFREE;
    long long sc = 0;   // pieces issued
    long long js = 0;   // tiles whose features were issued
    bool ok = true;
    auto stage_features = [&](long long tile) {
        const int b = (int)(js & 1);
        const long long use = js >> 1;   // earlier fills of this stage
        if (use >= 1 && !bar_wait(ffree + b, (uint32_t)((use - 1) & 1))) return false;
        bar_arrive_expect_tx(ffull + b, FEAT_BYTES);
        bulk_g2s(S.stage + b * FEAT_BYTES, feat + tile * NV, FEAT_BYTES, ffull + b);
        js++;
        return true;
    };
    if (first < ntiles) {
        bar_arrive_expect_tx(S.bars + B_W1, W1_BYTES);
        bulk_g2s(S.w1, img + IMG_L1, W1_BYTES, S.bars + B_W1);
        ok = stage_features(first);
    }
    for (long long tile = first; tile < ntiles && ok && !*S.abort_flag; tile += step) {
        if (tile + step < ntiles) ok = stage_features(tile + step);
        for (int pc = 0; pc < kPieces && ok; pc++) {
            const int slot = (int)(sc % kSlots);
            const long long use = sc / kSlots;
            if (use >= 1 && !bar_wait(sfree + slot, (uint32_t)((use - 1) & 1))) {
                ok = false;
                break;
            }
            int off, bytes;
            weight_piece(pc, off, bytes);
            bar_arrive_expect_tx(sfull + slot, (uint32_t)bytes);
            bulk_g2s(S.slots + slot * SLOT_BYTES, img + off, (uint32_t)bytes, sfull + slot);
            sc++;
        }
    }
    if (!ok) *S.abort_flag = 1;
    // no copy may still be writing shared memory when the CTA leaves: wait
    // for the last fill of every slot and stage (already complete unless a
    // wait ran out)
    for (int slot = 0; slot < kSlots; slot++)
        if (sc > slot && !bar_wait(sfull + slot, (uint32_t)(((sc - 1 - slot) / kSlots) & 1))) ok = false;
    for (int b = 0; b < 2; b++)
        if (js > b && !bar_wait(ffull + b, (uint32_t)(((js - 1 - b) >> 1) & 1))) ok = false;
    if (first < ntiles && !bar_wait(S.bars + B_W1, 0)) ok = false;
    return ok;
}

// The 24 accumulator columns of output block q and channel half h of the
// thread's lane (q * 48 + dz * 16 + 8 h + c; tl already holds 8 h): loads
// issued, not waited for.
__device__ __forceinline__ void load_half(uint32_t tl, int q, uint32_t (&d)[24])
{
    tpal::tc::tmem_ld8_async(tl + q * 48, &d[0]);
    tpal::tc::tmem_ld8_async(tl + q * 48 + 16, &d[8]);
    tpal::tc::tmem_ld8_async(tl + q * 48 + 32, &d[16]);
}

// The half block's outputs: the three dz partial sums of each channel added
// with the kz neighbours' (lanes of the same ky holding kz - 1 and kz + 1).
__device__ __forceinline__ void combine_half(const uint32_t (&d)[24], int lane, float (&y)[8])
{
    const int lm = (lane & ~7) | ((lane - 1) & 7), lp = (lane & ~7) | ((lane + 1) & 7);
#pragma unroll
    for (int c = 0; c < 8; c++)
        y[c] = __shfl_sync(0xffffffffu, __uint_as_float(d[c]), lm) + __uint_as_float(d[8 + c]) +
               __shfl_sync(0xffffffffu, __uint_as_float(d[16 + c]), lp);
}

// The 48 columns of output block q, all 16 channels (the head).
__device__ __forceinline__ void load_block(uint32_t tl, int q, uint32_t (&d)[48])
{
    uint32_t(&d0)[16] = *reinterpret_cast<uint32_t(*)[16]>(&d[0]);
    uint32_t(&d1)[16] = *reinterpret_cast<uint32_t(*)[16]>(&d[16]);
    uint32_t(&d2)[16] = *reinterpret_cast<uint32_t(*)[16]>(&d[32]);
    tpal::tc::tmem_ld16_async(tl + q * 48, d0);
    tpal::tc::tmem_ld16_async(tl + q * 48 + 16, d1);
    tpal::tc::tmem_ld16_async(tl + q * 48 + 32, d2);
}

__device__ __forceinline__ void combine_block(const uint32_t (&d)[48], int lane, float (&y)[16])
{
    const int lm = (lane & ~7) | ((lane - 1) & 7), lp = (lane & ~7) | ((lane + 1) & 7);
#pragma unroll
    for (int co = 0; co < 16; co++)
        y[co] = __shfl_sync(0xffffffffu, __uint_as_float(d[co]), lm) + __uint_as_float(d[16 + co]) +
                __shfl_sync(0xffffffffu, __uint_as_float(d[32 + co]), lp);
}

template <bool TRAIN>
__global__ void __launch_bounds__(kTcThreads, 1)
    mn_tc_forward_kernel(const uint8_t *img, const float *params, const uint16_t *feat, long long ntiles,
                         float conf_limit, float *p_out, uint8_t *fallback, __nv_bfloat16 *a1g, __nv_bfloat16 *a2g,
                         __nv_bfloat16 *a3g, int *err)
{
    using namespace tpal::tc;
    extern __shared__ __align__(1024) uint8_t smem[];
    TcShared S;
    S.A = smem + SM_A;
    S.in = smem + SM_IN;
    S.w1 = smem + SM_W1;
    S.slots = smem + SM_SLOT;
    S.stage = smem + SM_FEAT;
    S.bars = reinterpret_cast<uint64_t *>(smem + SM_BAR);
    S.abort_flag = reinterpret_cast<volatile int *>(smem + SM_FLAG);
    uint8_t *stash = smem + SM_STASH;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + SM_TSLOT);
    __shared__ float s_par[4 * NC + 1];   // b1, b2, b3, wh, bh
    __shared__ float red[2][kEpiWarps];   // [parity of the tile][warp]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (int i = t; i < 4 * NC + 1; i += kTcThreads) {
        const int off[5] = {OFF_B1, OFF_B2, OFF_B3, OFF_WH, OFF_BH};
        s_par[i] = params[off[i / NC] + i % NC];
    }
    if (t == 0) {
        for (int i = 0; i < NBAR; i++) {
            const bool per_warp = (i >= B_READY && i < B_READY + 5) || i == B_FFREE || i == B_FFREE + 1;
            bar_init(S.bars + i, per_warp ? kEpiWarps : 1);
        }
        *S.abort_flag = 0;
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const long long first = blockIdx.x, step = gridDim.x;
    bool ok = true;
    if (warp == kEpiWarps) {
        if (lane == 0) ok = tc_mma_role(S, tmem, first, step, ntiles);
        __syncwarp();
    } else if (warp == kEpiWarps + 1) {
        if (lane == 0) ok = tc_copy_role(S, img, feat, first, step, ntiles);
        __syncwarp();
    } else {
        uint64_t *full = S.bars + B_FULL, *ready = S.bars + B_READY, *ffull = S.bars + B_FFULL,
                 *ffree = S.bars + B_FFREE;
        const int qd = warp & 3, h = warp >> 2;       // lane quadrant, channel half
        const int kz = lane & 7;
        const uint32_t tq = tmem + ((uint32_t)(qd * 32) << 16);   // the warp's lanes, column 0
        uint32_t fbits = 0, pfull = 0;
        long long js = 0;   // tiles whose input was written
        bool bad = false;
        // A tile's input from its feature stage, by warps 4-7 (two rows a
        // thread): row r = (ky, kz), k = 2 q + c (c = 0: the bin, 1: its
        // mirror), zero-padded to 16. Every epilogue warp releases the stage
        // and the first layer's block-0 MMAs.
        auto write_input = [&]() {
            const int b = (int)(js & 1);
            bool done = true;
            if (h == 1) {
                done = bar_wait(ffull + b, (fbits >> b) & 1);
                if (done) {
                    fbits ^= 1u << b;
                    const __nv_bfloat16 *f = reinterpret_cast<const __nv_bfloat16 *>(S.stage + b * FEAT_BYTES);
                    for (int r = t - 128; r < 256; r += 128) {
                        const int ky = r >> 3, rz = r & 7;
                        __align__(16) __nv_bfloat16 v[16];
#pragma unroll
                        for (int q = 0; q < NQ; q++) {
                            v[2 * q] = f[(q * 8 + rz) * 32 + ky];
                            v[2 * q + 1] = f[((4 - q) * 8 + ((10 - rz) & 7)) * 32 + ((40 - ky) & 31)];
                        }
#pragma unroll
                        for (int k = 10; k < 16; k++) v[k] = __float2bfloat16_rn(0.f);
#pragma unroll
                        for (int c = 0; c < 2; c++) put_row(S.in, 32, ky, rz, c, reinterpret_cast<const uint4 *>(v)[c]);
                    }
                    fence_async_smem();
                }
            }
            __syncwarp();
            if (lane == 0) {
                bar_arrive(ffree + b);
                bar_arrive(ready + 0);
            }
            js++;
            return done;
        };
        if (first < ntiles) {
            bad = !write_input();
            // block 1's columns are free for the first tile
            if (lane == 0) bar_arrive(ready + 1);
        }
        long long it = 0;
        for (long long tile = first; tile < ntiles; tile += step, it++) {
            float conf = 0.f;
            const bool more = tile + step < ntiles;
            for (int L = 0; L < 3; L++) {
                for (int b = 0; b < 2; b++) {
                    if (bad) break;
                    if (!bar_wait(full + b, (pfull >> b) & 1)) {
                        bad = true;
                        break;
                    }
                    pfull ^= 1u << b;
                    fence_after();
                    const int erow = b * 128 + qd * 32 + lane;   // the row: ky = erow >> 3, kz
                    const int ky = erow >> 3;
                    if (L < 2) {
                        const uint32_t tl = tq + b * 256 + h * 8;
                        float bias[8];
#pragma unroll
                        for (int c = 0; c < 8; c++) bias[c] = s_par[L * NC + h * 8 + c];
                        auto step_q = [&](int q, uint32_t(&cur)[24], uint32_t(&nxt)[24]) {
                            tmem_wait_ld(cur);
                            // cleared for the next layer, whose MMAs all accumulate
                            tmem_zero8(tl + q * 48);
                            tmem_zero8(tl + q * 48 + 16);
                            tmem_zero8(tl + q * 48 + 32);
                            if (q + 1 < NQ) load_half(tl, q + 1, nxt);
                            float y[8];
                            combine_half(cur, lane, y);
                            __align__(16) __nv_bfloat16 o[8];
#pragma unroll
                            for (int c = 0; c < 8; c++)
                                o[c] = __float2bfloat16_rn(fmaxf(y[c] + bias[c], 0.f));
                            const uint4 ov = *reinterpret_cast<const uint4 *>(o);
                            const int ch = 2 * q + h;   // the 16-byte chunk of the input row
                            if (b == 0) {
                                // groups 16 (ky = 15) and 33 (the halo copy of
                                // ky = 0) are still read by block 1's MMAs
                                if (ky == 15)
                                    *reinterpret_cast<uint4 *>(stash + (kz * 10 + ch) * 16) = ov;
                                else
                                    *reinterpret_cast<uint4 *>(S.A + (ky + 1) * 1280 + ch * 128 + kz * 16) = ov;
                                if (ky == 0)
                                    *reinterpret_cast<uint4 *>(stash + ((8 + kz) * 10 + ch) * 16) = ov;
                            } else {
                                put_row(S.A, 160, ky, kz, ch, ov);
                                // the stashed rows of this thread's block-0 twin (same lane)
                                if (ky == 16)
                                    *reinterpret_cast<uint4 *>(S.A + (kGroupsA - 1) * 1280 + ch * 128 + kz * 16) =
                                        *reinterpret_cast<const uint4 *>(stash + ((8 + kz) * 10 + ch) * 16);
                                if (ky == 31)
                                    *reinterpret_cast<uint4 *>(S.A + 16 * 1280 + ch * 128 + kz * 16) =
                                        *reinterpret_cast<const uint4 *>(stash + (kz * 10 + ch) * 16);
                            }
                            if (TRAIN) {
                                __nv_bfloat16 *ag = L == 0 ? a1g : a2g;
                                *reinterpret_cast<uint4 *>(ag + act_at(tile, 8 * h, (q * 8 + kz) * 32 + ky)) = ov;
                            }
                            if (b == 1) {
                                // the next layer's input chunk q is complete
                                // (block 0's rows were written before) and
                                // block 1's columns 0..q are read; after the
                                // last step all of them are zeroed
                                fence_async_smem();
                                if (q == NQ - 1) tmem_wait_st();
                                fence_before();
                                __syncwarp();
                                if (lane == 0) bar_arrive(ready + q);
                            }
                        };
                        uint32_t ba[24], bb[24];
                        load_half(tl, 0, ba);
                        step_q(0, ba, bb);
                        step_q(1, bb, ba);
                        step_q(2, ba, bb);
                        step_q(3, bb, ba);
                        step_q(4, ba, bb);
                        if (b == 0) {
                            // block 0's rows and zeroed columns, before block
                            // 1's steps release the next layer's chunks
                            fence_async_smem();
                            tmem_wait_st();
                            fence_before();
                        }
                    } else {
                        // the sigmoid head over the row's 16 channels: warps
                        // 0-3 take output blocks q = 0..2, warps 4-7 q = 3..4
                        const uint32_t tl = tq + b * 256;
                        const float zh0 = s_par[4 * NC];
                        auto head_q = [&](int q, int qend, uint32_t(&cur)[48], uint32_t(&nxt)[48]) {
                            tmem_wait_ld(cur);
                            if (q + 1 < qend) load_block(tl, q + 1, nxt);
                            float y[16];
                            combine_block(cur, lane, y);
                            const int vox = (q * 8 + kz) * 32 + ky;
                            float zh = zh0;
                            __align__(16) __nv_bfloat16 a3[TRAIN ? NC : 1];
#pragma unroll
                            for (int co = 0; co < NC; co++) {
                                const float a = bfr(fmaxf(y[co] + s_par[2 * NC + co], 0.f));
                                if (TRAIN) a3[co] = __float2bfloat16_rn(a);
                                zh = __fmaf_rn(a, s_par[3 * NC + co], zh);
                            }
                            if (TRAIN)
#pragma unroll
                                for (int hc = 0; hc < 2; hc++)
                                    *reinterpret_cast<uint4 *>(a3g + act_at(tile, 8 * hc, vox)) =
                                        reinterpret_cast<const uint4 *>(a3)[hc];
                            const float p = 1.0f / (1.0f + expf(-zh));
                            p_out[tile * NV + vox] = p;
                            conf += fabsf(p - 0.5f);
                        };
                        uint32_t ba[48], bb[48];
                        if (h == 0) {
                            load_block(tl, 0, ba);
                            head_q(0, 3, ba, bb);
                            head_q(1, 3, bb, ba);
                            head_q(2, 3, ba, bb);
                        } else {
                            load_block(tl, 3, ba);
                            head_q(3, 5, ba, bb);
                            head_q(4, 5, bb, ba);
                        }
                        // block b's columns are read: the next tile's layer-1
                        // MMAs of block b may run. During block 0, warps 4-7
                        // then write the next tile's input (layer 1's operand
                        // region is free: this tile's layer-1 MMAs are long
                        // done) and warps 0-3 only release the feature stage.
                        fence_before();
                        __syncwarp();
                        if (more) {
                            if (b == 0) {
                                if (!write_input()) bad = true;
                            } else if (lane == 0) {
                                bar_arrive(ready + 1);
                            }
                        }
                    }
                }
            }
            // the tile's confidence; a failure anywhere stops every epilogue warp here
#pragma unroll
            for (int hh = 16; hh >= 1; hh >>= 1) conf += __shfl_xor_sync(0xffffffffu, conf, hh);
            if (lane == 0) red[it & 1][warp] = conf;
            if (epi_or(bad || *S.abort_flag != 0)) {
                bad = true;
                break;
            }
            if (t == 0 && fallback != nullptr) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < kEpiWarps; w++) sum += red[it & 1][w];
                fallback[tile] = (sum * (1.0f / NV) < conf_limit) ? 1 : 0;
            }
        }
        if (bad) *S.abort_flag = 1;
        ok = !bad;
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
    if (!ok) atomicExch(err, 1);
}

// ---------------------------------------------------------------------------
// The forward pass over features that repeat
// ---------------------------------------------------------------------------
// f(kz + 4, ky + 16) = f(kz, ky), as every spectrum of a tile does (the walk's
// Z stage says why). The network commutes with shifts along its periodic axes,
// so its output repeats the same way, bit for bit, and 128 of the 256 rows
// suffice: an M block is the ky < 16 of a tile of its own, in 18 row groups
// whose halo groups are its own ky = 15 and ky = 0 with kz moved by 4.
//
// What bounds it is the way from a layer's last MMA through the epilogue to
// the next layer's first: tensor-memory loads, shuffles, conversions and
// stores of dependent steps. The two M blocks share nothing but the weights,
// so each has eight epilogue warps and a thread that issues its MMAs, and one
// block's tensor work fills the other's epilogue. Chunk ks of a layer writes
// the columns of the outputs ks - 1 .. ks + 1 of the accumulators that the
// epilogue is still emptying, so it goes as soon as output ks + 1 is read. All
// weights stay in shared memory, so nothing is streamed but the features.
//
// 62,160 tiles: whole tiles 3.80 ms; halves with one epilogue of eight warps
// that the blocks took turns in 1.88 (tensor pipe 25 % busy, issue slots 38 %);
// this 1.53 (31 %, 41 %). Releasing two and three chunks at a time instead of one
// was 1 % slower, starting each output's sum with an MMA of its own instead of
// clearing the columns 1.5 %.
constexpr int kHalfThreads = 32 * (2 * kEpiWarps + 3);
constexpr int kGroupsH = 18;
constexpr int H_A = 0;                                  // [2 blocks][18 groups][8 rows][K 80]
constexpr int H_IN = H_A + 2 * kGroupsH * 8 * 160;      // [2][18][8][K 16]
constexpr int H_W = H_IN + 2 * kGroupsH * 8 * 32;       // the weight images
constexpr int H_FEAT = H_W + IMG_BYTES;                 // [2 blocks][2 stages]
constexpr int H_BAR = H_FEAT + 4 * FEAT_BYTES;
// barriers: a block's MMAs of a layer done (2); a release of a block's MMAs
// (2 x 5: chunk ks, and the input of layer 1 at 0); the weights landed;
// feature stages full and free (2 x 2 each); the final drains
constexpr int HB_FULL = 0, HB_READY = 2, HB_W = HB_READY + 10, HB_FFULL = HB_W + 1, HB_FFREE = HB_FFULL + 4,
              HB_DRAIN = HB_FFREE + 4, kHalfBars = HB_DRAIN + 2;
constexpr int H_TSLOT = H_BAR + 8 * kHalfBars;
constexpr int H_FLAG = H_TSLOT + 4;
constexpr int kHalfSmem = H_FLAG + 4;
static_assert(kHalfSmem + 2048 <= 227 * 1024, "shared memory of one CTA");
static_assert(H_IN % 16 == 0 && H_W % 16 == 0 && H_FEAT % 16 == 0 && H_BAR % 8 == 0 && IMG_BYTES % 16 == 0,
              "copy alignment");

// combine_half in pairs of channels, plus the bias: the same sums.
__device__ __forceinline__ void combine_pairs(const uint32_t (&d)[24], int lane, const float2 (&bias)[4], float2 (&y)[4])
{
    const int lm = (lane & ~7) | ((lane - 1) & 7), lp = (lane & ~7) | ((lane + 1) & 7);
    auto nb = [&](int i, int l) {
        return make_float2(__shfl_sync(0xffffffffu, __uint_as_float(d[i]), l),
                           __shfl_sync(0xffffffffu, __uint_as_float(d[i + 1]), l));
    };
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float2 m = make_float2(__uint_as_float(d[8 + 2 * c]), __uint_as_float(d[9 + 2 * c]));
        y[c] = __fadd2_rn(__fadd2_rn(__fadd2_rn(nb(2 * c, lm), m), nb(16 + 2 * c, lp)), bias[c]);
    }
}

// bf16(max(y, 0)) of a pair of channels
__device__ __forceinline__ __nv_bfloat162 relu_pair(float2 y)
{
    return __hmax2(__floats2bfloat162_rn(y.x, y.y), __floats2bfloat162_rn(0.f, 0.f));
}

// One 16-byte chunk c of row (ky, kz) of a block's input (rows of KB bytes):
// group ky + 1, and the halo groups at ky = -1 and 16.
__device__ __forceinline__ void put_row_half(uint8_t *A, int KB, int ky, int kz, int c, uint4 v)
{
    const int grp = 8 * KB;
    uint8_t *base = A + c * 128;
    *reinterpret_cast<uint4 *>(base + (ky + 1) * grp + kz * 16) = v;
    if (ky == 15) *reinterpret_cast<uint4 *>(base + (kz ^ 4) * 16) = v;
    if (ky == 0) *reinterpret_cast<uint4 *>(base + (kGroupsH - 1) * grp + (kz ^ 4) * 16) = v;
}

// The thread that issues block b's MMAs.
__device__ bool half_mma_role(uint8_t *smem, uint32_t tmem, int b, long long first, long long step, long long count,
                              volatile int *abort_flag)
{
    using namespace tpal::tc;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + H_BAR);
    uint64_t *full = bars + HB_FULL + b, *ready = bars + HB_READY + 5 * b;
    const uint64_t a1 = sdesc(smem_addr(smem + H_IN + b * kGroupsH * 256), 256),
                   a2 = sdesc(smem_addr(smem + H_A + b * kGroupsH * 1280), 1280), w = sdesc(smem_addr(smem + H_W), 256);
    const uint32_t d = tmem + 256 * b;
    uint32_t rbits = 0;   // parity of each release barrier's next phase
    auto take_ready = [&](int q) {
        if (!bar_wait(ready + q, (rbits >> q) & 1)) return false;
        rbits ^= 1u << q;
        fence_after();
        return true;
    };
    bool ok = first >= count || bar_wait(bars + HB_W, 0);
    fence_after();
    for (long long tile = first; tile < count && ok && !*abort_flag; tile += step) {
        ok = take_ready(0);
        if (ok) {
            mma_layer1<0>(d, a1, w);
            mma_layer1<1>(d, a1, desc_at(w, NCOL * 32));
            mma_layer1<2>(d, a1, desc_at(w, 2 * NCOL * 32));
        }
        mma_commit(full);
        for (int L = 1; L < 3 && ok; L++) {
            for (int ks = 0; ks < 5 && ok; ks++) {
                ok = take_ready(ks);
                if (ok) mma_band_any(ks, d, a2, desc_at(w, (L == 1 ? IMG_L2 : IMG_L3) + band_off(ks)));
            }
            mma_commit(full);
        }
    }
    if (!ok) *abort_flag = 1;
    // every MMA issued has completed before the tensor memory is released
    mma_commit(bars + HB_DRAIN + b);
    return bar_wait(bars + HB_DRAIN + b, 0) && ok;
}

// The thread that copies the weights once and each block's next features.
__device__ bool half_copy_role(uint8_t *smem, const uint8_t *img, const uint16_t *feat, long long first, long long step,
                               long long count, volatile int *abort_flag)
{
    using namespace tpal::tc;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + H_BAR);
    bool ok = true;
    long long n[2] = {0, 0};   // features issued per block
    auto stage = [&](int b) {
        const long long tile = first + b + n[b] * step;
        if (tile >= count) return;
        const int i = 2 * b + (int)(n[b] & 1);
        if (n[b] >= 2 && !bar_wait(bars + HB_FFREE + i, (uint32_t)(((n[b] >> 1) - 1) & 1))) {
            ok = false;
            return;
        }
        bar_arrive_expect_tx(bars + HB_FFULL + i, FEAT_BYTES);
        bulk_g2s(smem + H_FEAT + i * FEAT_BYTES, feat + tile * NV, FEAT_BYTES, bars + HB_FFULL + i);
        n[b]++;
    };
    if (first < count) {
        stage(0);
        stage(1);
        bar_arrive_expect_tx(bars + HB_W, IMG_BYTES);
        bulk_g2s(smem + H_W, img, IMG_L2, bars + HB_W);
        bulk_g2s(smem + H_W + IMG_L2, img + IMG_L2, IMG_L3 - IMG_L2, bars + HB_W);
        bulk_g2s(smem + H_W + IMG_L3, img + IMG_L3, IMG_BYTES - IMG_L3, bars + HB_W);
    }
    for (long long tile = first + step; tile < count && ok && !*abort_flag; tile += step)
        for (int b = 0; b < 2 && ok; b++) stage(b);
    if (!ok) *abort_flag = 1;
    // no copy may still be writing shared memory when the CTA leaves
    for (int b = 0; b < 2; b++)
        for (long long k = n[b] > 2 ? n[b] - 2 : 0; k < n[b]; k++)
            if (!bar_wait(bars + HB_FFULL + 2 * b + (int)(k & 1), (uint32_t)((k >> 1) & 1))) ok = false;
    if (first < count && !bar_wait(bars + HB_W, 0)) ok = false;
    return ok;
}

__global__ void __launch_bounds__(kHalfThreads, 1)
    mn_tc_half_kernel(const uint8_t *img, const float *params, const uint16_t *feat, long long count, float conf_limit,
                      float *p_out, uint8_t *fallback, int *err)
{
    using namespace tpal::tc;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + H_BAR);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + H_TSLOT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + H_FLAG);
    __shared__ float s_par[4 * NC + 1];         // b1, b2, b3, wh, bh
    __shared__ float red[2][2][kEpiWarps];      // [block][parity of the tile][warp]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (int i = t; i < 4 * NC + 1; i += kHalfThreads) {
        const int off[5] = {OFF_B1, OFF_B2, OFF_B3, OFF_WH, OFF_BH};
        s_par[i] = params[off[i / NC] + i % NC];
    }
    if (t == 0) {
        for (int i = 0; i < kHalfBars; i++) {
            const bool per_warp = (i >= HB_READY && i < HB_READY + 10) || (i >= HB_FFREE && i < HB_FFREE + 4);
            bar_init(bars + i, per_warp ? kEpiWarps : 1);
        }
        *abort_flag = 0;
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    // block b's tiles: first + b, + step, ...
    const long long first = 2 * (long long)blockIdx.x, step = 2 * (long long)gridDim.x;
    bool ok = true;
    if (warp == 2 * kEpiWarps + 2) {
        if (lane == 0) ok = half_copy_role(smem, img, feat, first, step, count, abort_flag);
        __syncwarp();
    } else if (warp >= 2 * kEpiWarps) {
        const int b = warp - 2 * kEpiWarps;
        if (lane == 0) ok = half_mma_role(smem, tmem, b, first + b, step, count, abort_flag);
        __syncwarp();
    } else {
        const int b = warp >> 3, qd = warp & 3, h = (warp >> 2) & 1;   // block, lane quadrant, channel half
        uint64_t *full = bars + HB_FULL + b, *ready = bars + HB_READY + 5 * b;
        uint8_t *A = smem + H_A + b * kGroupsH * 1280, *in = smem + H_IN + b * kGroupsH * 256;
        const int kz = lane & 7, ky = qd * 4 + (lane >> 3);           // the thread's row
        const uint32_t tq = tmem + 256 * b + ((uint32_t)(qd * 32) << 16);
        uint32_t pfull = 0;
        long long js = 0;   // tiles whose input was written
        bool bad = false;
        // A tile's input from its feature stage: row (ky, kz), k = 2 q + c (c =
        // 0: the bin, 1: its mirror), zero-padded to 16, a 16-byte chunk a
        // thread; the stage is released.
        auto write_input = [&]() {
            const int i = 2 * b + (int)(js & 1);
            const bool done = bar_wait(bars + HB_FFULL + i, (uint32_t)((js >> 1) & 1));
            if (done) {
                const __nv_bfloat16 *f = reinterpret_cast<const __nv_bfloat16 *>(smem + H_FEAT + i * FEAT_BYTES);
                __align__(16) __nv_bfloat16 v[8];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int q = 4 * h + k;
                    v[2 * k] = v[2 * k + 1] = __float2bfloat16_rn(0.f);
                    if (q < NQ) {
                        v[2 * k] = f[(q * 8 + kz) * 32 + ky];
                        v[2 * k + 1] = f[((4 - q) * 8 + ((10 - kz) & 7)) * 32 + ((40 - ky) & 31)];
                    }
                }
                put_row_half(in, 32, ky, kz, h, *reinterpret_cast<const uint4 *>(v));
                fence_async_smem();
            }
            __syncwarp();
            if (lane == 0) bar_arrive(bars + HB_FFREE + i);
            js++;
            return done;
        };
        if (first + b < count) {
            bad = !write_input();
            if (lane == 0) bar_arrive(ready + 0);
        }
        long long it = 0;
        for (long long tile = first + b; tile < count; tile += step, it++) {
            float conf = 0.f;
            const bool more = tile + step < count;
            for (int L = 0; L < 2 && !bad; L++) {
                if (!bar_wait(full, pfull)) {
                    bad = true;
                    break;
                }
                pfull ^= 1;
                fence_after();
                const uint32_t tl = tq + h * 8;
                float2 bias[4];
#pragma unroll
                for (int c = 0; c < 4; c++) bias[c] = make_float2(s_par[L * NC + h * 8 + 2 * c], s_par[L * NC + h * 8 + 2 * c + 1]);
                auto step_q = [&](int q, uint32_t(&cur)[24], uint32_t(&nxt)[24]) {
                    tmem_wait_ld(cur);
                    // cleared for the next layer, whose MMAs all accumulate
                    tmem_zero8(tl + q * 48);
                    tmem_zero8(tl + q * 48 + 16);
                    tmem_zero8(tl + q * 48 + 32);
                    if (q + 1 < NQ) load_half(tl, q + 1, nxt);
                    float2 y[4];
                    combine_pairs(cur, lane, bias, y);
                    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) o[c] = relu_pair(y[c]);
                    put_row_half(A, 160, ky, kz, 2 * q + h, *reinterpret_cast<const uint4 *>(o));
                    if (q == 0) return;
                    // chunks 0 .. q - 1 are written, columns 0 .. q read and zeroed
                    fence_async_smem();
                    tmem_wait_st();
                    fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        bar_arrive(ready + q - 1);
                        if (q == NQ - 1) bar_arrive(ready + q);
                    }
                };
                uint32_t ba[24], bb[24];
                load_half(tl, 0, ba);
                step_q(0, ba, bb);
                step_q(1, bb, ba);
                step_q(2, ba, bb);
                step_q(3, bb, ba);
                step_q(4, ba, bb);
            }
            // the next tile's input, while layer 3's MMAs run (layer 1's, which
            // read this region, are done)
            if (more && !bad && !write_input()) bad = true;
            if (!bad && !bar_wait(full, pfull)) bad = true;
            if (!bad) {
                pfull ^= 1;
                fence_after();
                // the sigmoid head over the row's 16 channels, eight at a
                // time: warps 0-3 take output blocks q = 0..2, warps 4-7 q = 3..4
                float zh = 0.f;
                auto head = [&](int q, int half, bool last, uint32_t(&cur)[24], uint32_t(&nxt)[24]) {
                    tmem_wait_ld(cur);
                    if (!last) load_half(tq + (half ? 0 : 8), half ? q + 1 : q, nxt);
                    float2 y[4], bias[4];
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        bias[c] = make_float2(s_par[2 * NC + 8 * half + 2 * c], s_par[2 * NC + 8 * half + 2 * c + 1]);
                    combine_pairs(cur, lane, bias, y);
                    if (half == 0) zh = s_par[4 * NC];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const __nv_bfloat162 a = relu_pair(y[c]);
                        zh = __fmaf_rn(__low2float(a), s_par[3 * NC + 8 * half + 2 * c], zh);
                        zh = __fmaf_rn(__high2float(a), s_par[3 * NC + 8 * half + 2 * c + 1], zh);
                    }
                    if (half == 0) return;
                    const float p = 1.0f / (1.0f + expf(-zh));
                    float *po = p_out + tile * NV;
                    po[(q * 8 + kz) * 32 + ky] = p;
                    po[(q * 8 + (kz ^ 4)) * 32 + ky + 16] = p;
                    conf += 2.f * fabsf(p - 0.5f);
                };
                uint32_t ba[24], bb[24];
                const int q0 = h == 0 ? 0 : 3, q1 = h == 0 ? 3 : 5;
                load_half(tq, q0, ba);
#pragma unroll 1
                for (int q = q0; q < q1; q++) {
                    head(q, 0, false, ba, bb);
                    head(q, 1, q + 1 == q1, bb, ba);
                }
                // the block's columns are read: the next tile's layer 1 may run
                fence_before();
                __syncwarp();
                if (more && lane == 0) bar_arrive(ready + 0);
            }
            // the tile's confidence; a failure anywhere stops the block's epilogue here
#pragma unroll
            for (int hh = 16; hh >= 1; hh >>= 1) conf += __shfl_xor_sync(0xffffffffu, conf, hh);
            if (lane == 0) red[b][it & 1][warp & 7] = conf;
            if (epi_or(bad || *abort_flag != 0, 1 + b)) {
                bad = true;
                break;
            }
            if ((t & 255) == 0 && fallback != nullptr) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < kEpiWarps; w++) sum += red[b][it & 1][w];
                fallback[tile] = (sum * (1.0f / NV) < conf_limit) ? 1 : 0;
            }
        }
        if (bad) *abort_flag = 1;
        ok = !bad;
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
    if (!ok) atomicExch(err, 1);
}

}  // namespace mn

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int mn_fail(const std::string &what, int code = CHDG_E_INVALID_ARG)
{
    chd::detail::set_last_error("chdg_masknet: " + what);
    return code;
}

static int mn_cuda(const char *what, cudaError_t e)
{
    return mn_fail(std::string(what) + ": " + cudaGetErrorString(e), CHDG_E_CUDA);
}

MaskNet::~MaskNet()
{
    for (void *p : {(void *)master_, (void *)used_, (void *)m_, (void *)v_, (void *)gpart_, (void *)a1_, (void *)a2_,
                    (void *)a3_, (void *)p_, (void *)scal_, (void *)grad_, (void *)img_, (void *)err_})
        if (p) cudaFree(p);
}

int MaskNet::init()
{
    cudaError_t e;
    const size_t pb = sizeof(float) * mn::NPARAM;
    for (float **p : {&master_, &used_, &m_, &v_, &grad_})
        if ((e = cudaMalloc(p, pb)) != cudaSuccess) return mn_cuda("cudaMalloc", e);
    cudaMemset(m_, 0, pb);
    cudaMemset(v_, 0, pb);
    if ((e = cudaMalloc(&scal_, 2 * sizeof(double))) != cudaSuccess) return mn_cuda("cudaMalloc", e);
    if ((e = cudaMalloc(&img_, mn::IMG_BYTES + 2 * mn::kWFragBytes)) != cudaSuccess) return mn_cuda("cudaMalloc", e);
    if ((e = cudaMalloc(&err_, sizeof(int))) != cudaSuccess) return mn_cuda("cudaMalloc", e);
    cudaMemset(err_, 0, sizeof(int));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    grid_ = sms > 0 ? sms : 1;
    if ((e = cudaMalloc(&gpart_, sizeof(float) * mn::NPARAM * 2 * (size_t)grid_)) != cudaSuccess)
        return mn_cuda("cudaMalloc", e);
    static bool attr[64] = {};
    if (dev >= 0 && dev < 64 && !attr[dev]) {
        const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (cudaFuncSetAttribute(mn::mn_forward_kernel<false>, a, (int)mn::kFwdSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mn::mn_forward_kernel<true>, a, (int)mn::kFwdSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mn::mn_backward_kernel, a, (int)mn::kBwdSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mn::mn_tc_forward_kernel<false>, a, mn::kTcSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mn::mn_tc_half_kernel, a, mn::kHalfSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mn::mn_tc_forward_kernel<true>, a, mn::kTcSmem) != cudaSuccess)
            return mn_cuda("cudaFuncSetAttribute", cudaGetLastError());
        attr[dev] = true;
    }
    return 0;
}

int MaskNet::set_weights(const float *host, size_t n)
{
    if (n != (size_t)mn::NPARAM) return mn_fail("expected " + std::to_string(mn::NPARAM) + " parameters");
    cudaError_t e = cudaMemcpy(master_, host, sizeof(float) * n, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return mn_cuda("cudaMemcpy", e);
    cudaMemset(m_, 0, sizeof(float) * n);
    cudaMemset(v_, 0, sizeof(float) * n);
    step_ = 0;
    mn::mn_round_kernel<<<(mn::NPARAM + 255) / 256, 256>>>(master_, used_);
    if (const int rc = build_images(nullptr); rc != 0) return rc;
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return mn_cuda("round", e);
    return 0;
}

int MaskNet::build_images(cudaStream_t s)
{
    mn::mn_build_images_kernel<<<256, 256, 0, s>>>(used_, img_);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : mn_cuda("weight images", e);
}

int MaskNet::sync(cudaStream_t s) const
{
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return mn_cuda("sync", e);
    int h = 0;
    if ((e = cudaMemcpy(&h, err_, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess) return mn_cuda("sync", e);
    if (h != 0) return mn_fail("a tensor-core completion wait ran out", CHDG_E_CUDA);
    return 0;
}

int MaskNet::get_weights(float *host, size_t n) const
{
    if (n != (size_t)mn::NPARAM) return mn_fail("expected " + std::to_string(mn::NPARAM) + " parameters");
    cudaError_t e = cudaMemcpy(host, master_, sizeof(float) * n, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? 0 : mn_cuda("cudaMemcpy", e);
}

int MaskNet::forward(const uint16_t *d_feat, long long ntiles, float *d_p, uint8_t *d_fallback, cudaStream_t s,
                     bool repeating) const
{
    if (ntiles <= 0) return 0;
    if (d_feat == nullptr || d_p == nullptr) return mn_fail("forward: null buffer");
    if (tc_ && reinterpret_cast<uintptr_t>(d_feat) % 16 != 0)
        return mn_fail("forward: the feature buffer must be 16-byte aligned");
    const unsigned blocks = (unsigned)std::min<long long>(ntiles, (long long)grid_ * 1);
    if (tc_ && repeating)
        mn::mn_tc_half_kernel<<<(unsigned)std::min<long long>((ntiles + 1) / 2, grid_), mn::kHalfThreads, mn::kHalfSmem,
                                s>>>(img_, used_, d_feat, ntiles, conf_limit_, d_p, d_fallback, err_);
    else if (tc_)
        mn::mn_tc_forward_kernel<false><<<blocks, mn::kTcThreads, mn::kTcSmem, s>>>(
            img_, used_, d_feat, ntiles, conf_limit_, d_p, d_fallback, nullptr, nullptr, nullptr, err_);
    else
        mn::mn_forward_kernel<false><<<blocks, mn::kThreads, mn::kFwdSmem, s>>>(used_, d_feat, ntiles, conf_limit_,
                                                                                d_p, d_fallback, nullptr, nullptr,
                                                                                nullptr);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : mn_cuda("forward launch", e);
}

int MaskNet::ensure_batch(long long ntiles)
{
    if (ntiles <= cap_) return 0;
    for (void *p : {(void *)a1_, (void *)a2_, (void *)a3_, (void *)p_})
        if (p) cudaFree(p);
    a1_ = a2_ = a3_ = nullptr;
    p_ = nullptr;
    cap_ = 0;
    cudaError_t e;
    const size_t act = sizeof(uint16_t) * mn::NC * mn::NV * (size_t)ntiles;
    if ((e = cudaMalloc(&a1_, act)) != cudaSuccess || (e = cudaMalloc(&a2_, act)) != cudaSuccess ||
        (e = cudaMalloc(&a3_, act)) != cudaSuccess ||
        (e = cudaMalloc(&p_, sizeof(float) * mn::NV * (size_t)ntiles)) != cudaSuccess)
        return mn_cuda("training buffers", e);
    cap_ = ntiles;
    return 0;
}

// Loss and gradients of a batch; with lr > 0 one Adam step follows.
int MaskNet::train_step(const uint16_t *d_feat, const float2 *d_ac, long long ntiles, float lr, double *loss,
                        float *host_grad, cudaStream_t s)
{
    if (ntiles <= 0 || d_feat == nullptr || d_ac == nullptr) return mn_fail("train_step: empty batch or null buffer");
    if (tc_ && reinterpret_cast<uintptr_t>(d_feat) % 16 != 0)
        return mn_fail("train_step: the feature buffer must be 16-byte aligned");
    if (const int rc = ensure_batch(ntiles); rc != 0) return rc;
    const unsigned blocks = (unsigned)std::min<long long>(ntiles, grid_);
    cudaMemsetAsync(scal_, 0, 2 * sizeof(double), s);
    if (tc_)
        mn::mn_tc_forward_kernel<true><<<blocks, mn::kTcThreads, mn::kTcSmem, s>>>(
            img_, used_, d_feat, ntiles, conf_limit_, p_, nullptr, (__nv_bfloat16 *)a1_, (__nv_bfloat16 *)a2_,
            (__nv_bfloat16 *)a3_, err_);
    else
        mn::mn_forward_kernel<true><<<blocks, mn::kThreads, mn::kFwdSmem, s>>>(
            used_, d_feat, ntiles, conf_limit_, p_, nullptr, (__nv_bfloat16 *)a1_, (__nv_bfloat16 *)a2_,
            (__nv_bfloat16 *)a3_);
    const long long n = ntiles * mn::NV;
    mn::mn_sum_kernel<<<256, 256, 0, s>>>(d_ac, n, scal_);
    const unsigned slices = (unsigned)std::min<long long>(ntiles, 2 * (long long)grid_);
    mn::mn_backward_kernel<<<slices, mn::kBwdThreads, mn::kBwdSmem, s>>>(
        used_, img_ + mn::IMG_BYTES, d_feat, (const __nv_bfloat16 *)a1_, (const __nv_bfloat16 *)a2_,
        (const __nv_bfloat16 *)a3_, p_, d_ac, scal_, ntiles, gpart_, scal_ + 1);
    float c1 = 1.f, c2 = 1.f;
    if (lr > 0.f) {
        step_++;
        c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)step_)));
        c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)step_)));
    }
    mn::mn_adam_kernel<<<(mn::NPARAM + 31) / 32, 256, 0, s>>>(master_, used_, m_, v_, gpart_, (int)slices, lr, 0.9f,
                                                               0.999f, 1e-8f, c1, c2, grad_);
    if (lr > 0.f)
        if (const int rc = build_images(s); rc != 0) return rc;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return mn_cuda("train launch", e);
    if (loss != nullptr || host_grad != nullptr) {
        if (const int rc = sync(s); rc != 0) return rc;
        if (loss != nullptr) {
            double h[2];
            cudaMemcpy(h, scal_, sizeof(h), cudaMemcpyDeviceToHost);
            *loss = h[1];
        }
        if (host_grad != nullptr)
            if ((e = cudaMemcpy(host_grad, grad_, sizeof(float) * mn::NPARAM, cudaMemcpyDeviceToHost)) != cudaSuccess)
                return mn_cuda("gradient copy", e);
    }
    return 0;
}

}  // namespace chdg

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
struct chdg_masknet {
    chdg::MaskNet net;
};

namespace chdg {
MaskNet *masknet_of(chdg_masknet *n) { return &n->net; }
}  // namespace chdg

#pragma GCC visibility push(default)
extern "C" {
int chdg_masknet_create(chdg_masknet **out)
{
    if (out == nullptr) return chdg::mn_fail("create: null argument");
    *out = nullptr;
    auto n = new (std::nothrow) chdg_masknet;
    if (n == nullptr) return chdg::mn_fail("create: out of memory", CHDG_E_OOM);
    if (const int rc = n->net.init(); rc != 0) {
        delete n;
        return rc;
    }
    *out = n;
    return 0;
}

void chdg_masknet_free(chdg_masknet *n) { delete n; }

int chdg_masknet_set_weights(chdg_masknet *n, const float *w, int64_t count)
{
    if (n == nullptr || w == nullptr) return chdg::mn_fail("set_weights: null argument");
    return n->net.set_weights(w, (size_t)count);
}

int chdg_masknet_get_weights(const chdg_masknet *n, float *w, int64_t count)
{
    if (n == nullptr || w == nullptr) return chdg::mn_fail("get_weights: null argument");
    return n->net.get_weights(w, (size_t)count);
}

int chdg_masknet_set_confidence(chdg_masknet *n, float limit)
{
    if (n == nullptr || !(limit >= 0.f && limit <= 0.5f)) return chdg::mn_fail("set_confidence: limit must be in [0, 0.5]");
    n->net.set_confidence(limit);
    return 0;
}

int chdg_masknet_set_tensor_cores(chdg_masknet *n, int32_t on)
{
    if (n == nullptr) return chdg::mn_fail("set_tensor_cores: null network");
    n->net.set_tensor_cores(on != 0);
    return 0;
}

int chdg_masknet_sync(const chdg_masknet *n, void *stream)
{
    if (n == nullptr) return chdg::mn_fail("sync: null network");
    return n->net.sync((cudaStream_t)stream);
}

int chdg_masknet_forward(const chdg_masknet *n, const uint16_t *d_feat, int64_t ntiles, float *d_p,
                         uint8_t *d_fallback, void *stream)
{
    if (n == nullptr) return chdg::mn_fail("forward: null network");
    return n->net.forward(d_feat, ntiles, d_p, d_fallback, (cudaStream_t)stream);
}

int chdg_masknet_train_step(chdg_masknet *n, const uint16_t *d_feat, const float *d_ac, int64_t ntiles,
                            float learning_rate, double *loss, float *grad, void *stream)
{
    if (n == nullptr) return chdg::mn_fail("train_step: null network");
    if (!(learning_rate >= 0.f)) return chdg::mn_fail("train_step: learning rate must be >= 0");
    return n->net.train_step(d_feat, reinterpret_cast<const float2 *>(d_ac), ntiles, learning_rate, loss, grad,
                             (cudaStream_t)stream);
}

int chdg_masknet_pairs(const float *d_spec_x, const float *d_spec_c, int64_t nbins, float *d_ac, void *stream)
{
    if (d_spec_x == nullptr || d_spec_c == nullptr || d_ac == nullptr || nbins < 0)
        return chdg::mn_fail("pairs: bad arguments");
    if (nbins == 0) return 0;
    chdg::mn::mn_pairs_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const float2 *>(d_spec_x),
                                                                       reinterpret_cast<const float2 *>(d_spec_c),
                                                                       nbins, reinterpret_cast<float2 *>(d_ac));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : chdg::mn_cuda("pairs launch", e);
}

}  // extern "C"
#pragma GCC visibility pop
