// tpal2d.cu -- Transform-PAL 2D chroma separation on sm_103a.
//
// Computes what the reference's TransformPal2D does
// (src/decoders/palcolour/transform_pal_2d.cpp:107-287): per field, 16-line x
// 32-sample raised-cosine-windowed tiles, half-overlapped, starting half a
// tile above/left of the active area; rows outside the field's active lines
// are black; forward real DFT; keep a bin and its mirror about the carrier
// (x_ref = 16 - x, y_ref = (8 - y) mod 16) when their squared magnitudes are
// within the threshold ratio, for x in [4, 8]; inverse DFT / 512 and
// overlap-add into the active window. GPU structure:
//
//  * one warp per tile position of a frame's two fields, packed in the halves
//    of f32x2 registers through the Y stages: lane (j, i) holds row i of field
//    j and computes its bins kx 4..12, the only ones the filter can keep;
//  * black and each row's mean are subtracted first (they only touch bins
//    kx in {0, +-1} of the windowed row), so invalid rows are exact zeros;
//  * the 16-point Y DFTs run as two radix-4 passes, four lanes a column, with
//    exchanges through shared memory (as in the 3D walk): eight columns on the
//    32 lanes, then the ninth;
//  * for the decisions lane (j, ky) owns the bins (kx 4..8, ky) of field j and
//    reads their mirrors; decisions are FP32 with a per-kx error bound, those
//    inside it recomputed in double-float from the raw samples by the whole
//    warp; both bins of a pair are masked in place;
//  * overlap-add: tiles of one (tileY parity, tileX parity) class tile the
//    active area without overlap, so each class writes its own partial plane
//    (the same layout the 3D kernel writes, read by the demodulator).
//
// One field a warp, with the two half-warps splitting kx, DFTs by shuffles and
// 16-bit row loads, took 1,866 warp instructions a tile at 46 % issue active:
// 2.17 ms for 300 fields. This form: see tp2_launch.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "tpal_common.cuh"
#include "tpal_kernels.h"

namespace tpal {

// X-stage tables as pairs for the f32x2 instructions, theta = 2 pi kx (x - 15.5)/32,
// kx = 4..12, x < 16:
__constant__ float2 c2_xf[9][16];   // w32(x) (cos theta, -sin theta)
__constant__ float2 c2_xi[9][16];   // (2/512) (cos theta, sin theta)
__constant__ float c2_wx[16];       // w32(x), x < 16
__constant__ float c2_wy[16];       // w16(i)
__constant__ float2 c2_tw16[16];    // exp(-2 pi i r/16)
__constant__ float c2_dfx[9][32][4];  // w32(x) exp(-2 pi i kx x/32) as double-float re/im
__constant__ float c2_dfwy[16][2];
__constant__ float c2_dftw16[16][4];

static bool g_tp2_ready[64];

constexpr int kWarps2 = 4;
constexpr float kBound2 = 2.0f;
constexpr float kEps = 5.9604645e-8f;

struct Thr2 {
    float f;
    df d;
};

__device__ __forceinline__ Thr2 thr2(const T2Params &P, int frame, int ky, int kx)
{
    if (P.thr_table == nullptr) {
        if (P.frame_t2 != nullptr) {   // a batch of captures: the threshold of this frame's capture
            const float *t = P.frame_t2 + 3 * frame;
            return {t[0], {t[1], t[2]}};
        }
        return {P.t2f, {P.t2hi, P.t2lo}};
    }
    const float *t = P.thr_table + 3 * (ky * 5 + (kx - 4));
    return {t[0], {t[1], t[2]}};
}

// Exact (double-float) squared magnitudes of bin (kyb, kxb) and of its mirror.
__device__ __noinline__ void exact_pair2(const T2Params &P, int f, int tileX, int tileY, int fl_first, int fl_last,
                                         int kyb, int kxb, df &mb, df &mr)
{
    const int lane = threadIdx.x & 31;
    const int h = lane >> 4, i = lane & 15;
    const int ky = h ? ((8 - kyb) & 15) : kyb;
    const int kx = h ? 16 - kxb : kxb;
    const int fl = tileY + i;
    dfc acc = {{0.f, 0.f}, {0.f, 0.f}};
    const uint16_t *fp = field_at(P, f);   // f is an output field: inside the buffer or the table
    if (fp != nullptr && fl >= fl_first && fl < fl_last) {
        const int at0 = fl * P.fw + tileX, end = P.fw * P.fh - 1;
        dfc x1 = acc;
        for (int x = 0; x < 32; x++) {
            // never outside the field: max(min(at, end), 0)
            const float a = (float)((int)fp[__vimin_s32_relu(at0 + x, end)] - P.black);
            const float *c = c2_dfx[kx - 4][x];
            x1.re = df_add(x1.re, df_mul_f({c[0], c[1]}, a));
            x1.im = df_add(x1.im, df_mul_f({c[2], c[3]}, a));
        }
        const int r = (ky * i) & 15;
        dfc w = {{c2_dftw16[r][0], c2_dftw16[r][1]}, {c2_dftw16[r][2], c2_dftw16[r][3]}};
        const df wy = {c2_dfwy[i][0], c2_dfwy[i][1]};
        w.re = df_mul(w.re, wy);
        w.im = df_mul(w.im, wy);
        acc = dfc_mul(x1, w);
    }
#pragma unroll
    for (int m = 1; m < 16; m <<= 1) acc = dfc_add(acc, dfc_shfl_xor(acc, m));
    const df mine = df_add(df_mul(acc.re, acc.re), df_mul(acc.im, acc.im));
    const df other = df_shfl_xor(mine, 16);
    mb = h ? other : mine;
    mr = h ? mine : other;
}

__device__ __forceinline__ bool sim2(float a, float b, float t)
{
    return (__fmaf_rn(-b, t, a) >= 0.f) && (__fmaf_rn(-a, t, b) >= 0.f);
}

__device__ __forceinline__ bool unc2(float a, float b, float t, float pa, float pb)
{
    // Two bins that are exactly zero with a zero error bound (a flat or
    // black tile) need no exact pass: both outputs are zero either way.
    return ((fabsf(__fmaf_rn(-b, t, a)) <= pa + t * pb) || (fabsf(__fmaf_rn(-a, t, b)) <= pb + t * pa)) &&
           (a + b + pa + pb > 0.f);
}

__device__ __forceinline__ bool df_sim2(df a, df b, df t)
{
    const df d1 = df_sub(a, df_mul(b, t));
    const df d2 = df_sub(b, df_mul(a, t));
    return !(df_sign(d1) < 0 || df_sign(d2) < 0);
}

// Shared memory per warp (float4 units): two buffers [9 kx][16 positions],
// rows of 20, and the bound terms [9][2 fields]. Position p of 16 is stored at
// p ^ (p >> 2) where four lanes hold four neighbours each (see tpal3d.cu).
constexpr int kBuf2 = 9 * 20;
constexpr int kWarpF4_2 = 2 * kBuf2 + 5;
constexpr int kTw2 = 4 * 3;   // Y twiddles per quarter r: (x, x, y, y)
constexpr int kBlocks2 = 5;   // resident blocks a SM

__device__ __forceinline__ tw2 twiddle2(const float4 *tw, int r, int v)
{
    const float4 a = tw[3 * r + v];
    const float2 y = make_float2(a.z, a.w);
    return {make_float2(a.x, a.y), y, __fmul2_rn(y, make_float2(-1.f, -1.f))};
}

// Forward Y stage of one column (16 rows in `x` to 16 bins in `s`, position p
// holding bin rev4(p)) and the L1 norms of its rows, by the four lanes r of
// `mask`'s groups.
__device__ __forceinline__ void y_forward2(const float4 *x, float4 *ex, float4 *s, float2 *bound, const float4 *tw,
                                           int r, unsigned mask)
{
    cp2 a[4];
#pragma unroll
    for (int n = 0; n < 4; n++) a[n] = cp_of(x[r + 4 * n]);
    float A0 = 0.f, A1 = 0.f;
#pragma unroll
    for (int n = 0; n < 4; n++) {
        A0 += fabsf(a[n].re.x) + fabsf(a[n].im.x);
        A1 += fabsf(a[n].re.y) + fabsf(a[n].im.y);
    }
#pragma unroll
    for (int h = 1; h < 4; h <<= 1) {
        A0 += __shfl_xor_sync(mask, A0, h);
        A1 += __shfl_xor_sync(mask, A1, h);
    }
    if (r == 0) *bound = make_float2(A0, A1);
    const cp2 u0 = cadd(a[0], a[2]), u1 = cadd(a[1], a[3]);
    const cp2 v0 = ctw(csub(a[0], a[2]), twiddle2(tw, r, 0), false), v1 = ctw(csub(a[1], a[3]), twiddle2(tw, r, 1), false);
    const tw2 t2 = twiddle2(tw, r, 2);
    ex[0 + r] = f4_of(cadd(u0, u1));
    ex[4 + (r ^ 1)] = f4_of(ctw(csub(u0, u1), t2, false));
    ex[8 + (r ^ 2)] = f4_of(cadd(v0, v1));
    ex[12 + (r ^ 3)] = f4_of(ctw(csub(v0, v1), t2, false));
    __syncwarp(mask);
#pragma unroll
    for (int n = 0; n < 4; n++) a[n] = cp_of(ex[4 * r + (n ^ r)]);
    const cp2 w0 = cadd(a[0], a[2]), w1 = cadd(a[1], a[3]), w2 = csub(a[0], a[2]), d3 = csub(a[1], a[3]);
    s[4 * r + (0 ^ r)] = f4_of(cadd(w0, w1));
    s[4 * r + (1 ^ r)] = f4_of(csub(w0, w1));
    s[4 * r + (2 ^ r)] = f4_of({add2(w2.re, d3.im), sub2(w2.im, d3.re)});   // odd branch times -i
    s[4 * r + (3 ^ r)] = f4_of({sub2(w2.re, d3.im), add2(w2.im, d3.re)});
}

// Inverse Y stage of one column: 16 bins in `s` (bit-reversed) to 16 rows in `x`.
__device__ __forceinline__ void y_inverse2(const float4 *s, float4 *ex, float4 *x, const float4 *tw, int r, unsigned mask)
{
    cp2 G[4];
#pragma unroll
    for (int n = 0; n < 4; n++) G[n] = cp_of(s[4 * r + (n ^ r)]);
    const cp2 w0 = cadd(G[0], G[1]), w1 = csub(G[0], G[1]), w2 = cadd(G[2], G[3]), d3 = csub(G[2], G[3]);
    ex[4 * r + (0 ^ r)] = f4_of(cadd(w0, w2));
    ex[4 * r + (2 ^ r)] = f4_of(csub(w0, w2));
    ex[4 * r + (1 ^ r)] = f4_of({sub2(w1.re, d3.im), add2(w1.im, d3.re)});   // odd branch times +i
    ex[4 * r + (3 ^ r)] = f4_of({add2(w1.re, d3.im), sub2(w1.im, d3.re)});
    __syncwarp(mask);
#pragma unroll
    for (int n = 0; n < 4; n++) G[n] = cp_of(ex[4 * n + (r ^ n)]);
    const tw2 t2 = twiddle2(tw, r, 2);
    const cp2 f1 = ctw(G[1], t2, true), f3 = ctw(G[3], t2, true);
    const cp2 g0 = cadd(G[0], f1), g1 = csub(G[0], f1);
    const cp2 g2 = ctw(cadd(G[2], f3), twiddle2(tw, r, 0), true), g3 = ctw(csub(G[2], f3), twiddle2(tw, r, 1), true);
    x[r] = f4_of(cadd(g0, g2));
    x[r + 4] = f4_of(cadd(g1, g3));
    x[r + 8] = f4_of(csub(g0, g2));
    x[r + 12] = f4_of(csub(g1, g3));
}

template <bool PER_BIN>
__global__ void __launch_bounds__(32 * kWarps2, kBlocks2) tpal2d_kernel(T2Params P)
{
    __shared__ float4 s_buf[kWarps2 * kWarpF4_2];
    __shared__ float4 s_tw[kTw2];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int j = lane >> 4, i = lane & 15;
    float4 *bx = s_buf + warp * kWarpF4_2, *be = bx + kBuf2;   // rows and spectra; exchanges
    float *bnd = reinterpret_cast<float *>(be + kBuf2);        // [9][2]: A per kx and field
    for (int e = threadIdx.x; e < 12; e += blockDim.x) {
        const int r = e / 3, v = e % 3;
        const float2 w = c2_tw16[v == 0 ? r : v == 1 ? r + 4 : 2 * r];
        s_tw[3 * r + v] = make_float4(w.x, w.x, w.y, w.y);
    }
    __syncthreads();
    const int tileX0 = P.avs - 16;
    const int ntx = (P.ave - tileX0 + 15) / 16;
    // tile rows: the larger of the two field parities' grids
    const int nty = max((((P.lafl - 0) / 2 + 1) - ((P.fafl + 1 - 0) / 2 - 8) + 7) / 8,
                        (((P.lafl - 1) / 2 + 1) - ((P.fafl + 1 - 1) / 2 - 8) + 7) / 8);
    const int per_frame = ntx * nty;
    const unsigned nitems = (unsigned)per_frame * (unsigned)(P.nout >> 1);
    const float wy = c2_wy[i];
    const int ky = rev4(i), kyr = (8 - ky) & 15;
    const int at = i ^ (i >> 2), atr = rev4(kyr) ^ (rev4(kyr) >> 2);   // positions of ky and its mirror
    unsigned n_exact = 0, n_flip = 0;
    for (unsigned item = blockIdx.x * kWarps2 + warp; item < nitems; item += gridDim.x * kWarps2) {
    const int o = 2 * (int)(item / per_frame) + j;   // this lane's field (nout is even: whole frames)
    const int t = (int)(item % per_frame);
    const int tx = t % ntx, ty = t / ntx;
    const int f = P.field_begin + o;
    const int off = (f & 1) ^ P.swap;   // SourceField::getOffset
    const int fl_first = (P.fafl + 1 - off) / 2;   // SourceField::getFirstActiveLine
    const int fl_last = ((P.lafl - off) / 2) + 1;  // SourceField::getLastActiveLine
    const int tileY = fl_first - 8 + 8 * ty;
    const int tileX = tileX0 + 16 * tx;
    const int cls = ((ty & 1) << 1) | (tx & 1);
    const int fl = tileY + i;
    const uint16_t *fp = (f >= 0 && f < P.nfields) ? field_at(P, f) : nullptr;
    const bool inside = fl >= fl_first && fl < fl_last;
    // a black gap frame of a batch: nothing reads its planes
    if (P.field_ptrs != nullptr && !__any_sync(0xffffffffu, fp != nullptr)) continue;

    // --- forward X: this lane's row, DC/black removed, folded about the window
    // centre: (s_x, d_x) = (a_x + a_31-x - 2 mean, a_x - a_31-x), exact in FP32
    float2 sd[16];
    float rowl1 = 0.f;
    if (fp != nullptr && inside) {
        uint32_t v[16];   // samples 2k, 2k+1
        if (tileX >= 0 && fl >= 1 && tileX + 40 <= (fl + 1 < P.fh ? 2 * P.fw : P.fw)) {
            // rows start on any 2-byte boundary: five aligned 16-byte vectors
            // cover the 32 samples, inside the field; they are lined up by
            // whole words, then by a half
            const uintptr_t pa = reinterpret_cast<uintptr_t>(fp + fl * P.fw + tileX);
            const uint4 *w4 = reinterpret_cast<const uint4 *>(pa & ~(uintptr_t)15);
            uint32_t w[20];
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const uint4 u = __ldg(w4 + k);
                w[4 * k] = u.x;
                w[4 * k + 1] = u.y;
                w[4 * k + 2] = u.z;
                w[4 * k + 3] = u.w;
            }
#pragma unroll
            for (int k = 0; k < 18; k++) w[k] = pa & 8 ? w[k + 2] : w[k];
#pragma unroll
            for (int k = 0; k < 17; k++) w[k] = pa & 4 ? w[k + 1] : w[k];
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = __funnelshift_r(w[k], w[k + 1], (unsigned)(pa & 2) * 8u);
        } else {
            // Never outside the field: a tile that hangs over the start of the
            // first line takes its first sample, one over the end of the last its last.
            const int at0 = fl * P.fw + tileX, end = P.fw * P.fh - 1;
#pragma unroll
            for (int k = 0; k < 16; k++)   // max(min(at, end), 0)
                v[k] = (uint32_t)__ldg(fp + __vimin_s32_relu(at0 + 2 * k, end)) |
                       ((uint32_t)__ldg(fp + __vimin_s32_relu(at0 + 2 * k + 1, end)) << 16);
        }
        // 2^23 + a from the sample's bits; subtracting 2^24 from one side of
        // each sum leaves a_x + a_31-x exactly
        float2 tt[8];
        float2 u = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 p = make_float2(__uint_as_float(__byte_perm(v[k], 0x4B000000u, 0x7610)),
                                         __uint_as_float(__byte_perm(v[k], 0x4B000000u, 0x7632)));
            const float2 q = make_float2(__uint_as_float(__byte_perm(v[15 - k], 0x4B000000u, 0x7632)),
                                         __uint_as_float(__byte_perm(v[15 - k], 0x4B000000u, 0x7610)));
            sd[2 * k].y = __fsub_rn(p.x, q.x);
            sd[2 * k + 1].y = __fsub_rn(p.y, q.y);
            tt[k] = add2(add2(p, make_float2(-16777216.f, -16777216.f)), q);
            u = add2(u, tt[k]);   // sums of 32 samples: exact
        }
        const float mean2 = __fmul_rn(__fadd_rn(u.x, u.y), 0.0625f);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            sd[2 * k].x = __fsub_rn(tt[k].x, mean2);
            sd[2 * k + 1].x = __fsub_rn(tt[k].y, mean2);
        }
        // |a_x - mean| + |a_31-x - mean| = max(|s_x|, |d_x|)
#pragma unroll
        for (int x = 0; x < 16; x++) rowl1 = __fmaf_rn(c2_wx[x], fmaxf(fabsf(sd[x].x), fabsf(sd[x].y)), rowl1);
    } else {
#pragma unroll
        for (int x = 0; x < 16; x++) sd[x] = make_float2(0.f, 0.f);
    }
    rowl1 *= wy;
#pragma unroll
    for (int m = 1; m < 16; m <<= 1) rowl1 += __shfl_xor_sync(0xffffffffu, rowl1, m);
    {
        // rows 8..15 write their imaginary part first: 32 different banks a store
        const bool upper = i >= 8;
        float *xr = reinterpret_cast<float *>(bx) + 4 * i + j;
        float *xs = xr + (upper ? 2 : 0), *xt = xr + (upper ? 0 : 2);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            float2 X = make_float2(0.f, 0.f);
#pragma unroll
            for (int x = 0; x < 16; x++) X = __ffma2_rn(c2_xf[k][x], sd[x], X);
            X = __fmul2_rn(X, make_float2(wy, wy));
            xs[80 * k] = upper ? X.y : X.x;
            xt[80 * k] = upper ? X.x : X.y;
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++)
        if (pass == 0 || lane < 4) {
            const int k = pass == 0 ? lane >> 2 : 8;
            y_forward2(bx + 20 * k, be + 20 * k, bx + 20 * k, reinterpret_cast<float2 *>(bnd) + k, s_tw, lane & 3,
                       pass == 0 ? 0xffffffffu : 0xFu);
        }
    __syncwarp();

    // --- decisions: lane (j, ky), bins A = (kx 4 + k, ky) and their mirrors
    // B = (kx 12 - k, kyr)
    const float *sa = reinterpret_cast<const float *>(bx + at) + j, *sr = reinterpret_cast<const float *>(bx + atr) + j;
    float2 A[5], B[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        A[k] = make_float2(sa[80 * k], sa[80 * k + 2]);
        B[k] = make_float2(sr[80 * (8 - k)], sr[80 * (8 - k) + 2]);
    }
    const float tf = (P.frame_t2 != nullptr) ? P.frame_t2[3 * (f >> 1)] : P.t2f;
    unsigned keep = 0, unc = 0;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const float Ea = kBound2 * kEps * (bnd[2 * k + j] + 0.5f * rowl1);
        const float Eb = kBound2 * kEps * (bnd[2 * (8 - k) + j] + 0.5f * rowl1);
        const bool self = (k == 4) && (ky == kyr);
        const float a = __fmaf_rn(A[k].x, A[k].x, __fmul_rn(A[k].y, A[k].y));
        const float b = __fmaf_rn(B[k].x, B[k].x, __fmul_rn(B[k].y, B[k].y));
        const float pa = 2.f * Ea * l1(A[k]) + Ea * Ea;
        const float pb = 2.f * Eb * l1(B[k]) + Eb * Eb;
        float tt = tf;
        if (PER_BIN) tt = thr2(P, f >> 1, ky, 4 + k).f;
        bool sm = sim2(a, b, tt);
        bool u = unc2(a, b, tt, pa, pb);
        if (PER_BIN && k == 4) {   // the mirror (also kx 8) visits with its own threshold
            const float t2 = thr2(P, f >> 1, kyr, 8).f;
            sm |= sim2(a, b, t2);
            u |= unc2(a, b, t2, pa, pb);
        }
        if (sm || self) keep |= 1u << k;
        if (u && !self) unc |= 1u << k;
    }
    unsigned any = __ballot_sync(0xffffffffu, unc != 0);
    while (any) {
        const int src = __ffs(any) - 1;
        const unsigned su = __shfl_sync(0xffffffffu, unc, src);
        const int k = __ffs(su) - 1;
        const int kyb = rev4(src & 15), kxb = 4 + k;
        const int fs = __shfl_sync(0xffffffffu, f, src), ys = __shfl_sync(0xffffffffu, tileY, src);
        const int first = __shfl_sync(0xffffffffu, fl_first, src), last = __shfl_sync(0xffffffffu, fl_last, src);
        df mb, mr;
        exact_pair2(P, fs, tileX, ys, first, last, kyb, kxb, mb, mr);
        const int kybr = (8 - kyb) & 15;
        bool sm = df_sim2(mb, mr, thr2(P, fs >> 1, kyb, kxb).d);
        if (kxb == 8) sm |= df_sim2(mb, mr, thr2(P, fs >> 1, kybr, 8).d);
        if (lane == src) {
            n_exact++;
            if ((((keep >> k) & 1u) != 0) != sm) n_flip++;
            keep = sm ? (keep | (1u << k)) : (keep & ~(1u << k));
            unc &= ~(1u << k);
        }
        if (kxb == 8 && lane == ((src & 16) | rev4(kybr))) {   // the kx-8 mirror is a visitor too
            keep = sm ? (keep | (1u << 4)) : (keep & ~(1u << 4));
            unc &= ~(1u << 4);
        }
        any = __ballot_sync(0xffffffffu, unc != 0);
    }
    // both bins of each pair, masked in place (kx 8's mirrors are other lanes' A)
    __syncwarp();
    {
        float *wa = reinterpret_cast<float *>(bx + at) + j, *wr = reinterpret_cast<float *>(bx + atr) + j;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const float m = ((keep >> k) & 1u) ? 1.f : 0.f;
            wa[80 * k] = A[k].x * m;
            wa[80 * k + 2] = A[k].y * m;
            if (k < 4) {
                wr[80 * (8 - k)] = B[k].x * m;
                wr[80 * (8 - k) + 2] = B[k].y * m;
            }
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++)
        if (pass == 0 || lane < 4) {
            const int k = pass == 0 ? lane >> 2 : 8;
            y_inverse2(bx + 20 * k, be + 20 * k, bx + 20 * k, s_tw, lane & 3, pass == 0 ? 0xffffffffu : 0xFu);
        }
    __syncwarp();

    // --- inverse X of this lane's row: kx 4..8 and kx 9..12 summed apart, then added
    if (inside) {
        float2 G[9];
        const float *gr = reinterpret_cast<const float *>(bx) + 4 * i + j;
#pragma unroll
        for (int k = 0; k < 9; k++) G[k] = make_float2(gr[80 * k], gr[80 * k + 2]);
        float v[32];
#pragma unroll
        for (int x = 0; x < 16; x++) {
            float2 c = make_float2(0.f, 0.f), d = c;
#pragma unroll
            for (int k = 0; k < 5; k++) c = __ffma2_rn(G[k], c2_xi[k][x], c);
#pragma unroll
            for (int k = 5; k < 9; k++) d = __ffma2_rn(G[k], c2_xi[k][x], d);
            c = add2(c, d);   // (cosine sum, sine sum)
            v[x] = c.x - c.y;
            v[31 - x] = c.x + c.y;
        }
        float *dst = P.partial + (long long)cls * P.part_class_stride + (long long)o * P.part_field_stride +
                     (long long)(fl - P.fl_lo) * P.part_row_stride - P.avs;
        // tileX - avs is a multiple of 16, so inside the active window each half
        // row starts on a 64-byte boundary whenever the planes' strides are
        // multiples of 4 floats and their base is 16-byte aligned: four vector
        // stores a half
        const bool vec = ((P.part_row_stride | P.part_field_stride | P.part_class_stride) & 3) == 0 &&
                         (reinterpret_cast<uintptr_t>(P.partial) & 15) == 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int x0 = tileX + 16 * h;
            if (vec && x0 >= P.avs && x0 + 16 <= P.ave) {
                float4 *d4 = reinterpret_cast<float4 *>(dst + x0);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    d4[q] = make_float4(v[16 * h + 4 * q], v[16 * h + 4 * q + 1], v[16 * h + 4 * q + 2], v[16 * h + 4 * q + 3]);
            } else {
#pragma unroll
                for (int x = 0; x < 16; x++)
                    if (x0 + x >= P.avs && x0 + x < P.ave) dst[x0 + x] = v[16 * h + x];
            }
        }
    }
    __syncwarp();   // the next item reuses the buffers
    }
    if (P.stats != nullptr) {
        if (n_exact) atomicAdd(P.stats + 0, n_exact);
        if (n_flip) atomicAdd(P.stats + 1, n_flip);
    }
}

static double rc_window2(int n, int N) { return 0.5 - (0.5 * cos((2 * M_PI * (n + 0.5)) / N)); }

static void split2(double v, float &hi, float &lo)
{
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

int tp2_init_constants(int device)
{
    if (device >= 0 && device < 64 && g_tp2_ready[device]) return 0;
    float cwx[9][16], swx[9][16], cix[9][16], six[9][16], wx[16], wy[16];
    for (int k = 0; k < 9; k++) {
        const int kx = 4 + k;
        for (int x = 0; x < 16; x++) {
            const double th = 2.0 * M_PI * kx * (x - 15.5) / 32.0;
            const double w = rc_window2(x, 32);
            cwx[k][x] = (float)(w * cos(th));
            swx[k][x] = (float)(w * sin(th));
            cix[k][x] = (float)((2.0 / 512.0) * cos(th));
            six[k][x] = (float)((2.0 / 512.0) * sin(th));
        }
    }
    for (int x = 0; x < 16; x++) wx[x] = (float)rc_window2(x, 32);
    for (int i = 0; i < 16; i++) wy[i] = (float)rc_window2(i, 16);
    float2 tw[16];
    for (int r = 0; r < 16; r++) tw[r] = make_float2((float)cos(-2 * M_PI * r / 16), (float)sin(-2 * M_PI * r / 16));
    float dfx[9][32][4], dfwy[16][2], dftw[16][4];
    for (int k = 0; k < 9; k++)
        for (int x = 0; x < 32; x++) {
            const double w = rc_window2(x, 32), a = -2.0 * M_PI * (4 + k) * x / 32.0;
            split2(w * cos(a), dfx[k][x][0], dfx[k][x][1]);
            split2(w * sin(a), dfx[k][x][2], dfx[k][x][3]);
        }
    for (int i = 0; i < 16; i++) split2(rc_window2(i, 16), dfwy[i][0], dfwy[i][1]);
    for (int r = 0; r < 16; r++) {
        split2(cos(-2 * M_PI * r / 16), dftw[r][0], dftw[r][1]);
        split2(sin(-2 * M_PI * r / 16), dftw[r][2], dftw[r][3]);
    }
#define TP2_CPY(sym, src) \
    if (cudaMemcpyToSymbol(sym, src, sizeof(src)) != cudaSuccess) return -1;
    float2 xf[9][16], xi[9][16];
    for (int k = 0; k < 9; k++)
        for (int x = 0; x < 16; x++) {
            xf[k][x] = make_float2(cwx[k][x], -swx[k][x]);
            xi[k][x] = make_float2(cix[k][x], six[k][x]);
        }
    TP2_CPY(c2_xf, xf);
    TP2_CPY(c2_xi, xi);
    TP2_CPY(c2_wx, wx);
    TP2_CPY(c2_wy, wy);
    TP2_CPY(c2_tw16, tw);
    TP2_CPY(c2_dfx, dfx);
    TP2_CPY(c2_dfwy, dfwy);
    TP2_CPY(c2_dftw16, dftw);
#undef TP2_CPY
    if (device >= 0 && device < 64) g_tp2_ready[device] = true;
    return 0;
}

int tp2_launch(const T2Params &P, cudaStream_t stream)
{
    const int tileX0 = P.avs - 16;
    const int ntx = (P.ave - tileX0 + 15) / 16;
    const int nty = std::max((((P.lafl - 0) / 2 + 1) - ((P.fafl + 1 - 0) / 2 - 8) + 7) / 8,
                             (((P.lafl - 1) / 2 + 1) - ((P.fafl + 1 - 1) / 2 - 8) + 7) / 8);
    const long long items = (long long)ntx * nty * (P.nout / 2);   // tile positions of whole frames
    if (items <= 0) return 0;
    // Resident blocks, each warp walking several items: 300 fields take 0.87 ms
    // (2.17 ms in the form before), 16 fields 62 us (125 us); 1,924 warp
    // instructions a pair of tiles (3,732), issue 62 % and the path of shared
    // memory and L1 70 % busy. Rows as 17 words instead of five vectors and the
    // twiddles' negatives from shared memory: 0.93 ms.
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned blocks = (unsigned)std::min<long long>((items + kWarps2 - 1) / kWarps2, (long long)kBlocks2 * std::max(sms, 1));
    if (P.thr_table != nullptr) tpal2d_kernel<true><<<blocks, 32 * kWarps2, 0, stream>>>(P);
    else tpal2d_kernel<false><<<blocks, 32 * kWarps2, 0, stream>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace tpal
