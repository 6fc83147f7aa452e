// demod.cu -- PALcolour demodulation of Transform-PAL chroma and on-device
// H.273 quantise/pack, sm_103a.
//
// Follows PalColour::decodeField / detectBurst / decodeLine<double, true>
// (src/decoders/palcolour/palcolour.cpp:307-409, 456-646) and
// OutputWriter::convertLine / convertToFloat
// (src/output/output_writer.cpp:402-486, 670-727), restructured:
//
//  * 4fsc sampling makes the reference carrier exact: sin(2 pi i fSC/fs) is
//    {0, 1, 0, -1}[i mod 4] (the reference's double tables differ only by
//    ~1e-16 residues at the zeros). The burst sums therefore run in exact
//    integer arithmetic, the V-switch test is an exact int64 comparison, and
//    each FIR tap touches either the sine or the cosine products, never both.
//  * The chroma input is the sum of the transform's four overlap-class planes;
//    chroma lines outside the field's active lines and samples outside the
//    active window are zero, exactly like the reference's zero-initialised
//    chroma buffer and its blackLine substitution (palcolour.cpp:466-473).
//  * Y = composite - chroma, the rotated U/V and the output scaling are fused;
//    planes are written straight into the frame's [Y | Cb | Cr] layout.
//
//  * CHD_DEC_PAL_2D (partial == NULL): the same 2D FIR runs on the composite
//    rows themselves (decodeLine<uint16_t, false>) and luma is the composite
//    minus the chroma the Y filter extracts, resynthesised on the carrier.
//  * luma_nr_level > 0: doYNR (palcolour.cpp:412-449) -- the 25-tap
//    high-pass of each line's luma, cored to +-nr_y and subtracted -- after a
//    pre-pass that puts the block's luma lines in shared memory.
//  * Every output format of the ABI is packed here: yuv444p16/ps, rgb48
//    (interleaved, truncating), rgbs, gray16, grays.
//
// One block: up to 16 field lines (8 with yNR) of one output field, 256
// threads; a work item produces 8 consecutive samples of one line from a
// register window of the four vertically combined chroma rows. Items start at
// the first active sample, so an item's samples are 8 aligned output pixels;
// XO, the carrier phase of that sample, is a template parameter.
//
// Measured on a 500-field capture against the kernel before it (items on the
// carrier phase, scalar FIR, run-time format): 1.85 -> 1.33 ms, 2,124 -> 1,395
// warp instructions per 32 items, 634 -> about 400 wavefronts; 160 fields of
// packed rgb48 with its border 1,465 -> 478 us. What bounds it now is the
// latency of the plane loads at the start of a block (two blocks of 8 warps a
// SM: 128 registers for the window). Four blocks of 8 lines (halo 1.75x),
// three of 10 or 14, two of 192 threads, L2 prefetches of the block 304 ahead
// and eight loads in flight a lane instead of four all measured slower.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "tpal_common.cuh"
#include "tpal_kernels.h"

namespace tpal {

__constant__ float cd_nrpal[25];     // doYNR high-pass (c_nrpal_b)
static bool g_demod_ready[64];

constexpr int kDemodThreads = 256;
constexpr int kLead = 8;                 // samples a row in shared memory starts before the first active one
constexpr int kNrHalf = 12;              // half length of the yNR filter
// Field lines per block: 16 (a 6-line halo re-read per 16 lines), 8 with
// yNR, whose luma lines also live in shared memory.
__host__ __device__ constexpr int demod_lines(bool ynr) { return ynr ? 8 : 16; }

__device__ __forceinline__ int first_line(int fafl, int off) { return (fafl + 1 - off) / 2; }
__device__ __forceinline__ int last_line(int lafl, int off) { return ((lafl - off) / 2) + 1; }

// Shared rows: samples avs - 8 .. avs + 8 n + 7 for n items, in 16-byte chunks;
// chunk c is stored at c ^ ((c >> 3) & 1), which spreads the chunks of
// consecutive items (2 apart) over all banks. The row length keeps the pattern
// the same in every row.
__host__ __device__ __forceinline__ int demod_items(int avs, int ave) { return (ave - avs + 7) / 8; }
__host__ __device__ __forceinline__ int demod_row(int avs, int ave) { return (8 * demod_items(avs, ave) + 2 * kLead + 63) & ~63; }
__device__ __forceinline__ int chunk_at(int c) { return c ^ ((c >> 3) & 1); }
__device__ __forceinline__ int float_at(int i) { return 4 * chunk_at(i >> 2) + (i & 3); }

// 4fsc reference carrier at sample x: sine {0, 1, 0, -1}, cosine {1, 0, -1, 0}.
__device__ __forceinline__ float carrier_sin(int x) { return (x & 1) ? ((x & 2) ? -1.f : 1.f) : 0.f; }
__device__ __forceinline__ float carrier_cos(int x) { return (x & 1) ? 0.f : ((x & 2) ? -1.f : 1.f); }

// The vertical combinations (palcolour.cpp:557-567 without the carrier) of 22
// columns, sample s of the item at column s + 7:
//   v0 = c0, v1 = -c(-2) - c(+2), v2 = c(-1) - c(+1), v3 = -c(-3) + c(+3)
// as the pairs (v0, v2) and (v1, v3) for the f32x2 instructions.
struct Window {
    float2 v02[22], v13[22];
};

// Chunks N0 .. N1 - 1 of the six an item's window spans. ch: the row three
// lines above the item's; the item's first chunk is 2 seg. Samples 0..3 need
// chunks 0..4 only.
template <int N0, int N1>
__device__ __forceinline__ void load_window(const float *ch, int row_floats, int seg, Window &W)
{
#pragma unroll
    for (int n = N0; n < N1; n++) {
        const float *p = ch + 4 * chunk_at(2 * seg + n);
        float4 r[7];
#pragma unroll
        for (int k = 0; k < 7; k++) r[k] = *reinterpret_cast<const float4 *>(p + k * row_floats);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int q = 4 * n + i - 1;
            if (q < 0 || q >= 22) continue;
            auto at = [&](int k) { return i == 0 ? r[k].x : i == 1 ? r[k].y : i == 2 ? r[k].z : r[k].w; };
            W.v02[q] = make_float2(at(3), at(2) - at(4));
            W.v13[q] = make_float2(-at(1) - at(5), -at(0) + at(6));
        }
    }
}

// The 2D FIR at sample s of an item: (PU, QU, PV, QV), and (PY, QY) from the
// luma taps with WITH_Y. Taps b = 0..7 of the launch's filter (a filter of
// size 6, at PAL-M's sample rate, has zero taps at b = 7). Each tap touches
// either the sine or the cosine products. swap: the reference's PAL-M tables
// (sine and cosine exchanged at fieldHeight 263, palcolour.cpp:158-173) make
// each P sum the other table's Q sum and vice versa: (PU, QU, PV, QV)
// become (QV, PV, QU, PU); the luma resynthesis is unchanged.
template <int N>
struct Num {
    static constexpr int value = N;
};
struct FirOut {
    float PU, QU, PV, QV, PY, QY;
};

template <int XO, int S, bool CHROMA, bool WITH_Y>
__device__ __forceinline__ FirOut fir(const DemodParams &P, const Window &W)
{
    float2 Pab = make_float2(0.f, 0.f), Qab = Pab;   // (A, B): the v0, v1 and the v2, v3 parts
    float PY = 0.f, QY = 0.f;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const int r = S + b + 7, l = S - b + 7, phase = (S + XO + b) & 3;
        float2 s02, s13;
        if (CHROMA) {
            s02 = (b & 1) ? sub2(W.v02[r], W.v02[l]) : add2(W.v02[r], W.v02[l]);
            s13 = (b & 1) ? sub2(W.v13[r], W.v13[l]) : add2(W.v13[r], W.v13[l]);
            const float2 ab = __ffma2_rn(make_float2(P.cfilt[b][2], P.cfilt[b][3]), s13,
                                         __fmul2_rn(make_float2(P.cfilt[b][0], P.cfilt[b][1]), s02));
            if (phase == 1) Pab = add2(Pab, ab);
            if (phase == 3) Pab = sub2(Pab, ab);
            if (phase == 0) Qab = add2(Qab, ab);
            if (phase == 2) Qab = sub2(Qab, ab);
        } else {
            s02.x = (b & 1) ? W.v02[r].x - W.v02[l].x : W.v02[r].x + W.v02[l].x;
            s13.x = (b & 1) ? W.v13[r].x - W.v13[l].x : W.v13[r].x + W.v13[l].x;
        }
        if (WITH_Y) {
            const float y = __fmaf_rn(P.yfilt[b][1], s13.x, P.yfilt[b][0] * s02.x);
            if (phase == 1) PY += y;
            if (phase == 3) PY -= y;
            if (phase == 0) QY += y;
            if (phase == 2) QY -= y;
        }
    }
    FirOut o;
    o.PY = PY;
    o.QY = QY;
    if (P.swap_carrier) {
        o.PU = Qab.x + Pab.y;
        o.PV = Qab.x - Pab.y;
        o.QU = Pab.x - Qab.y;
        o.QV = Pab.x + Qab.y;
    } else {
        o.PU = Pab.x + Qab.y;
        o.PV = Pab.x - Qab.y;
        o.QU = Qab.x - Pab.y;
        o.QV = Qab.x + Pab.y;
    }
    return o;
}

// 4 samples of a composite row, at any 2-byte boundary, as floats: three
// aligned words and a funnel shift, the bits 2^23 + a, less `off` + 2^23
// (exact). first: the first sample's index within the field.
__device__ __forceinline__ void samples4(const uint16_t *field, int first, int field_len, float off, float (&v)[4])
{
    const float bias = 8388608.0f + off;
    if (first >= 1 && first + 6 <= field_len) {
        const uintptr_t pa = reinterpret_cast<uintptr_t>(field + first);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(pa & ~(uintptr_t)3);
        const unsigned sh = (unsigned)(pa & 2) * 8u;
        const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
        const uint32_t a = __funnelshift_r(w0, w1, sh), b = __funnelshift_r(w1, w2, sh);
        v[0] = __uint_as_float(__byte_perm(a, 0x4B000000u, 0x7610)) - bias;
        v[1] = __uint_as_float(__byte_perm(a, 0x4B000000u, 0x7632)) - bias;
        v[2] = __uint_as_float(__byte_perm(b, 0x4B000000u, 0x7610)) - bias;
        v[3] = __uint_as_float(__byte_perm(b, 0x4B000000u, 0x7632)) - bias;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = (float)__ldg(field + min(max(first + i, 0), field_len - 1)) - off;
    }
}

// An integer-format code (H.273 Round(x) = Sign(x) * Floor(Abs(x) + 0.5),
// then the clamp, output_writer.cpp:52-76), zero + Round(v * (k_hi + k_lo)) for v = v_hi + v_lo,
// without FP32 rounding at the code's magnitude: the product is formed as
// p + e (p = v_hi k_hi rounded, e its error and the low-order terms), the
// nearest integer n of p split off exactly, and only the remainder
// (p - n) + e, below one in magnitude, rounded. zero is an integer, so
// zero + n + Floor(r + 1/2) is H.273's Round of the whole sum wherever that
// sum is non-negative; below zero both clamp to the bound lo >= 0. Returns
// the clamped code plus 2^23, exact, so the code is the low half of its bits
// (conversions run on a quarter-rate pipe; rounding to the nearest integer is
// the addition of 3 * 2^22, exact for |p| below 2^22 -- beyond the code's range
// by a factor of 64 -- and clamped to it).
constexpr float kCode0 = 8388608.0f;
__device__ __forceinline__ float code_of(float zero, float v_hi, float v_lo, float k_hi, float k_lo, float lo, float hi)
{
    const float p = fminf(fmaxf(v_hi * k_hi, -4194304.0f), 4194303.0f);
    const float e = __fmaf_rn(v_hi, k_hi, -p) + __fmaf_rn(v_hi, k_lo, v_lo * k_hi);
    const float n = __fsub_rn(__fadd_rn(p, 12582912.0f), 12582912.0f);
    const float r = (p - n) + e;   // p - n is exact
    return fminf(fmaxf((kCode0 + zero) + n + floorf(r + 0.5f), kCode0 + lo), kCode0 + hi);
}
__device__ __forceinline__ uint32_t code_pair(float a, float b)
{
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x5410);
}

// One sample's outputs in the units its format stores: the codes of code_of
// (yuv444p16, gray16), 0..65535 before truncation (rgb48) or the float value.
// OutputWriter::convertLine, convertToFloat, convertToFloatRGB
// (output_writer.cpp:402-486, 670-779). Luma arrives as Y - black = yb.hi +
// yb.lo (exact for the Transform kinds: an integer composite sample minus the
// FP32 chroma, by two-sum).
__device__ __forceinline__ float luma_value(const DemodParams &P, int format, df yb)
{
    if (format == 0 || format == 4)
        return code_of(16.0f * 256.0f, yb.hi, yb.lo, P.qy_hi, P.qy_lo, P.y_lo, P.y_hi);
    return fminf(fmaxf((yb.hi + yb.lo) * P.ey_scale, P.y_lo), P.y_hi);
}
__device__ __forceinline__ void chroma_values(const DemodParams &P, int format, float U, float V, float &o1, float &o2)
{
    if (format == 0) {
        o1 = code_of(128.0f * 256.0f, U, 0.f, P.qcb_hi, P.qcb_lo, P.c_lo, P.c_hi);
        o2 = code_of(128.0f * 256.0f, V, 0.f, P.qcr_hi, P.qcr_lo, P.c_lo, P.c_hi);
    } else {
        o1 = fminf(fmaxf(U * P.ecb_scale, P.c_lo), P.c_hi);
        o2 = fminf(fmaxf(V * P.ecr_scale, P.c_lo), P.c_hi);
    }
}
__device__ __forceinline__ void rgb_values(const DemodParams &P, int format, df yb, float U, float V, float &o0,
                                           float &o1, float &o2)
{
    const float rU = U * P.rgb_uv_scale, rV = V * P.rgb_uv_scale;
    if (format == 2) {
        const float rY = fminf(fmaxf((yb.hi + yb.lo) * P.rgb_y_scale, 0.f), 65535.f);
        o0 = fminf(fmaxf(__fmaf_rn(P.r_from_v, rV, rY), 0.f), 65535.f);
        o1 = fminf(fmaxf(__fmaf_rn(P.g_from_v, rV, __fmaf_rn(P.g_from_u, rU, rY)), 0.f), 65535.f);
        o2 = fminf(fmaxf(__fmaf_rn(P.b_from_u, rU, rY), 0.f), 65535.f);
    } else {
        const float ey = (yb.hi + yb.lo) * P.ey_scale;
        o0 = fminf(fmaxf(__fmaf_rn(P.r_from_v, rV, ey), P.r_lo), P.r_hi);
        o1 = fminf(fmaxf(__fmaf_rn(P.g_from_v, rV, __fmaf_rn(P.g_from_u, rU, ey)), P.g_lo), P.g_hi);
        o2 = fminf(fmaxf(__fmaf_rn(P.b_from_u, rU, ey), P.b_lo), P.b_hi);
    }
}

// 4 consecutive outputs of one plane at element e, `n` of them inside the
// picture; align: the elements by which every such e is aligned (4, 2 or 1).
__device__ __forceinline__ void store4(bool wide, void *out, long long e, int n, int align, const float (&a)[4])
{
    if (wide) {   // FP32 planes
        float *o = (float *)out + e;
        if (n == 4 && align == 4) {
            *reinterpret_cast<float4 *>(o) = make_float4(a[0], a[1], a[2], a[3]);
        } else if (n == 4 && align == 2) {
            reinterpret_cast<float2 *>(o)[0] = make_float2(a[0], a[1]);
            reinterpret_cast<float2 *>(o)[1] = make_float2(a[2], a[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i < n) o[i] = a[i];
        }
    } else {
        uint16_t *o = (uint16_t *)out + e;
        const uint32_t p0 = code_pair(a[0], a[1]), p1 = code_pair(a[2], a[3]);
        if (n == 4 && align == 4) {
            *reinterpret_cast<uint2 *>(o) = make_uint2(p0, p1);
        } else if (n == 4 && align == 2) {
            reinterpret_cast<uint32_t *>(o)[0] = p0;
            reinterpret_cast<uint32_t *>(o)[1] = p1;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i < n) o[i] = (uint16_t)__float_as_uint(a[i]);
        }
    }
}

// 4 pixels of interleaved R'G'B' (truncating) at pixel pix, the same rules
__device__ __forceinline__ void store_rgb48(void *out, long long e, int n, int align, const float (&r)[4],
                                            const float (&g)[4], const float (&b)[4])
{
    uint16_t *o = (uint16_t *)out + e;
    uint32_t c[12];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c[3 * i] = __float2uint_rz(r[i]);
        c[3 * i + 1] = __float2uint_rz(g[i]);
        c[3 * i + 2] = __float2uint_rz(b[i]);
    }
    if (n == 4 && align >= 2) {
        uint32_t w[6];
#pragma unroll
        for (int i = 0; i < 6; i++) w[i] = c[2 * i] | (c[2 * i + 1] << 16);
        if (align == 4) {
#pragma unroll
            for (int i = 0; i < 3; i++) reinterpret_cast<uint2 *>(o)[i] = make_uint2(w[2 * i], w[2 * i + 1]);
        } else {
#pragma unroll
            for (int i = 0; i < 6; i++) reinterpret_cast<uint32_t *>(o)[i] = w[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < 12; i++)
            if (i < 3 * n) o[i] = (uint16_t)c[i];
    }
}

// Double-float pieces of the burst normalisation (FP64 is scarce on this
// GPU and one lane per line waiting on it stalls the block).
__device__ __forceinline__ df two_prod(float a, float b)
{
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

// max(sqrt(pn^2 + qn^2), floor), the square root refined by one Newton step
__device__ __forceinline__ df burst_norm(float pn, float qn, float floor_v)
{
    const df s = df_add(two_prod(pn, pn), two_prod(qn, qn));
    df r = df_make(0.f);
    if (s.hi > 0.f) {
        const float x = __fsqrt_rn(s.hi);
        const df d = df_sub(s, two_prod(x, x));
        r = quick_two_sum(x, __fdiv_rn(d.hi, 2.0f * x));
    }
    if (r.hi > floor_v || (r.hi == floor_v && r.lo > 0.f)) return r;
    return df_make(floor_v);
}

// a / d for an exact float a
__device__ __forceinline__ df df_div_f(float a, df d)
{
    const float q1 = __fdiv_rn(a, d.hi);
    const df r = df_sub(df_sub(df_make(a), two_prod(q1, d.hi)), df_make(q1 * d.lo));
    return quick_two_sum(q1, __fdiv_rn(r.hi, d.hi));
}

__device__ __forceinline__ float df_round(df v) { return __fadd_rn(v.hi, v.lo); }

// FMT: the output format as a constant (yuv444p16 0, yuv444ps 1, rgb48 2, rgbs
// 3), or -1: the launch's, any. With the format known the item loop has no branches and half
// the code (instruction fetch stalled it).
template <int XO, int FMT, bool COMPOSITE, bool YNR>
__global__ void __launch_bounds__(kDemodThreads, 2) demod_kernel(const __grid_constant__ DemodParams P)
{
    const int format = FMT >= 0 ? FMT : P.format;
    extern __shared__ float4 smem4[];
    constexpr int kMaxLines = demod_lines(YNR);
    const int lines = P.lines;                        // field lines of a block, at most kMaxLines
    const int o = blockIdx.x / P.blocks_per_field;
    const int blk = blockIdx.x % P.blocks_per_field;
    const int f = P.field_begin + o;
    const int off = (f & 1) ^ P.swap;   // SourceField::getOffset
    const int fl_first = first_line(P.fafl, off);
    const int fl_last = last_line(P.lafl, off);
    const int fl0 = fl_first + blk * lines;
    if (fl0 >= fl_last) return;

    const int cols = P.ave - P.avs;
    const int items = demod_items(P.avs, P.ave);      // per line
    const int SW = demod_row(P.avs, P.ave);           // floats per shared row
    const int YW = 8 * items + 2 * kNrHalf;           // luma line length (yNR)
    const int rows = lines + 6;                       // input lines fl0-3 .. fl0+lines+2
    float *ch = reinterpret_cast<float *>(smem4);     // [rows][SW]
    float *ys = ch + rows * SW;                       // [lines][YW] luma before coring (yNR only)
    __shared__ float s_bp[kMaxLines], s_bq[kMaxLines], s_vsw[kMaxLines];

    // where this field's frame goes: the frame slot of the output array, or
    // (batches of captures) the frame's own pointer, absent for the black
    // gap frames between captures
    void *out_base = P.out;
    long long frame_slot = o >> 1;   // field_begin is even: fields 2k, 2k+1 form frame k
    if (P.frame_out != nullptr) {
        out_base = P.frame_out[f >> 1];
        frame_slot = 0;
        if (out_base == nullptr) return;
    }
    const uint16_t *field = field_at(P, f);
    if (field == nullptr) return;   // a black batch gap: nothing to write
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kDemodThreads / 32;
    const int field_len = P.fw * P.fh;

    // 1. input rows, zero outside the field's active lines: the summed
    //    overlap-class chroma planes (zero outside the active window, the
    //    reference's zero-initialised chroma buffer), or the composite
    //    itself for the PALcolour filter (blackLine = 0, palcolour.cpp:466-473).
    const bool vec = !COMPOSITE && ((cols | P.part_row_stride) & 3) == 0 &&
                     ((P.part_class_stride | P.part_field_stride) & 3) == 0;
    const int chunks = 2 * items + 4;
    for (int r = warp; r < rows; r += kWarps) {
        const int fl = fl0 - 3 + r;
        float4 *dst = reinterpret_cast<float4 *>(ch + r * SW);
        if (fl < fl_first || fl >= fl_last) {
            for (int c = lane; c < chunks; c += 32) dst[chunk_at(c)] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else if (COMPOSITE) {
            for (int c = lane; c < chunks; c += 32) {
                const int x = P.avs - kLead + 4 * c;
                float v[4];
                samples4(field, fl * P.fw + x, field_len, 0.f, v);
                if (x < 0 || x + 4 > P.fw)
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (x + i < 0 || x + i >= P.fw) v[i] = 0.f;
                dst[chunk_at(c)] = make_float4(v[0], v[1], v[2], v[3]);
            }
        } else if (vec) {
            const int c4 = cols >> 2;
            const long long cs4 = P.part_class_stride >> 2;
            const float4 *src = reinterpret_cast<const float4 *>(P.partial + (long long)o * P.part_field_stride +
                                                                 (long long)(fl - P.fl_lo) * P.part_row_stride);
            if (lane < 2) dst[chunk_at(lane)] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < chunks - 2 - c4) dst[chunk_at(2 + c4 + lane)] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int q = lane; q < c4; q += 32) {
                const float4 a = __ldg(src + q), b = __ldg(src + cs4 + q), c = __ldg(src + 2 * cs4 + q),
                             d = __ldg(src + 3 * cs4 + q);
                dst[chunk_at(2 + q)] = make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y),
                                                   (a.z + b.z) + (c.z + d.z), (a.w + b.w) + (c.w + d.w));
            }
        } else {
            const float *src = P.partial + (long long)o * P.part_field_stride +
                               (long long)(fl - P.fl_lo) * P.part_row_stride - kLead;
            for (int i = lane; i < 4 * chunks; i += 32) {
                float v = 0.f;
                if (i >= kLead && i < kLead + cols)
                    for (int k = 0; k < P.nclasses; k++) v += src[(long long)k * P.part_class_stride + i];
                ch[r * SW + float_at(i)] = v;
            }
        }
    }
    if (YNR)
        for (int idx = threadIdx.x; idx < lines * YW; idx += blockDim.x) ys[idx] = 0.f;

    // 2. burst detection: one warp per line (detectBurst, palcolour.cpp:344-409).
    //    The window is the caller's (a capture's metadata): only what it has
    //    of the line is read, at most 1,135 samples of at most 2^18, whose sums
    //    fit 32 bits.
    const bool gray = format >= 4;
    const int burst0 = max(P.burst_start, 0), burst1 = min(P.burst_end, P.fw);
    if (!gray)
    for (int ln = warp; ln < lines; ln += kWarps) {
        const int fl = fl0 + ln;
        if (fl >= fl_last) continue;
        int Ps = 0, Qs = 0, POs = 0, QOs = 0;
        auto px = [&](int line, int i) -> int {
            return (line < 0 || line >= P.fh) ? 0 : (int)__ldg(field + line * P.fw + i);
        };
        for (int i = burst0 + lane; i < burst1; i += 32) {
            const int d = 2 * px(fl, i) - px(fl - 2, i) - px(fl + 2, i);   // 4 * ((in0 - (in3+in4)/2) / 2)
            const int e = px(fl + 1, i) - px(fl - 1, i);                   // 2 * ((in2 - in1) / 2)
            switch (i & 3) {
            case 0: Qs += d; QOs += e; break;    // cosine +1
            case 1: Ps += d; POs += e; break;    // sine +1
            case 2: Qs -= d; QOs -= e; break;    // cosine -1
            default: Ps -= d; POs -= e; break;   // sine -1
            }
        }
        Ps = __reduce_add_sync(0xffffffffu, Ps);
        Qs = __reduce_add_sync(0xffffffffu, Qs);
        POs = __reduce_add_sync(0xffffffffu, POs);
        QOs = __reduce_add_sync(0xffffffffu, QOs);
        if (P.swap_carrier) {   // the PAL-M tables: the sine sums are the cosine sums and vice versa
            const int t0 = Ps, t1 = POs;
            Ps = Qs;
            Qs = t0;
            POs = QOs;
            QOs = t1;
        }
        if (lane == 0) {
            // bp = P/(4 len), bpo = PO/(2 len): the V-switch test scaled by (4 len)^2
            const long long a = (long long)Ps - 2 * (long long)POs, b = (long long)Qs - 2 * (long long)QOs;
            const bool vpos = (a * a + b * b) < 2 * ((long long)Ps * Ps + (long long)Qs * Qs);
            // bp / max(|(bp, bq)|, 130000/128) with bp = pn / (8 len): the
            // 8 len cancels, leaving pn / max(|(pn, qn)|, 8 len 130000/128).
            // pn, qn are integers below 2^23 (exact in FP32); the rest runs
            // in double-float (about 2^-46), so the rounded results are the
            // double computation's.
            const float pn = (float)((long long)Ps - 2 * (long long)QOs), qn = (float)((long long)Qs + 2 * (long long)POs);
            const df n = burst_norm(pn, qn, 8.0f * (float)(P.burst_end - P.burst_start) * (130000.0f / 128.0f));
            const df nbp = df_div_f(pn, n), nbq = df_div_f(qn, n);
            s_bp[ln] = df_round(df_sub(df_mul_f(nbp, P.gain_cos), df_mul_f(nbq, P.gain_sin)));
            s_bq[ln] = df_round(df_add(df_mul_f(nbp, P.gain_sin), df_mul_f(nbq, P.gain_cos)));
            s_vsw[ln] = vpos ? 1.f : -1.f;
        }
    }
    __syncthreads();

    // 3. yNR pre-pass: the block's luma lines (zero outside the active window)
    if (YNR) {
        for (int item = threadIdx.x; item < lines * items; item += blockDim.x) {
            const int t = item / items, seg = item % items;
            const int fl = fl0 + t;
            if (fl >= fl_last) continue;
            float cv[8], Yv[8];
            samples4(field, fl * P.fw + P.avs + 8 * seg, field_len, 0.f, reinterpret_cast<float(&)[4]>(cv[0]));
            samples4(field, fl * P.fw + P.avs + 8 * seg + 4, field_len, 0.f, reinterpret_cast<float(&)[4]>(cv[4]));
            if (COMPOSITE) {
                Window W;
                load_window<0, 6>(ch + t * SW, SW, seg, W);
                auto luma = [&](auto S) {
                    constexpr int s = decltype(S)::value;
                    const FirOut q = fir<XO, s, false, true>(P, W);
                    Yv[s] = cv[s] - 2.0f * __fmaf_rn(q.PY, carrier_sin(s + XO), q.QY * carrier_cos(s + XO));
                };
                luma(Num<0>{}), luma(Num<1>{}), luma(Num<2>{}), luma(Num<3>{});
                luma(Num<4>{}), luma(Num<5>{}), luma(Num<6>{}), luma(Num<7>{});
            } else {
#pragma unroll
                for (int s = 0; s < 8; s++) Yv[s] = cv[s] - ch[(t + 3) * SW + float_at(kLead + 8 * seg + s)];
            }
#pragma unroll
            for (int s = 0; s < 8; s++)
                if (8 * seg + s < cols) ys[t * YW + kNrHalf + 8 * seg + s] = Yv[s];
        }
        __syncthreads();
    }

    // 4. 2D FIR + rotation + pack; work item = (line, 8-sample segment), 4
    // pixels stored at a time: vectors where the output's rows, planes and
    // frames allow, else element by element.
    const bool wide = format == 1 || format == 3 || format == 5;
    const long long plane = (long long)P.out_w * P.out_h;
    int align = 4;
    {
        const int elem = wide ? 4 : 2;
        const uintptr_t u = reinterpret_cast<uintptr_t>(out_base);
        const long long units = format == 2 ? P.out_frame_stride / 3 : P.out_frame_stride;
        const long long all = P.out_w | P.left_pad | units | plane;
        if ((all & 3) != 0 || u % (4 * elem) != 0) align = 2;
        if ((all & 1) != 0 || u % (2 * elem) != 0) align = 1;
    }
    int t = threadIdx.x / items, seg = threadIdx.x % items;
    const int dt = kDemodThreads / items, dseg = kDemodThreads % items;
    for (int item = threadIdx.x; item < lines * items;
         item += kDemodThreads, t += dt, seg += dseg, t += seg >= items, seg -= seg >= items ? items : 0) {
        const int fl = fl0 + t;
        if (fl >= fl_last) break;
        // the composite samples luma needs, less black, loaded before the FIR
        // so their latency hides behind it
        float cb[8];
        if (!YNR) {
            samples4(field, fl * P.fw + P.avs + 8 * seg, field_len, (float)P.black, reinterpret_cast<float(&)[4]>(cb[0]));
            samples4(field, fl * P.fw + P.avs + 8 * seg + 4, field_len, (float)P.black, reinterpret_cast<float(&)[4]>(cb[4]));
        }
        const int orow = P.top_pad + 2 * fl + off - P.fafl;
        const long long pix = (long long)orow * P.out_w + P.left_pad + 8 * seg;
        const long long e0 = frame_slot * P.out_frame_stride + (format == 2 ? 3 * pix : pix);
        // Y - black of sample s
        auto luma = [&](int s, float v0, float PY, float QY) -> df {
            if (YNR) {
                // doYNR: a = sum_i b_i Y[x + 12 - i], cored to +-nr_y, subtracted
                const float *yl = ys + t * YW + kNrHalf + 8 * seg + s;
                float a = 0.f;
#pragma unroll
                for (int i = 0; i < 25; i++) a = __fmaf_rn(cd_nrpal[i], yl[kNrHalf - i], a);
                a = fminf(fmaxf(a, -P.nr_y), P.nr_y);
                return two_sum(yl[0] - (float)P.black, -a);
            }
            if (COMPOSITE)
                return two_sum(cb[s], -2.0f * __fmaf_rn(PY, carrier_sin(s + XO), QY * carrier_cos(s + XO)));
            return two_sum(cb[s], -v0);
        };
        constexpr bool kLumaFir = COMPOSITE && !YNR;   // luma needs the window
        if (gray && !kLumaFir) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int n = min(4, cols - 8 * seg - 4 * h);
                if (n <= 0) break;
                float y[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    y[i] = luma_value(P, format, luma(4 * h + i, YNR ? 0.f : ch[(t + 3) * SW + float_at(kLead + 8 * seg + 4 * h + i)], 0.f, 0.f));
                store4(wide, out_base, e0 + 4 * h, n, align, y);
            }
            continue;
        }
        Window W;
        load_window<0, 5>(ch + t * SW, SW, seg, W);
        const float bp = gray ? 0.f : s_bp[t], bq = gray ? 0.f : s_bq[t], vsw = gray ? 1.f : s_vsw[t];
        auto half = [&](auto H) {
            constexpr int h = decltype(H)::value;
            const int n = min(4, cols - 8 * seg - 4 * h);
            if (n <= 0) return;
            float o0[4], o1[4], o2[4];
            auto sample = [&](auto I) {
                constexpr int i = decltype(I)::value, s = 4 * h + i;
                const FirOut q = fir<XO, s, true, kLumaFir>(P, W);
                const df yb = luma(s, W.v02[s + 7].x, q.PY, q.QY);
                const float U = -(q.PU * bp + q.QU * bq) * 2.0f;
                const float V = vsw * -(q.QV * bp - q.PV * bq) * 2.0f;
                if (format == 2 || format == 3) {
                    rgb_values(P, format, yb, U, V, o0[i], o1[i], o2[i]);
                } else {
                    o0[i] = luma_value(P, format, yb);
                    chroma_values(P, format, U, V, o1[i], o2[i]);
                }
            };
            sample(Num<0>{}), sample(Num<1>{}), sample(Num<2>{}), sample(Num<3>{});
            if (format == 2) {
                store_rgb48(out_base, e0 + 12 * h, n, align, o0, o1, o2);
            } else {
                const long long e = e0 + 4 * h;
                store4(wide, out_base, e, n, align, o0);
                if (!gray) {
                    store4(wide, out_base, e + plane, n, align, o1);
                    store4(wide, out_base, e + 2 * plane, n, align, o2);
                }
            }
        };
        half(Num<0>{});
        load_window<5, 6>(ch + t * SW, SW, seg, W);
        half(Num<1>{});
    }
}

// PalColour::buildLookUpTables chroma taps (palcolour.cpp:197-276), in double,
// for the sample rate; -2 when the filter is longer than the kernel's 8 taps.
int demod_taps(double sample_rate, float (&cfilt)[8][4], float (&yfilt)[8][2])
{
    const double chromaBandwidthHz = 1100000.0 / 0.93;
    const double ca = 0.5 * sample_rate / chromaBandwidthHz;
    int fs = 1;
    if ((int)ca > fs) fs = (int)ca;
    if (fs > 7) return -2;
    double cf[8][4] = {}, yf[8][2] = {};
    double cdiv = 0, ydiv = 0;
    for (int f = 0; f <= fs; f++) {
        const double fc = std::min(ca, (double)f);
        const double ff = std::min(ca, sqrt((double)(f * f + 4)));
        const double fff = std::min(ca, sqrt((double)(f * f + 16)));
        const double ffff = std::min(ca, sqrt((double)(f * f + 36)));
        const int d = (f == 0) ? 2 : 1;
        cf[f][0] = (1 + cos(M_PI * fc / ca)) / d;
        cf[f][2] = (1 + cos(M_PI * ff / ca)) / d;
        cf[f][1] = (1 + cos(M_PI * fff / ca)) / d;
        cf[f][3] = (1 + cos(M_PI * ffff / ca)) / d;
        cdiv += 2 * (1 * cf[f][0] + 2 * cf[f][2] + 2 * cf[f][1] + 2 * cf[f][3]);
        // luma-extraction taps (ya = ca at this bandwidth)
        const double fy = std::min(ca, (double)f);
        const double fffy = std::min(ca, sqrt((double)(f * f + 16)));
        yf[f][0] = (1 + cos(M_PI * fy / ca)) / d;
        yf[f][1] = 0.2 * (1 + cos(M_PI * fffy / ca)) / d;
        ydiv += 2 * (1 * yf[f][0] + 2 * yf[f][1]);
    }
    for (int f = 0; f < 8; f++) {
        static const int order[4] = {0, 2, 1, 3};
        for (int i = 0; i < 4; i++) cfilt[f][i] = (float)(cf[f][order[i]] / cdiv);
        for (int i = 0; i < 2; i++) yfilt[f][i] = (float)(yf[f][i] / ydiv);
    }
    return 0;
}

// The doYNR high-pass, once per device.
int demod_init_constants(int device)
{
    if (device >= 0 && device < 64 && g_demod_ready[device]) return 0;
    // c_nrpal_b, src/decoders/filter/deemp.h:620-628
    static const double nrpal[25] = {
        1.141291975113614e-04, -1.857019211291029e-03, -4.499636864042073e-03, -5.577680979937061e-03,
        -4.423694440267179e-04, 1.309163063177155e-02, 2.861211356202848e-02, 3.029931283148555e-02,
        1.098965697652802e-03, -6.398130386469833e-02, -1.492080690537196e-01, -2.223459379380252e-01,
        7.479077367478024e-01, -2.223459379380252e-01, -1.492080690537196e-01, -6.398130386469833e-02,
        1.098965697652803e-03, 3.029931283148557e-02, 2.861211356202848e-02, 1.309163063177156e-02,
        -4.423694440267185e-04, -5.577680979937061e-03, -4.499636864042074e-03, -1.857019211291030e-03,
        1.141291975113614e-04};
    float nrf[25];
    for (int i = 0; i < 25; i++) nrf[i] = (float)nrpal[i];
    if (cudaMemcpyToSymbol(cd_nrpal, nrf, sizeof(nrf)) != cudaSuccess) return -1;
    if (device >= 0 && device < 64) g_demod_ready[device] = true;
    return 0;
}

static size_t demod_smem_bytes(int avs, int ave, int lines, bool ynr)
{
    const size_t rows = sizeof(float) * (size_t)(lines + 6) * demod_row(avs, ave);
    return rows + (ynr ? sizeof(float) * (size_t)lines * (8 * demod_items(avs, ave) + 2 * kNrHalf) : 0);
}

template <int XO, int FMT, bool COMPOSITE, bool YNR>
static int demod_start(const DemodParams &P, unsigned blocks, size_t smem, cudaStream_t stream)
{
    // function attributes are per device
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -1;
    if (!attr_set[dev]) {
        if (cudaFuncSetAttribute(demod_kernel<XO, FMT, COMPOSITE, YNR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 110 * 1024) != cudaSuccess)
            return -1;
        attr_set[dev] = true;
    }
    demod_kernel<XO, FMT, COMPOSITE, YNR><<<blocks, kDemodThreads, smem, stream>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// The kernels with a constant format: the Y'CbCr planar and the two R'G'B'
// formats at the carrier phases of the PAL (1) and PAL-M (0) presets, without
// yNR. R'G'B' as a constant: PALcolour to rgb48, 160 fields, 565 -> 478 us, PAL-M
// 3D to rgbs, 82 fields, 825 -> 788 us; gray, whose luma needs no filter, stays
// with the general kernel.
template <int XO, bool COMPOSITE>
static int demod_launch_xo(const DemodParams &P, unsigned blocks, size_t smem, bool ynr, cudaStream_t stream)
{
    if (ynr) return demod_start<XO, -1, COMPOSITE, true>(P, blocks, smem, stream);
    if constexpr (XO < 2) {
        if (P.format == 0) return demod_start<XO, 0, COMPOSITE, false>(P, blocks, smem, stream);
        if (P.format == 1) return demod_start<XO, 1, COMPOSITE, false>(P, blocks, smem, stream);
        if (P.format == 2) return demod_start<XO, 2, COMPOSITE, false>(P, blocks, smem, stream);
        if (P.format == 3) return demod_start<XO, 3, COMPOSITE, false>(P, blocks, smem, stream);
    }
    return demod_start<XO, -1, COMPOSITE, false>(P, blocks, smem, stream);
}

int demod_launch(const DemodParams &launch, cudaStream_t stream)
{
    if (launch.nout <= 0) return 0;
    DemodParams P = launch;
    const bool composite = P.partial == nullptr;
    const bool ynr = P.nr_y > 0.f;
    // a few fields: shorter blocks, so that every SM (152) has one
    const int field_lines = (P.lafl - P.fafl) / 2 + 1;
    P.lines = demod_lines(ynr);
    while (P.lines > 4 && (long long)P.nout * ((field_lines + P.lines - 1) / P.lines) < 152) P.lines /= 2;
    P.blocks_per_field = (field_lines + P.lines - 1) / P.lines;
    const size_t smem = demod_smem_bytes(P.avs, P.ave, P.lines, ynr);
    if (smem > 110 * 1024) return -1;   // two blocks per SM
    const unsigned blocks = (unsigned)(P.nout * P.blocks_per_field);
    auto launch_kind = [&](auto C) {
        constexpr bool c = decltype(C)::value != 0;
        switch (P.avs & 3) {
        case 0: return demod_launch_xo<0, c>(P, blocks, smem, ynr, stream);
        case 1: return demod_launch_xo<1, c>(P, blocks, smem, ynr, stream);
        case 2: return demod_launch_xo<2, c>(P, blocks, smem, ynr, stream);
        default: return demod_launch_xo<3, c>(P, blocks, smem, ynr, stream);
        }
    };
    return composite ? launch_kind(Num<1>{}) : launch_kind(Num<0>{});
}

}  // namespace tpal
