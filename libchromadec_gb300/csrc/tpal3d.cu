// tpal3d.cu -- Transform-PAL 3D chroma separation on sm_103a.
//
// Computes exactly what the reference's TransformPal3D does
// (src/decoders/palcolour/transform_pal_3d.cpp:123-333): 8x32x16 (fields x
// frame lines x samples) raised-cosine-windowed tiles, half-overlapped, with
// the Z tiles anchored per frame (tiles start at fields 2k-4 and 2k for frame
// k), a forward real DFT, the mirror-about-the-subcarrier threshold, the
// inverse DFT and overlap-add -- restructured for the GPU:
//
//  * One warp owns one spatial tile position (tileX, tileY) and walks forward
//    through a chunk of frames. The 3D DFT is separable, and the X (samples)
//    and Y (frame lines) stages of a field do not depend on which Z tile the
//    field sits in, so each field's 2D spectrum S_f[ky][kx] is computed once
//    and reused by the four Z tiles that contain it. Only kx = 2..6 is ever
//    needed: the filter reads and writes bins x in [XTILE/8, XTILE/4] and
//    their mirrors 8-x (transform_pal_3d.cpp:294-331), so every other bin of
//    the inverse is zero.
//  * Rows of the other field's parity are black (transform_pal_3d.cpp:185-190).
//    Subtracting black (and each row's own mean) before the DFT changes only
//    bins kx in {0, +-1} because the raised cosine's spectrum is supported on
//    {0, +-1}; so those rows become exact zeros and the 32-point Y DFT of a
//    field is a 16-point DFT of its own-parity rows plus a parity twiddle.
//  * Output field 2k gets slice 0 of tile 2k and slice 4 of tile 2k-4
//    (transform_pal_3d.cpp:214-215); the two are summed in the spectral domain
//    and one inverse Y/X transform runs per output field.
//  * Overlap-add across spatial tiles: tiles of one (tileY parity, tileX
//    parity) class never overlap and cover the active area, so each class
//    writes its own partial plane and the demodulator sums the four planes.
//    No atomics; results are deterministic.
//  * Threshold decisions: the spectrum is computed in FP32 with a per-bin
//    error estimate E = K * 2^-24 * (sum_z w_z (A_z[kx] + R_z/2) + sum_z w_z |S_z|_1)
//    where A is the L1 norm of the field's column-DFT outputs for that kx and R
//    the L1 norm of its DC-removed windowed rows. A decision whose margin is
//    inside that band is taken again from the raw samples, in 64-bit fixed
//    point, by the resolve pass, so every decision equals the FP64 reference's.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "tpal_common.cuh"
#include "tpal_kernels.h"

namespace tpal {

// ---------------------------------------------------------------------------
// Constant tables (filled by tp3_init_constants from double precision)
// ---------------------------------------------------------------------------
// X-stage tables as (re, im) pairs for the paired FP32 instructions
// (fma.rn.f32x2: two independent round-to-nearest FMAs, the same results as
// two scalar FMAs, in one instruction):
__constant__ float2 c3_xf[5][8];   // forward X: w(x) (cos theta_kx, -sin theta_kx), theta = 2 pi kx (x - 7.5) / 16
__constant__ float2 c3_xi[5][8];   // inverse X: (2/4096) (cos theta, sin theta)
__constant__ float c3_wy[2][16];   // w_y(y0 + 2i), 32-point raised cosine
__constant__ float c3_wx[16];      // w_x(x)
__constant__ float c3_wz[8];       // w_z(z)
__constant__ float2 c3_tw16[16];   // exp(-2 pi i r / 16)
__constant__ float2 c3_tw32[32];   // exp(-2 pi i r / 32)
// Fixed-point tables of the exact decision path:
// w_x(x) exp(-2 pi i kx x/16), c * 2^60 = hi * 2^30 + lo (lo in [0, 2^30)):
// re.hi, re.lo, im.hi, im.lo
__constant__ int c3_qx[5][16][4];
// w_z(z) w_y(y) exp(-2 pi i r/32), c * 2^59 = hi * 2^29 + lo (lo in [0, 2^29)),
// for z < 4 and y < 16 (both windows are symmetric): [z][y][r], the same order
constexpr int kQYZ = 4 * 16 * 32;
__device__ int4 g3_qyz[kQYZ];

static bool g_tp3_constants_ready[64];

// kappa(lane): the ky a lane owns in the Z stage (bit-reversed low nibble: the
// positions in which the Y stage leaves the spectrum in shared memory); an
// involution.
__device__ __forceinline__ int kappa(int l) { return rev4(l & 15) | (l & 16); }

template <int N>
struct Int {
    static constexpr int value = N;
};

__device__ __forceinline__ float2 shfl_xor2(float2 v, int m)
{
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// Squared threshold of visited bin (z, y, x-2) for x in 2..4.
struct Thr {
    float f;
    df d;
};

__device__ __forceinline__ Thr thr_of(const T3Params &P, int m, int kz, int ky, int kx)
{
    if (P.thr_table == nullptr) {
        if (P.frame_t2 != nullptr) {   // a batch of captures: the threshold of frame m's capture
            const float *t = P.frame_t2 + 3 * max(m, 0);   // warm-up steps before frame 0 take frame 0's
            return {t[0], {t[1], t[2]}};
        }
        return {P.t2f, {P.t2hi, P.t2lo}};
    }
    const float *t = P.thr_table + 3 * ((kz * 32 + ky) * 3 + (kx - 2));
    return {t[0], {t[1], t[2]}};
}

// ---------------------------------------------------------------------------
// Exact decisions in fixed point
// ---------------------------------------------------------------------------
// A bin is a sum over 8 fields x 16 rows of a row's X-stage value times
// w_z w_y exp(-2 pi i (ky y + 4 kz z) / 32). Both factors are integers of two
// words, every product an exact 64-bit integer product, the sums exact; what
// is rounded is each row's value (at 2^-39), the product of the two low words
// (dropped, below 2^-40) and each lane's sum (at 2^-38), against bins of 2^8 and
// more: the result is at least as near the true spectrum as FP64's.
struct fx2 {
    int rh, rl, ih, il;   // value * 2^39 = hi * 2^29 + lo, lo in [0, 2^29)
};

__device__ __forceinline__ void fx_split(long long hi_acc, long long lo_acc, int &h, int &l)
{
    // v = hi_acc * 2^-30 + lo_acc * 2^-60; hi_acc and lo_acc are below 2^51
    const long long v = (hi_acc << 9) + ((lo_acc + (1 << 20)) >> 21);
    h = (int)(v >> 29);
    l = (int)v & ((1 << 29) - 1);
}

// X stage of one row for columns kx and 8 - kx. The second column's
// coefficients are the first's conjugated with sign (-1)^x
// (w(x) exp(-2 pi i (8-k) x / 16) = (-1)^x conj(w(x) exp(-2 pi i k x / 16))),
// so the products are formed once: even and odd samples summed apart, column
// kx is even + odd, column 8 - kx the conjugate of even - odd.
__device__ __forceinline__ void x_row_pair(const uint16_t *field, long long base, long long field_len, int black,
                                           int kx, fx2 &xa, fx2 &xb)
{
    long long e[4] = {0, 0, 0, 0}, o[4] = {0, 0, 0, 0};   // re.hi, re.lo, im.hi, im.lo
    int a[16];
    if (base >= 1 && base + 18 <= field_len) {
        // nine aligned 32-bit words and a funnel shift, as the walk's rows
        const uintptr_t pa = reinterpret_cast<uintptr_t>(field + base);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(pa & ~(uintptr_t)3);
        const unsigned sh = (unsigned)(pa & 2) * 8u;
        uint32_t wd[9];
#pragma unroll
        for (int k = 0; k < 9; k++) wd[k] = __ldg(w + k);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t v = __funnelshift_r(wd[k], wd[k + 1], sh);
            a[2 * k] = (int)(v & 0xFFFFu) - black;
            a[2 * k + 1] = (int)(v >> 16) - black;
        }
    } else {
#pragma unroll
        for (int x = 0; x < 16; x++) {
            const long long idx = base + x < 0 ? 0 : base + x;   // never outside the field
            a[x] = (int)__ldg(field + (idx < field_len ? idx : field_len - 1)) - black;
        }
    }
#pragma unroll
    for (int x = 0; x < 16; x++) {
        const int *c = c3_qx[kx - 2][x];
        long long *acc = (x & 1) ? o : e;
#pragma unroll
        for (int k = 0; k < 4; k++) acc[k] += (long long)a[x] * c[k];
    }
    fx_split(e[0] + o[0], e[1] + o[1], xa.rh, xa.rl);
    fx_split(e[2] + o[2], e[3] + o[3], xa.ih, xa.il);
    fx_split(e[0] - o[0], e[1] - o[1], xb.rh, xb.rl);
    fx_split(o[2] - e[2], o[3] - e[3], xb.ih, xb.il);
}

// (high, middle) sums of complex products: high counts 2^-40, middle 2^-69.
struct fxsum {
    long long rh, rm, ih, im;
    __device__ __forceinline__ void mac(const fx2 &x, int4 c)   // c: re.hi, re.lo, im.hi, im.lo
    {
        const int nh = -c.z, nl = -c.w;
        rh += (long long)x.rh * c.x;
        rh += (long long)x.ih * nh;
        rm += (long long)x.rh * c.y;
        rm += (long long)x.rl * c.x;
        rm += (long long)x.ih * nl;
        rm += (long long)x.il * nh;
        ih += (long long)x.rh * c.z;
        ih += (long long)x.ih * c.x;
        im += (long long)x.rh * c.w;
        im += (long long)x.rl * c.z;
        im += (long long)x.ih * c.y;
        im += (long long)x.il * c.x;
    }
};

// a 64-bit integer below 2^63 in magnitude as double-float (about 2^-48 of
// it), through 32-bit conversions (the 64-bit ones run on the FP64 pipe,
// which this GPU has little of)
__device__ __forceinline__ df df_from_i64(long long v)
{
    const float fh = (float)(int)(v >> 40) * 1099511627776.0f;              // below 2^23: exact
    const float fm = (float)(int)((v >> 20) & 0xFFFFF) * 1048576.0f;        // 20 bits: exact
    const float fl = (float)(int)(v & 0xFFFFF);
    return df_add(two_sum(fh, fm), df_make(fl));
}

__device__ __forceinline__ long long shfl_xor_i64(long long v, int m)
{
    const int lo = __shfl_xor_sync(0xffffffffu, (int)v, m), hi = __shfl_xor_sync(0xffffffffu, (int)(v >> 32), m);
    return (long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo);
}

// sim(a, b, t) = !(a < b t || b < a t) evaluated in double-float
__device__ __forceinline__ bool df_sim(df a, df b, df t)
{
    const df d1 = df_sub(a, df_mul(b, t));
    const df d2 = df_sub(b, df_mul(a, t));
    return !(df_sign(d1) < 0 || df_sign(d2) < 0);
}

// ---------------------------------------------------------------------------
// The walk: layout and per-lane constants
// ---------------------------------------------------------------------------
// One warp walks one tile position through a chunk of frames, two fields (one
// frame) a step. What bounds it is the number of instructions it issues, so
// each stage's data is laid out where that stage needs no exchange:
//
//  * X stage: lane (j, i) owns row i of field j of the pair. Component j of
//    every packed pair is that field.
//  * Y stage: lanes 0..19 own one (kx, quarter) each: 4 of the column's 16
//    points, both fields packed in f32x2 registers, two radix-4 passes with
//    one exchange through shared memory. The shuffle version ran the 4
//    radix-2 stages across 16 lanes: 8 shuffles, 8 selects and the twiddles
//    of both halves per column and field.
//  * Z stage: a field's spectrum at ky + 16 is +- its value at ky, the sign
//    by the parity of its rows, which alternates with z. So a tile's bin at
//    (kz, ky + 16) is +- the bin at (kz + 4, ky), bit for bit in the radix-2
//    order used here: 16 values of ky are transformed, compared and masked,
//    and the other 16 reuse them. Half-warp h takes the columns kx = 2 + h
//    and, at the mirror ky, 6 - h: both bins of every pair the filter
//    compares are in one lane, no shuffles of magnitudes or decisions. kx = 4
//    mirrors onto itself; its pass runs all 32 ky.
//  * Signs: everything at ky >= 16 is kept with the sign of odd z, which
//    is the true value or its negative for the whole launch; the inverse Y
//    stage folds the two halves with the factors (1, -1).
//
// Shared memory per warp (float4 units): the window [4 pairs][5 kx][16]
// as (re0, re1, im0, im1) of the pair's two fields, the Z carries
// [m & 1][5 kx][32] as (slice 4, slice 5), the buffers of the forward and the
// inverse Y stage, [5 kx][16] in rows of 20 (the columns of a quarter-warp
// fall on different banks; the inverse one starts with the output spectra,
// already folded to 16 positions, and ends with the output rows), and the
// bound terms: 13.7 KB. With 128 registers a thread 16 warps are resident on
// an SM; the per-bin walk holds two sets of decisions and takes 168 registers
// and 12 warps.
//
// The inverse Y stage of one step runs together with the forward Y stage of
// the next: two independent chains through the same exchange.
//
// Measured against the walk before it (one ky per lane in the Z stage, shuffle
// DFTs in the Y stages, every bin's guard band in the loop): 2,671 -> 1,541
// warp instructions a step, 526 -> 325 us for 60 fields. The path of shared
// memory and L1 is 72 % busy and the issue slots 69 %; the rest is latency
// (short scoreboard) and instruction fetch: unrolling the kx pairs, a second
// copy of the rare path or straight-line code for both passes each measured
// slower. So did samples by asynchronous 16-byte copies (coalesced, but with
// nine shared loads a lane and the addresses: 413 us) and two or three warps
// a block.
constexpr int kWarps3 = 4;
constexpr float kBoundFactor = 2.0f;   // guard band, in units of the per-bin error estimate
constexpr float kEps32 = 5.9604645e-8f;
// a + b + E^2 + rE^2 below this (with a margin for the FP32 magnitudes)
// keeps the effect of a decision under 1/4 sample unit: (4/4096) * 256 = 1/4
constexpr float kTinyPair = 65000.0f;
constexpr int kWinF4 = 4 * 5 * 16;
constexpr int kCarryF4 = 2 * 5 * 32;
constexpr int kExchF4 = 5 * 20;
constexpr int kOutF4 = 5 * 20;         // output spectra, the inverse exchange, then the output rows
constexpr int kBndF4 = 4 * 4;          // [4 pairs][8] float2: kx 0..4 and the row term at 5
constexpr int kWarpF4 = kWinF4 + kCarryF4 + kExchF4 + kOutF4 + kBndF4;
constexpr int kTwF4 = 4 * 7;           // Y twiddles per quarter r, per block
constexpr int kThrF4 = 3 * 8 * 32 / 4; // squared per-bin thresholds, per block (per-bin walks only)
constexpr size_t walk_smem(bool per_bin)
{
    return sizeof(float4) * (size_t)(kWarps3 * kWarpF4 + kTwF4 + (per_bin ? kThrF4 : 0));
}

// A position p of 16 or 32 is stored at p ^ ((p >> 2) & 3): lanes that read
// or write 4r + e for fixed e and lanes that access consecutive positions
// both fall on distinct banks.
__device__ __forceinline__ int swz(int p) { return p ^ ((p >> 2) & 3); }

struct LaneConst {
    int j, i;             // field of the pair, row
    float wy;             // w_y(y0 + 2i), y0 the parity of the field's rows
    int rowL;             // frame line of this lane's row
    bool row_ok, row_fast;
    int row_off;          // its first sample within the field (negative before the first line)
    int ky;               // of position lane & 15 (below 16)
    int posA, posB;       // window positions of ky and its mirror
    int laneB;            // position (of 32) of the mirror ky
    float2 wzB[4];        // w_z of fields 2q, 2q+1, odd fields negated for a mirror ky >= 16
};

__device__ __forceinline__ LaneConst lane_const(const T3Params &P, int lane, int tileX, int tileY)
{
    LaneConst c;
    c.j = lane >> 4;
    c.i = lane & 15;
    const int odd = 1 ^ ((P.swap ^ tileY) & 1);   // the field whose rows have parity 1 within the tile
    const int y0 = c.j == odd;
    c.wy = c3_wy[y0][c.i];
    c.rowL = tileY + y0 + 2 * c.i;
    c.row_ok = c.rowL >= P.fafl && c.rowL <= P.lafl;
    const int fl = c.rowL >> 1;
    // Three aligned vectors around the row stay inside the field: the row is not
    // its first, and it is not the last unless the vectors end inside it.
    c.row_fast = tileX >= 0 && fl >= 1 && tileX + 24 <= (fl + 1 < P.fh ? 2 * P.fw : P.fw);
    c.row_off = fl * P.fw + tileX;
    c.ky = rev4(c.i);
    c.laneB = kappa((40 - c.ky) & 31);
    c.posA = swz(c.i);
    c.posB = swz(c.laneB & 15);
#pragma unroll
    for (int q = 0; q < 4; q++)
        c.wzB[q] = make_float2(c3_wz[2 * q], c.laneB >= 16 ? -c3_wz[2 * q + 1] : c3_wz[2 * q + 1]);
    return c;
}

// w_z of fields 2q, 2q+1 of a Z tile for a ky below 16 (high = false) or not
__device__ __forceinline__ void z_window(float2 (&wz)[4], bool high)
{
#pragma unroll
    for (int q = 0; q < 4; q++) wz[q] = make_float2(c3_wz[2 * q], high ? -c3_wz[2 * q + 1] : c3_wz[2 * q + 1]);
}

// The block's Y twiddles, per quarter r: exp(-2 pi i n / 16) for n = r, r + 4
// and 2r in both components, then for the positions 4r + e (bin k =
// rev4(4r + e)) exp(-2 pi i k / 32) in the component of the field with odd
// rows and 1 in the other. Entry v of quarter r: (x0, x1, y0, y1) at
// tw[7 r + v]; (-y0, -y1) is a multiplication, cheaper than two more wavefronts
// of the shared-memory path that bounds the walk (3,970 -> 3,940 us for 500
// fields, demodulator included).
__device__ __forceinline__ void fill_twiddles(const T3Params &P, float4 *tw)
{
    const int odd = 1 ^ ((P.swap ^ P.tileY0) & 1);   // tile rows start 16 lines apart
    for (int t = threadIdx.x; t < 4 * 7; t += blockDim.x) {
        const int r = t / 7, v = t % 7;
        float2 w = v < 3 ? c3_tw16[v == 0 ? r : v == 1 ? r + 4 : 2 * r] : c3_tw32[rev4(4 * r + v - 3)];
        float2 w0 = w, w1 = w;
        if (v >= 3) (odd ? w0 : w1) = make_float2(1.f, 0.f);
        tw[7 * r + v] = make_float4(w0.x, w1.x, w0.y, w1.y);
    }
    __syncthreads();
}
__device__ __forceinline__ tw2 twiddle(const float4 *tw, int r, int v)
{
    const float4 a = tw[7 * r + v];
    const float2 y = make_float2(a.z, a.w);
    return {make_float2(a.x, a.y), y, __fmul2_rn(y, make_float2(-1.f, -1.f))};
}

constexpr unsigned kYLanes = 0xFFFFFu;   // lanes 0..19 run the Y stages

// The 16 samples of this lane's row of field 2q + j, as words that a funnel
// shift lines up.
struct RowWords {
    uint32_t w[12];
    unsigned at;  // byte of the first sample within w
    bool valid;   // else the row is black: outside the capture or the active lines
};

__device__ __forceinline__ void load_row(const T3Params &P, int q, const LaneConst &LC, RowWords &r)
{
    const int f = 2 * q + LC.j;
    const uint16_t *fp = (f >= 0 && f < P.nfields) ? field_at(P, f) : nullptr;
    r.valid = fp != nullptr && LC.row_ok;
    r.at = 0;
    if (!r.valid) return;
    if (LC.row_fast) {
        // Rows start on any 2-byte boundary (odd line and field lengths):
        // three aligned 16-byte vectors cover the 16 samples. A warp's load
        // touches 32 rows however wide it is: as nine words the rows took 98
        // of a step's 464 wavefronts (3,970 -> 3,930 us for 500 fields).
        const uintptr_t pa = reinterpret_cast<uintptr_t>(fp + LC.row_off);
        const uint4 *w = reinterpret_cast<const uint4 *>(pa & ~(uintptr_t)15);
        r.at = (unsigned)pa & 15u;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint4 u = __ldg(w + k);
            r.w[4 * k] = u.x;
            r.w[4 * k + 1] = u.y;
            r.w[4 * k + 2] = u.z;
            r.w[4 * k + 3] = u.w;
        }
    } else {
        // Never outside the field: a tile that hangs over the start of the first
        // line takes its first sample, one over the end of the last its last.
        const int end = P.fw * P.fh - 1;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int e = LC.row_off + 2 * k;
            r.w[k] = (uint32_t)__ldg(fp + __vimin_s32_relu(e, end)) |   // max(min(e, end), 0)
                     ((uint32_t)__ldg(fp + __vimin_s32_relu(e + 1, end)) << 16);
        }
#pragma unroll
        for (int k = 8; k < 12; k++) r.w[k] = 0;
    }
}

// Forward X stage of fields 2q and 2q+1: this lane's row into the exchange
// buffer, and R, the L1 norm of the field's DC-removed windowed rows, into bnd.
__device__ __forceinline__ void x_forward(const RowWords &row, int q, const LaneConst &LC, float4 *exch, float2 *bnd)
{
    // Row samples with the row mean removed, folded about the window's
    // centre: s_x = a_x + a_15-x - 2*mean, d_x = a_x - a_15-x. Both are exact
    // in FP32 and free of the black level. |a_x - mean| + |a_15-x - mean| is
    // max(|s_x|, |d_x|).
    float2 sd[8];   // (s_x, d_x)
    float rowl1 = 0.0f;
    if (row.valid) {
        // the words lined up by whole words, then by a half
        uint32_t e[10], g[9], v[8];   // v: samples 2k, 2k+1
#pragma unroll
        for (int k = 0; k < 10; k++) e[k] = row.at & 8u ? row.w[k + 2] : row.w[k];
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = row.at & 4u ? e[k + 1] : e[k];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __funnelshift_r(g[k], g[k + 1], (row.at & 2u) * 8u);
        // 2^23 + a from the sample's bits; subtracting 2^24 from one side of
        // each sum leaves a_x + a_15-x exactly
        float2 t[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 p = make_float2(__uint_as_float(__byte_perm(v[k], 0x4B000000u, 0x7610)),
                                         __uint_as_float(__byte_perm(v[k], 0x4B000000u, 0x7632)));
            const float2 o = make_float2(__uint_as_float(__byte_perm(v[7 - k], 0x4B000000u, 0x7632)),
                                         __uint_as_float(__byte_perm(v[7 - k], 0x4B000000u, 0x7610)));
            sd[2 * k].y = __fsub_rn(p.x, o.x);
            sd[2 * k + 1].y = __fsub_rn(p.y, o.y);
            t[k] = add2(add2(p, make_float2(-16777216.f, -16777216.f)), o);
        }
        const float2 u = add2(add2(t[0], t[1]), add2(t[2], t[3]));
        const float mean2 = __fmul_rn(__fadd_rn(u.x, u.y), 0.125f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            sd[2 * k].x = __fsub_rn(t[k].x, mean2);
            sd[2 * k + 1].x = __fsub_rn(t[k].y, mean2);
        }
#pragma unroll
        for (int x = 0; x < 8; x++) rowl1 = __fmaf_rn(c3_wx[x], fmaxf(fabsf(sd[x].x), fabsf(sd[x].y)), rowl1);
    } else {
#pragma unroll
        for (int x = 0; x < 8; x++) sd[x] = make_float2(0.f, 0.f);
    }
    rowl1 *= LC.wy;
#pragma unroll
    for (int h = 1; h < 16; h <<= 1) rowl1 += __shfl_xor_sync(0xffffffffu, rowl1, h);
    float *bq = reinterpret_cast<float *>(bnd + 8 * (q & 3));
    if (LC.i == 0) bq[2 * 5 + LC.j] = rowl1;

    // column DFT bin kx = k+2 of this row (window and centre phase folded)
    // rows 8..15 write their imaginary part first: 32 different banks a store
    float *xr = reinterpret_cast<float *>(exch) + 4 * LC.i + LC.j;
    const bool upper = LC.i >= 8;
    float *xs = xr + (upper ? 2 : 0), *xt = xr + (upper ? 0 : 2);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        float2 X = make_float2(0.f, 0.f);
#pragma unroll
        for (int x = 0; x < 8; x++) X = __ffma2_rn(c3_xf[k][x], sd[x], X);
        X = __fmul2_rn(X, make_float2(LC.wy, LC.wy));
        xs[80 * k] = upper ? X.y : X.x;
        xt[80 * k] = upper ? X.x : X.y;
    }
}

// Y stages, lanes 0..19: the forward one of fields 2q and 2q+1 from their
// rows in `exch` to window slot q & 3 (and A per kx, the L1 norm of the
// column-DFT outputs over the rows, into bnd); with INV the inverse one of the
// folded output spectra R (re0, re1, im0, im1), in place.
template <bool INV>
__device__ __forceinline__ void y_stages(int q, const LaneConst &LC, int lane, float4 *win, float4 *exch, float4 *R,
                                         float2 *bnd, const float4 *tw)
{
    const int k = lane >> 2, r = lane & 3;
    float4 *x = exch + 20 * k, *y = R + 20 * k;
    cp2 a[4], G[4];
#pragma unroll
    for (int n = 0; n < 4; n++) a[n] = cp_of(x[r + 4 * n]);
    const tw2 t0 = twiddle(tw, r, 0), t1 = twiddle(tw, r, 1), t2 = twiddle(tw, r, 2);
    if (INV) {
#pragma unroll
        for (int n = 0; n < 4; n++) {
            // exp(+i pi kk / 16) for the odd field
            G[n] = ctw(cp_of(y[4 * r + (n ^ r)]), twiddle(tw, r, 3 + n), true);
        }
    }
    float A0 = 0.f, A1 = 0.f;
#pragma unroll
    for (int n = 0; n < 4; n++) {
        A0 += fabsf(a[n].re.x) + fabsf(a[n].im.x);
        A1 += fabsf(a[n].re.y) + fabsf(a[n].im.y);
    }
#pragma unroll
    for (int h = 1; h < 4; h <<= 1) {
        A0 += __shfl_xor_sync(kYLanes, A0, h);
        A1 += __shfl_xor_sync(kYLanes, A1, h);
    }
    if (r == 0) bnd[8 * (q & 3) + k] = make_float2(A0, A1);
    // Forward: 16-point DFT over the rows, radix-2 DIF: spans 8 and 4 over
    // the rows r + 4n, spans 2 and 1 over the positions 4r + e; position p
    // ends with bin rev4(p). Inverse: bit-reversed input to natural order
    // (DIT), spans 1 and 2 over 4r + e, spans 4 and 8 over r + 4n.
    const cp2 u0 = cadd(a[0], a[2]), u1 = cadd(a[1], a[3]);
    const cp2 v0 = ctw(csub(a[0], a[2]), t0, false), v1 = ctw(csub(a[1], a[3]), t1, false);
    __syncwarp(kYLanes);   // rows and spectra have been read: both buffers may be written
    x[0 + r] = f4_of(cadd(u0, u1));
    x[4 + (r ^ 1)] = f4_of(ctw(csub(u0, u1), t2, false));
    x[8 + (r ^ 2)] = f4_of(cadd(v0, v1));
    x[12 + (r ^ 3)] = f4_of(ctw(csub(v0, v1), t2, false));
    if (INV) {
        const cp2 w0 = cadd(G[0], G[1]), w1 = csub(G[0], G[1]), w2 = cadd(G[2], G[3]), d3 = csub(G[2], G[3]);
        y[4 * r + (0 ^ r)] = f4_of(cadd(w0, w2));
        y[4 * r + (2 ^ r)] = f4_of(csub(w0, w2));
        // the odd branch of span 2 times exp(+i pi/2): (-d3.im, d3.re)
        y[4 * r + (1 ^ r)] = f4_of({sub2(w1.re, d3.im), add2(w1.im, d3.re)});
        y[4 * r + (3 ^ r)] = f4_of({add2(w1.re, d3.im), sub2(w1.im, d3.re)});
    }
    __syncwarp(kYLanes);
#pragma unroll
    for (int n = 0; n < 4; n++) {
        a[n] = cp_of(x[4 * r + (n ^ r)]);
        if (INV) G[n] = cp_of(y[4 * n + (r ^ n)]);
    }
    const cp2 w0 = cadd(a[0], a[2]), w1 = cadd(a[1], a[3]), w2 = csub(a[0], a[2]), d3 = csub(a[1], a[3]);
    // the odd branch of span 2 times exp(-i pi/2): (d3.im, -d3.re)
    const cp2 o[4] = {cadd(w0, w1), csub(w0, w1), {add2(w2.re, d3.im), sub2(w2.im, d3.re)},
                      {sub2(w2.re, d3.im), add2(w2.im, d3.re)}};
    // parity twiddle of the odd field: S[kk] = exp(-2 pi i kk/32) A[kk]
    float4 *dst = win + (5 * (q & 3) + k) * 16 + 4 * r;
#pragma unroll
    for (int n = 0; n < 4; n++) dst[n ^ r] = f4_of(ctw(o[n], twiddle(tw, r, 3 + n), false));
    if (INV) {
        const cp2 f1 = ctw(G[1], t2, true), f3 = ctw(G[3], t2, true);
        const cp2 g0 = cadd(G[0], f1), g1 = csub(G[0], f1);
        const cp2 g2 = ctw(cadd(G[2], f3), t0, true), g3 = ctw(csub(G[2], f3), t1, true);
        __syncwarp(kYLanes);   // the exchange has been read
        y[r] = f4_of(cadd(g0, g2));
        y[r + 4] = f4_of(cadd(g1, g3));
        y[r + 8] = f4_of(csub(g0, g2));
        y[r + 12] = f4_of(csub(g1, g3));
    }
}

// 8-point forward DFT of one windowed column (natural order out): radix-2
// DIF, the first two stages on the packed fields (z, z+1), the twiddles 1 and
// -i applied exactly, exp(-i pi/4) and exp(-3i pi/4) by complex multiplication.
__device__ __forceinline__ void z_dft(const float4 *win, int m, int k, int pos, const float2 (&wz)[4], float2 (&Y)[8])
{
    cp2 a[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const cp2 v = cp_of(win[(5 * ((m + q) & 3) + k) * 16 + pos]);
        a[q] = {__fmul2_rn(v.re, wz[q]), __fmul2_rn(v.im, wz[q])};
    }
    const cp2 b01 = cadd(a[0], a[2]), b23 = cadd(a[1], a[3]);   // b0, b1 / b2, b3
    const cp2 d01 = csub(a[0], a[2]), d23 = csub(a[1], a[3]);   // a0 - a4, a1 - a5 / a2 - a6, a3 - a7
    const float2 b5 = cmul(make_float2(d01.re.y, d01.im.y), c3_tw32[4]);
    const float2 b7 = cmul(make_float2(d23.re.y, d23.im.y), c3_tw32[12]);
    const cp2 c01 = cadd(b01, b23), c23 = csub(b01, b23);       // c0, c1 / c2, b1 - b3
    Y[0] = make_float2(__fadd_rn(c01.re.x, c01.re.y), __fadd_rn(c01.im.x, c01.im.y));
    Y[4] = make_float2(__fsub_rn(c01.re.x, c01.re.y), __fsub_rn(c01.im.x, c01.im.y));
    Y[2] = make_float2(__fadd_rn(c23.re.x, c23.im.y), __fsub_rn(c23.im.x, c23.re.y));   // c3 = -i (b1 - b3)
    Y[6] = make_float2(__fsub_rn(c23.re.x, c23.im.y), __fadd_rn(c23.im.x, c23.re.y));
    // b4 = a0 - a4, b6 = -i (a2 - a6)
    const float2 c4 = make_float2(__fadd_rn(d01.re.x, d23.im.x), __fsub_rn(d01.im.x, d23.re.x));
    const float2 c6 = make_float2(__fsub_rn(d01.re.x, d23.im.x), __fadd_rn(d01.im.x, d23.re.x));
    const float2 c5 = add2(b5, b7), v = sub2(b5, b7);           // c7 = -i v
    Y[1] = add2(c4, c5);
    Y[5] = sub2(c4, c5);
    Y[3] = make_float2(__fadd_rn(c6.x, v.y), __fsub_rn(c6.y, v.x));
    Y[7] = make_float2(__fsub_rn(c6.x, v.y), __fadd_rn(c6.y, v.x));
}

__device__ __forceinline__ float mag2(float2 y) { return __fmaf_rn(y.x, y.x, __fmul_rn(y.y, y.y)); }

// Inverse Z of one masked column to slices 0, 1, 4, 5: the even and odd parts
// of slices 0 and 1, each a sum in the order of kz.
struct ZInverse {
    float2 E0, E1, O0, O1;
    // y: the masked bins; o[i]: bin 2i + 1 times exp(+2 pi i (2i + 1) / 8)
    __device__ __forceinline__ void sum(const float2 (&y)[8], const float2 (&o)[4])
    {
        E0 = add2(add2(add2(y[0], y[2]), y[4]), y[6]);
        O0 = add2(add2(add2(y[1], y[3]), y[5]), y[7]);
        // slice 1: even part y0 + i y2 - y4 - i y6
        E1.x = __fadd_rn(__fsub_rn(__fsub_rn(y[0].x, y[2].y), y[4].x), y[6].y);
        E1.y = __fsub_rn(__fsub_rn(__fadd_rn(y[0].y, y[2].x), y[4].y), y[6].x);
        O1 = add2(add2(add2(o[0], o[1]), o[2]), o[3]);
    }
    // the sums of ky + 16 where its masked bins are those of ky moved by 4
    // (O1 negated: exp(2 pi i (kz + 4) / 8) = -exp(2 pi i kz / 8))
    __device__ __forceinline__ void sum_moved(const float2 (&y)[8], const float2 (&o)[4])
    {
        const float2 ym[8] = {y[4], y[5], y[6], y[7], y[0], y[1], y[2], y[3]};
        const float2 om[4] = {o[2], o[3], o[0], o[1]};
        sum(ym, om);
        O1 = make_float2(-O1.x, -O1.y);
    }
    // slices 4 and 5
    __device__ __forceinline__ float4 later() const
    {
        const float2 d0 = sub2(E0, O0);
        return make_float4(d0.x, d0.y, __fsub_rn(E1.x, O1.x), __fsub_rn(E1.y, O1.y));
    }
    // The output spectra at one ky, field 2m: slice 0 + carried slice 4 of
    // tile 2m-4, field 2m+1: slice 1 + carried slice 5; then this tile's
    // slices 4, 5 are carried for frame m+2.
    __device__ __forceinline__ cp2 finish(float4 *carry) const
    {
        const float4 c = *carry;
        const float2 s0 = add2(E0, O0);
        const float2 s1 = make_float2(__fadd_rn(E1.x, O1.x), __fadd_rn(E1.y, O1.y));
        *carry = later();
        return {make_float2(__fadd_rn(s0.x, c.x), __fadd_rn(s1.x, c.z)),
                make_float2(__fadd_rn(s0.y, c.y), __fadd_rn(s1.y, c.w))};
    }
};

// The inverse Y stage's first step: ky and ky + 16 of the two fields added
// (even rows) or subtracted (odd rows).
__device__ __forceinline__ cp2 fold_ky(cp2 lo, cp2 hi)
{
    const float2 s = make_float2(1.f, -1.f);
    return {__ffma2_rn(hi.re, s, lo.re), __ffma2_rn(hi.im, s, lo.im)};
}

__device__ __forceinline__ void z_rotate(const float2 (&y)[8], float2 (&o)[4])
{
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = cmulc(y[2 * i + 1], c3_tw32[4 * (2 * i + 1)]);
}

// Masks column Y at ky (position `at` of 32) by k and at ky +- 16 by kh,
// inverse Z and overlap-add of both, and their folded output spectrum into R.
// MOVED: kh is k moved by 4, the sums share the masked bins.
template <bool MOVED>
__device__ __forceinline__ void z_inverse(const float2 (&Y)[8], const float (&k)[8], const float (&kh)[8],
                                          float4 *carry, float4 *R, int col, int at)
{
    float2 y[8], o[4];
#pragma unroll
    for (int z = 0; z < 8; z++) y[z] = __fmul2_rn(Y[z], make_float2(k[z], k[z]));
    z_rotate(y, o);
    ZInverse Z;
    Z.sum(y, o);
    const cp2 a = Z.finish(carry + 32 * col + at);
    if (MOVED) {
        Z.sum_moved(y, o);
    } else {
        float2 yh[8];
#pragma unroll
        for (int z = 0; z < 8; z++) yh[z] = __fmul2_rn(Y[z ^ 4], make_float2(kh[z], kh[z]));
        z_rotate(yh, o);
        Z.sum(yh, o);
    }
    const cp2 b = Z.finish(carry + 32 * col + (at ^ 16));
    cp2 g = fold_ky(a, b);
    if (at >= 16) {   // a is the upper half: component 1 is b - a
        g.re.y = -g.re.y;
        g.im.y = -g.im.y;
    }
    R[20 * col + swz(at & 15)] = f4_of(g);
}

__device__ __forceinline__ bool fsim(float a, float b, float t) { return (__fmaf_rn(-b, t, a) >= 0.f) && (__fmaf_rn(-a, t, b) >= 0.f); }

__device__ __forceinline__ bool funcertain(float a, float b, float t, float pa, float pb)
{
    return (fabsf(__fmaf_rn(-b, t, a)) <= pa + t * pb) || (fabsf(__fmaf_rn(-a, t, b)) <= pb + t * pa);
}

__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The error bounds of one step. Lane k of 0..4 holds, for kx = k+2,
//   ek = sum_z w_z (A_z[kx] + R_z / 2), the part of the per-bin estimate
//        E = K 2^-24 (ek + sum_z w_z |S_z|_1) every ky shares, and
//   em = an upper bound of E over every ky of columns kx and 8 - kx:
//        |S_z|_1 <= sqrt(2) |S_z| <= sqrt(2) A_z.
struct StepBounds {
    float ek, em;
};

__device__ __forceinline__ StepBounds step_bounds(const float2 *bnd, int m, int lane)
{
    const int kk = lane & 7, q = lane >> 3;
    const float2 b = bnd[8 * ((m + q) & 3) + kk];
    float v = __fmaf_rn(c3_wz[2 * q], b.x, c3_wz[2 * q + 1] * b.y);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    const float r = __shfl_sync(0xffffffffu, v, 5);
    StepBounds o;
    o.ek = __fmaf_rn(0.5f, r, v);
    const float es = kBoundFactor * kEps32 * 1.001f * __fmaf_rn(2.41422f, v, 0.5f * r);
    o.em = fmaxf(es, __shfl_sync(0xffffffffu, es, (4 - kk) & 7));
    return o;
}

// A column with everything its guard band needs, recomputed from the window
// (the same magnitudes the walk decided on).
struct Col {
    float2 Y[8];
    float mag[8], E;
};

__device__ __forceinline__ void z_column(const float4 *win, int m, int k, int pos, const float2 (&wz)[4], float ek,
                                         Col &c)
{
    float B = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const cp2 v = cp_of(win[(5 * ((m + q) & 3) + k) * 16 + pos]);
        B = __fmaf_rn(fabsf(wz[q].x), fabsf(v.re.x) + fabsf(v.im.x), B);
        B = __fmaf_rn(fabsf(wz[q].y), fabsf(v.re.y) + fabsf(v.im.y), B);
    }
    z_dft(win, m, k, pos, wz, c.Y);
#pragma unroll
    for (int kz = 0; kz < 8; kz++) c.mag[kz] = mag2(c.Y[kz]);
    c.E = kBoundFactor * kEps32 * (ek + B);
}

// The guard band of one kx group of a step, bin by bin, and its record for
// tp3_resolve_kernel. `last` is the warp's latest record of this item (the
// records of one item form a list in the order of (m, g)).
template <bool PER_BIN>
__device__ __forceinline__ void record_group(const T3Params &P, const LaneConst &LC, const float4 *win,
                                             const float *thr, int item, int m, int g, int lane, float tf_m, float ekA,
                                             float ekB, int &last)
{
    // all 32 ky, one per lane, each with its mirror
    const int ky = kappa(lane), kyr = (40 - ky) & 31, laneB = kappa(kyr);
    float2 wz[4];
    Col A, B;
    z_window(wz, lane >= 16);
    z_column(win, m, g, LC.posA, wz, ekA, A);
    z_window(wz, laneB >= 16);
    z_column(win, m, 4 - g, LC.posB, wz, ekB, B);
    unsigned keep = 0, unc = 0;
    // A pair too small to matter is left to FP32: toggling bins of
    // magnitudes |Y_b|, |Y_r| moves any output sample by at most
    // (2/4096)(|Y_b| + |Y_r|) <= (4/4096) sqrt(a + b + E^2 + rE^2)
    // (true magnitudes within E of the computed ones), so under
    // kTinyPair the change is below 1/4 of a composite sample unit
    // (0.38 LSB of yuv444p16, 7e-6 of yuv444ps).
    const float tiny_lim = kTinyPair - __fmaf_rn(A.E, A.E, B.E * B.E);
#pragma unroll
    for (int kz = 0; kz < 8; kz++) {
        const int kzr = (10 - kz) & 7;
        const float a = A.mag[kz], b = B.mag[kzr];
        const float pa = 2.f * A.E * l1(A.Y[kz]) + A.E * A.E;
        const float pb = 2.f * B.E * l1(B.Y[kzr]) + B.E * B.E;
        float t = tf_m;
        if (PER_BIN) t = thr[(8 * g + kz) * 32 + lane];
        bool sim = fsim(a, b, t);
        bool u = funcertain(a, b, t, pa, pb);
        if (PER_BIN && g == 2) {   // kx = 4: the mirror bin visits too, with its own threshold
            const float t2 = thr[(16 + kzr) * 32 + laneB];
            sim |= fsim(a, b, t2);
            u |= funcertain(a, b, t2, pa, pb);
        }
        // a carrier (its own mirror) is always kept
        const bool self = (g == 2) && (kz == kzr) && (ky == kyr);
        if (sim || self) keep |= 1u << kz;
        if (u && !self && !(a + b < tiny_lim)) unc |= 1u << kz;
    }
    // (a flat or black tile, whose bound is zero, never has any)
    if (!__any_sync(0xffffffffu, unc != 0)) return;
    unsigned slot = 0;
    if (lane == 0) slot = atomicAdd(P.counters, 1u);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (slot >= P.unc_cap) return;   // sized for every kx group of the launch
    UncRecord &rec = P.unc_rec[slot];
    if (lane == 0) {
        rec.item = item;
        rec.mg = m * 4 + g;
        rec.prev = last;
        rec.next = -1;
        if (last >= 0) P.unc_rec[last].next = (int)slot;
    }
    rec.unc[lane] = (uint8_t)unc;
    rec.keep[lane] = (uint8_t)keep;
    last = (int)slot;
}

// Inverse X stage of step m's output rows, and the store of each lane's row
// into its overlap class.
__device__ __forceinline__ void x_inverse_store(const T3Params &P, const LaneConst &LC, const float4 *rows, int m,
                                                int tileX, int cls)
{
    float2 CS[8];   // (cosine sum, sine sum) of row i
#pragma unroll
    for (int x = 0; x < 8; x++) CS[x] = make_float2(0.f, 0.f);
    const float *yr = reinterpret_cast<const float *>(rows) + 4 * LC.i + LC.j;
    const bool upper = LC.i >= 8;   // reads its imaginary part first: 32 different banks a load
    const float *ys = yr + (upper ? 2 : 0), *yt = yr + (upper ? 0 : 2);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const float u = ys[80 * k], v = yt[80 * k];
        const float2 G = make_float2(upper ? v : u, upper ? u : v);
#pragma unroll
        for (int x = 0; x < 8; x++) CS[x] = __ffma2_rn(G, c3_xi[k][x], CS[x]);
    }
    // Store row i of field 2m + j.
    if (LC.row_ok) {
        const int ofield = 2 * (m - P.frame_begin) + LC.j;
        float *dst = P.partial + (long long)cls * P.part_class_stride + (long long)ofield * P.part_field_stride +
                     (long long)((LC.rowL >> 1) - P.fl_lo) * P.part_row_stride - P.avs;
        // tileX - avs is a multiple of 8, so an interior tile's row starts
        // on a 32-byte boundary whenever the planes' strides are multiples
        // of 4 floats and their base is 16-byte aligned: four vector stores
        const bool vec = ((P.part_row_stride | P.part_field_stride | P.part_class_stride) & 3) == 0 &&
                         (reinterpret_cast<uintptr_t>(P.partial) & 15) == 0 && tileX >= P.avs &&
                         tileX + 16 <= P.ave;
        if (vec) {
            float o[16];
#pragma unroll
            for (int x = 0; x < 8; x++) {
                o[x] = CS[x].x - CS[x].y;
                o[15 - x] = CS[x].x + CS[x].y;
            }
            float4 *d4 = reinterpret_cast<float4 *>(dst + tileX);
#pragma unroll
            for (int q = 0; q < 4; q++) d4[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        } else {
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const int X0 = tileX + x, X1 = tileX + 15 - x;
                if (X0 >= P.avs && X0 < P.ave) dst[X0] = CS[x].x - CS[x].y;
                if (X1 >= P.avs && X1 < P.ave) dst[X1] = CS[x].x + CS[x].y;
            }
        }
    }
}

// TMODE: 0 = one uniform threshold, 1 = per-bin table, 2 = per-frame
// thresholds (batches of captures). Guard-band decisions are taken in FP32 and
// recorded for tp3_resolve_kernel (an exact path inside this loop, however
// rarely taken, slows the whole walk by a third).
template <int TMODE>
__global__ void __launch_bounds__(32 * kWarps3, TMODE == 1 ? 3 : 4) tpal3d_kernel(T3Params P)
{
    constexpr bool PER_BIN = (TMODE == 1);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int ntiles = P.ntx * P.nty;
    extern __shared__ float4 s_dyn[];
    float4 *win = s_dyn + (size_t)warp * kWarpF4;
    float4 *carry_base = win + kWinF4;
    float4 *exch = carry_base + kCarryF4;
    float4 *R = exch + kExchF4;
    float2 *bnd = reinterpret_cast<float2 *>(R + kOutF4);
    float4 *tw = s_dyn + kWarps3 * kWarpF4;
    float *thr = reinterpret_cast<float *>(tw + kTwF4);   // [g][kz][lane], per-bin walks only
    if (PER_BIN)
        for (int i = threadIdx.x; i < 3 * 8 * 32; i += blockDim.x)
            thr[i] = P.thr_table[3 * ((((i >> 5) & 7) * 32 + kappa(i & 31)) * 3 + (i >> 8))];
    fill_twiddles(P, tw);
    // Work items (tile position, chunk of frames); a grid smaller than the
    // item count walks them persistently.
    const unsigned nitems = (unsigned)(ntiles * P.nchunks);
    for (unsigned w = blockIdx.x * kWarps3 + warp; w < nitems; w += gridDim.x * kWarps3) {
    const int item = (int)w;
    const int tile = item % ntiles;
    const int chunk = item / ntiles;
    const int tx = tile % P.ntx, ty = tile / P.ntx;
    const int tileX = P.tileX0 + 8 * tx;
    const int tileY = P.tileY0 + 16 * ty;
    const int m0 = P.frame_begin + chunk * P.chunk_frames;
    const int m1 = min(m0 + P.chunk_frames, P.frame_end);
    const int cls = ((ty & 1) << 1) | (tx & 1);
    const LaneConst LC = lane_const(P, lane, tileX, tileY);
    int last = -1;   // the item's latest record
    RowWords row;
    load_row(P, m0 - 2, LC, row);

    // Steps m0-5 .. m0-3 only fill the window (fields 2(m0-2) .. 2(m0-2)+5);
    // steps m0-2 and m0-1 also run the Z stage for the carries; the rest
    // output, each with the next step's forward stages (step m1: only that).
    for (int m = m0 - 5; m <= m1; m++) {
        __syncwarp();
        if (m < m1) x_forward(row, m + 3, LC, exch, bnd);   // fields 2m+6, 2m+7
        __syncwarp();
        if (m + 1 < m1) load_row(P, m + 4, LC, row);   // the next step's
        if (lane < 20) y_stages<true>(m + 3, LC, lane, win, exch, R, bnd, tw);
        __syncwarp();
        if (m > m0) x_inverse_store(P, LC, R, m - 1, tileX, cls);
        if (m < m0 - 2 || m == m1) continue;
        __syncwarp();   // the output rows have been read: R may be written

        const StepBounds SB = step_bounds(bnd, m, lane);
        float4 *carry = carry_base + (m & 1) * (5 * 32);
        const float tf_m = (TMODE == 2) ? P.frame_t2[3 * max(m, 0)] : P.t2f;   // uniform threshold of frame m

        // One decision: bin magnitude a against its mirror's b. Beside it a
        // screen for the guard band, an upper bound of the bin's band: with
        // ab <= sqrt(2 a), a band pa + t pb is at most
        // 2 sqrt(2) E (sqrt a + t sqrt b) + (1 + t) E^2
        // <= (1 + t) (2 sqrt(2) E sqrt(a + b) + E^2). The nearer margin is
        // the one of the smaller magnitude against t times the larger (for
        // t > 1 both tests fail unless both magnitudes are zero). A pair under
        // the limit of tiny pairs cannot be recorded. Only groups that pass
        // the screen run the bin-by-bin test (record_group).
        float e1, e2, lim;
        bool u;
        auto bounds = [&](float Em) {
            const float t1 = PER_BIN ? 1.f : 1.f + tf_m;
            e1 = 2.83f * t1 * Em;
            e2 = 1.01f * t1 * Em * Em;
            lim = kTinyPair - 2.01f * Em * Em;
            u = false;
        };
        auto similar = [&](float a, float b, float t) -> bool {
            const float d = __fmaf_rn(-fmaxf(a, b), t, fminf(a, b));
            const float s = a + b;
            const float band = __fmaf_rn(e1, sqrt_approx(s), e2);
            u |= (s >= lim) && (fabsf(d) <= (PER_BIN ? (1.f + t) * band : band));
            return d >= 0.f;
        };
        unsigned hits = 0;   // kx groups that reached the screen's bound

        // Pass 1: the pairs (kx 2, kx 6) in half-warp 0, (kx 3, kx 5) in half-warp 1
        {
            const int h = lane >> 4;
            float2 YA[8], YB[8], wz[4];
            z_window(wz, false);
            z_dft(win, m, h, LC.posA, wz, YA);
            z_dft(win, m, 4 - h, LC.posB, LC.wzB, YB);
            bounds(__shfl_sync(0xffffffffu, SB.em, h));
            float k[8], kh[8], kr[8], khr[8];   // at ky, at ky + 16; the same for the mirror column
            float ma[8], mb[8];
#pragma unroll
            for (int kz = 0; kz < 8; kz++) {
                ma[kz] = mag2(YA[kz]);
                mb[kz] = mag2(YB[kz]);
            }
#pragma unroll
            for (int kz = 0; kz < 8; kz++) {
                const int kzr = (10 - kz) & 7;
                const bool sim = similar(ma[kz], mb[kzr], PER_BIN ? thr[(8 * h + kz) * 32 + (lane & 15)] : tf_m);
                k[kz] = sim ? 1.f : 0.f;
                if (PER_BIN) {
                    const bool simh = similar(ma[kz ^ 4], mb[kzr ^ 4], thr[(8 * h + kz) * 32 + 16 + (lane & 15)]);
                    kh[kz] = simh ? 1.f : 0.f;
                }
            }
#pragma unroll
            for (int kz = 0; kz < 8; kz++) {
                kr[kz] = k[(10 - kz) & 7];
                khr[kz] = PER_BIN ? kh[(10 - kz) & 7] : 0.f;
            }
            z_inverse<!PER_BIN>(YA, k, kh, carry, R, h, lane & 15);
            z_inverse<!PER_BIN>(YB, kr, khr, carry, R, 4 - h, LC.laneB);
            const unsigned b = __ballot_sync(0xffffffffu, u);
            hits = ((b & 0xFFFFu) != 0 ? 1u : 0u) | (b >> 16 != 0 ? 2u : 0u);
        }
        // Pass 2: kx 4, whose mirror bins' magnitudes come from the lanes
        // that own them; all 32 ky.
        {
            const int laneB = LC.laneB ^ (lane & 16);
            float2 Y[8], wz[4];
            z_window(wz, lane >= 16);
            z_dft(win, m, 2, LC.posA, wz, Y);
            bounds(__shfl_sync(0xffffffffu, SB.em, 2));
            float2 y[8], o[4];
#pragma unroll
            for (int kz = 0; kz < 8; kz++) {
                const int kzr = (10 - kz) & 7;
                const float a = mag2(Y[kz]), b = __shfl_sync(0xffffffffu, mag2(Y[kzr]), laneB);
                bool sim = similar(a, b, PER_BIN ? thr[(16 + kz) * 32 + lane] : tf_m);
                if (PER_BIN) sim |= similar(a, b, thr[(16 + kzr) * 32 + laneB]);   // the mirror bin visits too
                if (kz == kzr) sim |= laneB == lane;   // a carrier (its own mirror) is always kept
                const float k = sim ? 1.f : 0.f;
                y[kz] = __fmul2_rn(Y[kz], make_float2(k, k));
            }
            z_rotate(y, o);
            ZInverse Z;
            Z.sum(y, o);
            const cp2 own = Z.finish(carry + 32 * 2 + lane);
            const cp2 high = {shfl_xor2(own.re, 16), shfl_xor2(own.im, 16)};
            if (lane < 16) R[20 * 2 + LC.posA] = f4_of(fold_ky(own, high));
            if (__any_sync(0xffffffffu, u)) hits |= 4u;
        }
        if (hits != 0) {   // one copy of the rare path
#pragma unroll 1
            for (int g = 0; g < 3; g++) {
                if (!(hits >> g & 1)) continue;
                const float ekA = __shfl_sync(0xffffffffu, SB.ek, g), ekB = __shfl_sync(0xffffffffu, SB.ek, 4 - g);
                record_group<PER_BIN>(P, LC, win, thr, item, m, g, lane, tf_m, ekA, ekB, last);
            }
        }
    }
    __syncwarp();   // the next item reuses this warp's shared window
    }
}

// ---------------------------------------------------------------------------
// Learned-mask form: feature pass and apply pass
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint16_t bf16_bits(float x)
{
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t *>(&h);
}

// PASS 0: features (+ spectrum, + threshold decisions) of every Z tile the
// walk computes; PASS 1: the same walk with each bin scaled by its fraction
// (or, on fallback tiles, masked by the FP32 threshold decisions), then the
// inverse and overlap-add of the plain walk.
// Four blocks an SM, as the walk: 12 frames' tiles are two waves instead of three
// (the learned clip 2,058 -> 2,010 us).
template <int PASS>
__global__ void __launch_bounds__(32 * kWarps3, 4) tpal3d_learned_kernel(T3Params P, T3Learn L)
{
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int ntiles = P.ntx * P.nty;
    extern __shared__ float4 s_dyn[];
    float4 *win = s_dyn + (size_t)warp * kWarpF4;
    float4 *carry_base = win + kWinF4;
    float4 *exch = carry_base + kCarryF4;
    float4 *R = exch + kExchF4;
    float2 *bnd = reinterpret_cast<float2 *>(R + kOutF4);
    float4 *tw = s_dyn + kWarps3 * kWarpF4;
    fill_twiddles(P, tw);
    const unsigned nitems = (unsigned)(ntiles * P.nchunks);
    for (unsigned w = blockIdx.x * kWarps3 + warp; w < nitems; w += gridDim.x * kWarps3) {
    const int item = (int)w;
    const int tile = item % ntiles;
    const int chunk = item / ntiles;
    const int tx = tile % P.ntx, ty = tile / P.ntx;
    const int tileX = P.tileX0 + 8 * tx;
    const int tileY = P.tileY0 + 16 * ty;
    const int m0 = P.frame_begin + chunk * P.chunk_frames;
    const int m1 = min(m0 + P.chunk_frames, P.frame_end);
    const int cls = ((ty & 1) << 1) | (tx & 1);
    const LaneConst LC = lane_const(P, lane, tileX, tileY);

    RowWords row;
    load_row(P, m0 - 2, LC, row);
    for (int m = m0 - 5; m <= m1; m++) {
        __syncwarp();
        if (m < m1) x_forward(row, m + 3, LC, exch, bnd);
        __syncwarp();
        if (m + 1 < m1) load_row(P, m + 4, LC, row);
        if (lane < 20) y_stages<PASS == 1>(m + 3, LC, lane, win, exch, R, bnd, tw);
        __syncwarp();
        if (PASS == 1 && m > m0) x_inverse_store(P, LC, R, m - 1, tileX, cls);
        if (m < m0 - 2 || m == m1) continue;
        __syncwarp();
        const long long base = ((long long)(m - L.z0) * ntiles + tile) * 1280;
        float4 *carry = carry_base + (m & 1) * (5 * 32);
        const bool fb = (PASS == 1) ? (L.fallback[(long long)(m - L.z0) * ntiles + tile] != 0) : false;
        // the walk's two passes: the column pairs of both half-warps, then
        // kx 4 (both half-warps at ky < 16; half-warp 0 writes)
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
            const int h = lane >> 4;
            const int ka = pass == 0 ? h : 2, kb = 4 - ka;
            float2 YA[8], YB[8], wz[4];
            z_window(wz, false);
            z_dft(win, m, ka, LC.posA, wz, YA);
            z_dft(win, m, kb, LC.posB, LC.wzB, YB);
            const int kyr = (40 - LC.ky) & 31;
            const long long va = base + ka * 256 + LC.ky, vb = base + kb * 256 + kyr;
            const int hb = kyr < 16 ? 16 : -16;   // from the mirror ky to its other half
            const bool wa = pass == 0 || h == 0, wb = pass == 0;   // column A, column B written
            unsigned keep = 0;   // FP32 decisions: bit kz = column A's bin kz and column B's (10 - kz) & 7
            if (PASS == 0 ? L.plain_p != nullptr : fb) {
#pragma unroll
                for (int kz = 0; kz < 8; kz++) {
                    const int kzr = (10 - kz) & 7;
                    const bool self = pass == 1 && kz == kzr && LC.ky == kyr;
                    if (fsim(mag2(YA[kz]), mag2(YB[kzr]), P.t2f) || self) keep |= 1u << kz;
                }
            }
            if (PASS == 0) {
#pragma unroll
                for (int kz = 0; kz < 8; kz++) {
                    const int v = 32 * kz, vm = 32 * (kz ^ 4);
                    if (wa) {
                        const uint16_t f = bf16_bits(log1pf(sqrtf(mag2(YA[kz]))) * 0.0625f);
                        L.feat[va + v] = f;
                        L.feat[va + vm + 16] = f;
                    }
                    if (wb) {
                        const uint16_t f = bf16_bits(log1pf(sqrtf(mag2(YB[kz]))) * 0.0625f);
                        L.feat[vb + v] = f;
                        L.feat[vb + vm + hb] = f;
                    }
                }
                if (L.spec != nullptr) {
                    const float s = ((P.swap ^ P.tileY0) & 1) ? -1.f : 1.f;   // the sign of ky >= 16
                    const float sb = kyr < 16 ? 1.f : s, sm = kyr < 16 ? s : 1.f;
#pragma unroll
                    for (int kz = 0; kz < 8; kz++) {
                        const int v = 32 * kz, vm = 32 * (kz ^ 4);
                        if (wa) {
                            L.spec[va + v] = YA[kz];
                            L.spec[va + vm + 16] = make_float2(s * YA[kz].x, s * YA[kz].y);
                        }
                        if (wb) {
                            L.spec[vb + v] = make_float2(sb * YB[kz].x, sb * YB[kz].y);
                            L.spec[vb + vm + hb] = make_float2(sm * YB[kz].x, sm * YB[kz].y);
                        }
                    }
                }
                if (L.plain_p != nullptr) {
#pragma unroll
                    for (int kz = 0; kz < 8; kz++) {
                        const int kzr = (10 - kz) & 7;
                        const float p = (float)((keep >> kz) & 1u);
                        if (wa) L.plain_p[va + 32 * kz] = L.plain_p[va + 32 * (kz ^ 4) + 16] = p;
                        if (wb) L.plain_p[vb + 32 * kzr] = L.plain_p[vb + 32 * (kzr ^ 4) + hb] = p;
                    }
                }
            } else {
                float k[8], kh[8], kr[8], khr[8];
#pragma unroll
                for (int kz = 0; kz < 8; kz++) {
                    const int kzr = (10 - kz) & 7;
                    if (fb) {
                        k[kz] = (float)((keep >> kz) & 1u);
                        kh[kz] = (float)((keep >> (kz ^ 4)) & 1u);
                        kr[kz] = (float)((keep >> kzr) & 1u);
                        khr[kz] = (float)((keep >> (kzr ^ 4)) & 1u);
                    } else {
                        k[kz] = __ldg(L.p + va + 32 * kz);
                        kh[kz] = __ldg(L.p + va + 32 * kz + 16);
                        kr[kz] = wb ? __ldg(L.p + vb + 32 * kz) : 0.f;
                        khr[kz] = wb ? __ldg(L.p + vb + 32 * kz + hb) : 0.f;
                    }
                }
                if (wa) z_inverse<false>(YA, k, kh, carry, R, ka, lane & 15);
                if (wb) z_inverse<false>(YB, kr, khr, carry, R, kb, LC.laneB);
            }
        }
    }
    __syncwarp();
    }
}

int tp3_learned_launch(const T3Params &P, const T3Learn &L, int pass, cudaStream_t stream)
{
    const long long items = (long long)P.ntx * P.nty * P.nchunks;
    if (items <= 0) return 0;
    const unsigned blocks = (unsigned)((items + kWarps3 - 1) / kWarps3);
    const size_t smem = walk_smem(false);
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -1;
    if (!attr_set[dev]) {
        const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (cudaFuncSetAttribute(tpal3d_learned_kernel<0>, a, (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(tpal3d_learned_kernel<1>, a, (int)smem) != cudaSuccess)
            return -1;
        attr_set[dev] = true;
    }
    if (pass == 0) {
        if (L.feat == nullptr) return -1;
        tpal3d_learned_kernel<0><<<blocks, 32 * kWarps3, smem, stream>>>(P, L);
    } else {
        if (L.p == nullptr || L.fallback == nullptr || P.partial == nullptr) return -1;
        tpal3d_learned_kernel<1><<<blocks, 32 * kWarps3, smem, stream>>>(P, L);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// ---------------------------------------------------------------------------
// Deferred exact decisions
// ---------------------------------------------------------------------------
// One warp per record: decide its guard-band bins exactly and, where an exact
// decision differs from the FP32 one the walk used, correct the record's
// decisions and list it for tpal3d_exact_kernel. The X stage of the record's two kx
// columns is computed once for all its bins; lane (z, part) owns rows
// 4 part .. 4 part + 3 of field 2m + z. A bin at (kz + 4, ky + 16) has the
// magnitudes of the bin at (kz, ky) (see the walk), so both are decided from
// one evaluation.
//
// Bound by integer multiplies: 256 for a record's X stage, 96 a bin a lane.
// 615 -> 258 us for a 500-field capture (90 -> 38 us for 60); double-float Y
// and Z stages, which this replaces, took about 1,500 instructions a bin, and
// ran twice, for ky and ky + 16.
__global__ void __launch_bounds__(32 * kWarps3) tp3_resolve_kernel(T3Params P)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned n = min(P.counters[0], P.unc_cap);
    if (blockIdx.x * kWarps3 >= n) return;
    unsigned n_exact = 0, n_flip = 0;
    const int z = lane >> 2, part = lane & 3;
    extern __shared__ int4 s_qyz[];
    for (int i = threadIdx.x; i < kQYZ; i += blockDim.x) s_qyz[i] = g3_qyz[i];
    __syncthreads();
    for (unsigned rec = blockIdx.x * kWarps3 + warp; rec < n; rec += gridDim.x * kWarps3) {
        UncRecord &R = P.unc_rec[rec];
        const int tile = R.item % (P.ntx * P.nty), m = R.mg >> 2, g = R.mg & 3;
        const int tileX = P.tileX0 + 8 * (tile % P.ntx), tileY = P.tileY0 + 16 * (tile / P.ntx);
        const int kxa = 2 + g;
        unsigned keep = R.keep[lane];
        const unsigned unc = R.unc[lane];
        const int f = 2 * m + z;
        const int p = (f & 1) ^ P.swap;
        const int y0 = (p - tileY) & 1;
        fx2 xa[4], xb[4];
        const uint16_t *fp = (f >= 0 && f < P.nfields) ? field_at(P, f) : nullptr;
#pragma unroll
        for (int r4 = 0; r4 < 4; r4++) {
            xa[r4] = xb[r4] = {0, 0, 0, 0};
            const int L = tileY + y0 + 2 * (part * 4 + r4);
            if (fp == nullptr || L < P.fafl || L > P.lafl) continue;
            const long long base = (long long)(L >> 1) * P.fw + tileX;   // within the field
            x_row_pair(fp, base, (long long)P.fh * P.fw, P.black, kxa, xa[r4], xb[r4]);
        }
        // bins of ky < 16 to evaluate: this lane's own and those of ky + 16 moved by 4
        const unsigned up = __shfl_xor_sync(0xffffffffu, unc, 16);
        unsigned todo = lane < 16 ? unc | ((up << 4 | up >> 4) & 0xFFu) : 0u;
        bool flipped = false;
        unsigned any = __ballot_sync(0xffffffffu, todo != 0);
        while (any) {
            const int src = __ffs(any) - 1;
            const int kz = __ffs(__shfl_sync(0xffffffffu, todo, src)) - 1;
            const int ky = kappa(src), kzr = (10 - kz) & 7, kyr = (40 - ky) & 31;
            fxsum b = {0, 0, 0, 0}, r = b;
            const int4 *q = s_qyz + (z < 4 ? z : 7 - z) * (16 * 32);
#pragma unroll
            for (int r4 = 0; r4 < 4; r4++) {
                const int y = y0 + 2 * (part * 4 + r4);
                const int4 *c = q + (y < 16 ? y : 31 - y) * 32;
                b.mac(xa[r4], c[(ky * y + 4 * kz * z) & 31]);
                r.mac(xb[r4], c[(kyr * y + 4 * kzr * z) & 31]);
            }
            // the sums of the 32 lanes, in units of 2^-38: lanes 0-7 end with
            // the bin's real part, 8-15 its imaginary part, 16-31 the mirror's
            const long long v0 = (b.rh >> 2) + (b.rm >> 31), v1 = (b.ih >> 2) + (b.im >> 31);
            const long long v2 = (r.rh >> 2) + (r.rm >> 31), v3 = (r.ih >> 2) + (r.im >> 31);
            const bool h16 = lane & 16, h8 = lane & 8;
            const long long s0 = (h16 ? v2 : v0) + shfl_xor_i64(h16 ? v0 : v2, 16);
            const long long s1 = (h16 ? v3 : v1) + shfl_xor_i64(h16 ? v1 : v3, 16);
            long long s = (h8 ? s1 : s0) + shfl_xor_i64(h8 ? s0 : s1, 8);
#pragma unroll
            for (int h = 4; h >= 1; h >>= 1) s += shfl_xor_i64(s, h);
            const df v = df_from_i64(s);
            const df sq = df_mul({v.hi * 3.637978807091713e-12f, v.lo * 3.637978807091713e-12f},   // 2^-38
                                 {v.hi * 3.637978807091713e-12f, v.lo * 3.637978807091713e-12f});
            const df mag = df_add(sq, df_shfl_xor(sq, 8));
            const df oth = df_shfl_xor(mag, 16);
            const df mb = h16 ? oth : mag, mr = h16 ? mag : oth;
            bool sim = df_sim(mb, mr, thr_of(P, m, kz, ky, kxa).d);
            if (kxa == 4) sim |= df_sim(mb, mr, thr_of(P, m, kzr, kyr, 4).d);
            bool simh = sim;   // of (kz + 4, ky + 16)
            if (P.thr_table != nullptr) {
                simh = df_sim(mb, mr, thr_of(P, m, kz ^ 4, ky + 16, kxa).d);
                if (kxa == 4) simh |= df_sim(mb, mr, thr_of(P, m, kzr ^ 4, kyr ^ 16, 4).d);
            }
            // the bins decided: this one, its copy at ky + 16, and for kx = 4
            // the mirrors of both, which visit too
            const int lr = kappa(kyr);
            const unsigned bit = 1u << kz, bith = 1u << (kz ^ 4), bitr = 1u << kzr, bitrh = 1u << (kzr ^ 4);
            if (g == 2) {
                if (lane == lr) todo &= ~bitr;
                if (lane == (lr ^ 16)) todo &= ~bitrh;
            }
            if (lane == src) {
                todo &= ~bit;
                const bool was = keep & bit;
                n_exact += (unc & bit) != 0;
                if (was != sim) {
                    n_flip++;
                    keep ^= bit;
                    flipped = true;
                }
            }
            if (lane == src + 16) {
                const bool was = keep & bith;
                n_exact += (unc & bith) != 0;
                if (was != simh) {
                    n_flip++;
                    keep ^= bith;
                    flipped = true;
                }
            }
            if (g == 2 && lane == lr) keep = sim ? keep | bitr : keep & ~bitr;
            if (g == 2 && lane == (lr ^ 16)) keep = simh ? keep | bitrh : keep & ~bitrh;
            any = __ballot_sync(0xffffffffu, todo != 0);
        }
        if (__any_sync(0xffffffffu, flipped)) {   // tpal3d_exact_kernel takes this group's decisions from the record
            R.keep[lane] = (uint8_t)keep;
            if (lane == 0) {
                const unsigned at = atomicAdd(P.counters + 1, 1u);
                if (at < P.unc_cap) P.rerun[at] = rec;   // at most one entry per record
            }
        }
    }
    if (P.stats != nullptr) {
        if (n_exact) atomicAdd(P.stats + 0, n_exact);
        if (n_flip) atomicAdd(P.stats + 1, n_flip);
    }
}

// ---------------------------------------------------------------------------
// The outputs that corrected decisions reach, once more
// ---------------------------------------------------------------------------
// The record of (step m, kx group g) in the list of `rec`'s item, or -1.
__device__ __forceinline__ int find_record(const T3Params &P, int rec, int mg)
{
    int at = rec;
    while (at >= 0 && P.unc_rec[at].mg > mg) at = P.unc_rec[at].prev;
    while (at >= 0 && P.unc_rec[at].mg < mg) at = P.unc_rec[at].next;
    return at >= 0 && P.unc_rec[at].mg == mg ? at : -1;
}

// Two outputs per corrected record, the one of its own step mf and the one its
// carries feed (step mf + 2), recomputed with the decisions of the corrected
// records; they are written where the walk wrote them. The operations and
// their order are the walk's.
//
// There are few of them, so what counts is how long one takes: a block owns an
// output, its six pairs of fields are transformed by a warp each (a seventh
// looks the records up), the Z stages of the two tiles that meet in the output
// by four. 31 -> 8.4 us for a few outputs (the walk's own loop over the steps, a
// warp an output), 30 -> 15 us for a 200-field capture, 20 for the 900 corrected
// decisions of a 500-field one.
constexpr int kWarpsX = 7;
constexpr int kPairsX = 6;
template <int TMODE>
__global__ void __launch_bounds__(32 * kWarpsX, 2) tpal3d_exact_kernel(T3Params P)
{
    constexpr bool PER_BIN = (TMODE == 1);
    __shared__ float4 win[kPairsX * 80 + 80];   // one more, for the output's unused forward stage
    __shared__ float4 exch[kPairsX * kExchF4], carry[5 * 32], R[kOutF4], tw[kTwF4];
    __shared__ float2 bnd[(kPairsX + 1) * 8];
    __shared__ float thr[PER_BIN ? 3 * 8 * 32 : 1];
    __shared__ uint8_t s_keep[2][3][32];        // decisions of step mo (0) and mo - 2 (1) per kx group
    __shared__ int s_fix[2][3];                 // their records, or -1
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nitems = 2 * min(P.counters[1], P.unc_cap);
    if (blockIdx.x >= nitems) return;
    const int ntiles = P.ntx * P.nty;
    if (PER_BIN)
        for (int i = threadIdx.x; i < 3 * 8 * 32; i += blockDim.x)
            thr[i] = P.thr_table[3 * ((((i >> 5) & 7) * 32 + kappa(i & 31)) * 3 + (i >> 8))];
    fill_twiddles(P, tw);
    for (unsigned w = blockIdx.x; w < nitems; w += gridDim.x) {
        const int rec = (int)P.rerun[w >> 1];
        const int item = P.unc_rec[rec].item, tile = item % ntiles, chunk = item / ntiles;
        const int tx = tile % P.ntx, ty = tile / P.ntx;
        const int tileX = P.tileX0 + 8 * tx, tileY = P.tileY0 + 16 * ty;
        const int mo = (P.unc_rec[rec].mg >> 2) + 2 * (int)(w & 1);
        const int m0 = P.frame_begin + chunk * P.chunk_frames;
        if (mo < m0 || mo >= min(m0 + P.chunk_frames, P.frame_end)) continue;   // the whole block
        const LaneConst LC = lane_const(P, lane, tileX, tileY);
        if (warp < kPairsX) {   // pair mo - 2 + warp
            RowWords row;
            load_row(P, mo - 2 + warp, LC, row);
            x_forward(row, 0, LC, exch + kExchF4 * warp, bnd + 8 * warp);
            __syncwarp();
            if (lane < 20) y_stages<false>(0, LC, lane, win + 80 * warp, exch + kExchF4 * warp, R, bnd + 8 * warp, tw);
        } else {
            const int st = lane / 3, g = lane % 3;
            const int at = lane < 6 ? find_record(P, rec, (mo - 2 * st) * 4 + g) : -1;
            if (lane < 6) s_fix[st][g] = at;
#pragma unroll
            for (int i = 0; i < 6; i++) {
                const int r = __shfl_sync(0xffffffffu, at, i);
                if (r >= 0) s_keep[i / 3][i % 3][lane] = P.unc_rec[r].keep[lane];
            }
        }
        __syncthreads();
        // warps 0, 1: pass 1 and pass 2 of step mo; 2, 3: of step mo - 2
        const int st = warp >> 1, pass = warp & 1;
        const int h = lane >> 4;
        ZInverse Z[4];   // pass 1: column kx = 2 + h at ky and ky + 16, the mirror column likewise; pass 2: kx = 4
        if (warp < 4) {
            const float4 *tile4 = win + (st == 0 ? 2 * 80 : 0);
            const int m = mo - 2 * st;
            const float tf_m = (TMODE == 2) ? P.frame_t2[3 * max(m, 0)] : P.t2f;
            auto similar = [](float a, float b, float t) -> bool { return __fmaf_rn(-fmaxf(a, b), t, fminf(a, b)) >= 0.f; };
            float2 wz[4], y[8], o[4];
            if (pass == 0) {
                float2 YA[8], YB[8];
                z_window(wz, false);
                z_dft(tile4, 0, h, LC.posA, wz, YA);
                z_dft(tile4, 0, 4 - h, LC.posB, LC.wzB, YB);
                const bool fixed = s_fix[st][h] >= 0;
                const unsigned fl = s_keep[st][h][lane & 15], fh = s_keep[st][h][16 + (lane & 15)];
                float k[8], kh[8];
#pragma unroll
                for (int kz = 0; kz < 8; kz++) {
                    const int kzr = (10 - kz) & 7;
                    bool sim = similar(mag2(YA[kz]), mag2(YB[kzr]), PER_BIN ? thr[(8 * h + kz) * 32 + (lane & 15)] : tf_m);
                    if (fixed) sim = (fl >> kz) & 1u;
                    k[kz] = sim ? 1.f : 0.f;
                    if (PER_BIN) {
                        bool simh = similar(mag2(YA[kz ^ 4]), mag2(YB[kzr ^ 4]), thr[(8 * h + kz) * 32 + 16 + (lane & 15)]);
                        if (fixed) simh = (fh >> kz) & 1u;
                        kh[kz] = simh ? 1.f : 0.f;
                    }
                }
                // masked by k; at ky + 16 by k moved by 4 or, per bin, kh
                auto sums = [&](const float2 (&Y)[8], bool mirror, ZInverse &lo, ZInverse &hi) {
#pragma unroll
                    for (int z = 0; z < 8; z++) {
                        const float kk = mirror ? k[(10 - z) & 7] : k[z];
                        y[z] = __fmul2_rn(Y[z], make_float2(kk, kk));
                    }
                    z_rotate(y, o);
                    lo.sum(y, o);
                    if constexpr (PER_BIN) {
#pragma unroll
                        for (int z = 0; z < 8; z++) {
                            const float kk = mirror ? kh[(10 - z) & 7] : kh[z];
                            y[z] = __fmul2_rn(Y[z ^ 4], make_float2(kk, kk));
                        }
                        z_rotate(y, o);
                        hi.sum(y, o);
                    } else {
                        hi.sum_moved(y, o);
                    }
                };
                sums(YA, false, Z[0], Z[1]);
                sums(YB, true, Z[2], Z[3]);
            } else {
                const int laneB = LC.laneB ^ (lane & 16);
                float2 Y[8];
                z_window(wz, lane >= 16);
                z_dft(tile4, 0, 2, LC.posA, wz, Y);
                const bool fixed = s_fix[st][2] >= 0;
                const unsigned f = s_keep[st][2][lane];
#pragma unroll
                for (int kz = 0; kz < 8; kz++) {
                    const int kzr = (10 - kz) & 7;
                    const float a = mag2(Y[kz]), b = __shfl_sync(0xffffffffu, mag2(Y[kzr]), laneB);
                    bool sim = similar(a, b, PER_BIN ? thr[(16 + kz) * 32 + lane] : tf_m);
                    if (PER_BIN) sim |= similar(a, b, thr[(16 + kzr) * 32 + laneB]);   // the mirror bin visits too
                    if (kz == kzr) sim |= laneB == lane;   // a carrier (its own mirror) is always kept
                    if (fixed) sim = (f >> kz) & 1u;
                    const float k = sim ? 1.f : 0.f;
                    y[kz] = __fmul2_rn(Y[kz], make_float2(k, k));
                }
                z_rotate(y, o);
                Z[0].sum(y, o);
            }
        }
        // where Z[i] meets its carry
        auto slot = [&](int i) -> float4 * {
            if (pass == 1) return carry + 32 * 2 + lane;
            const int at = i < 2 ? lane & 15 : LC.laneB;
            return carry + 32 * (i < 2 ? h : 4 - h) + ((i & 1) ? at ^ 16 : at);
        };
        if (warp == 2 || warp == 3) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (pass == 0 || i == 0) *slot(i) = Z[i].later();
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int at = c == 0 ? lane & 15 : LC.laneB, col = c == 0 ? h : 4 - h;
                const cp2 a = Z[2 * c].finish(slot(2 * c)), b = Z[2 * c + 1].finish(slot(2 * c + 1));
                cp2 g = fold_ky(a, b);
                if (at >= 16) {   // a is the upper half: component 1 is b - a
                    g.re.y = -g.re.y;
                    g.im.y = -g.im.y;
                }
                R[20 * col + swz(at & 15)] = f4_of(g);
            }
        } else if (warp == 1) {
            const cp2 own = Z[0].finish(slot(0));
            const cp2 high = {shfl_xor2(own.re, 16), shfl_xor2(own.im, 16)};
            if (lane < 16) R[20 * 2 + LC.posA] = f4_of(fold_ky(own, high));
        }
        __syncthreads();
        if (warp == 0) {
            if (lane < 20) y_stages<true>(0, LC, lane, win + 80 * kPairsX, exch, R, bnd + 8 * kPairsX, tw);
            __syncwarp();
            x_inverse_store(P, LC, R, mo, tileX, ((ty & 1) << 1) | (tx & 1));
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static double rc_window(int n, int N) { return 0.5 - (0.5 * cos((2 * M_PI * (n + 0.5)) / N)); }

int tp3_init_constants(int device)
{
    if (device >= 0 && device < 64 && g_tp3_constants_ready[device]) return 0;
    float cwx[5][8], swx[5][8], cix[5][8], six[5][8];
    for (int k = 0; k < 5; k++) {
        const int kx = k + 2;
        for (int x = 0; x < 8; x++) {
            const double th = 2.0 * M_PI * kx * (x - 7.5) / 16.0;
            const double w = rc_window(x, 16);
            cwx[k][x] = (float)(w * cos(th));
            swx[k][x] = (float)(w * sin(th));
            cix[k][x] = (float)((2.0 / 4096.0) * cos(th));
            six[k][x] = (float)((2.0 / 4096.0) * sin(th));
        }
    }
    float wy[2][16], wx[16], wz[8];
    for (int y0 = 0; y0 < 2; y0++)
        for (int i = 0; i < 16; i++) wy[y0][i] = (float)rc_window(y0 + 2 * i, 32);
    for (int x = 0; x < 16; x++) wx[x] = (float)rc_window(x, 16);
    for (int z = 0; z < 8; z++) wz[z] = (float)rc_window(z, 8);
    float2 tw16[16], tw32[32];
    for (int r = 0; r < 16; r++) tw16[r] = make_float2((float)cos(-2 * M_PI * r / 16), (float)sin(-2 * M_PI * r / 16));
    for (int r = 0; r < 32; r++) tw32[r] = make_float2((float)cos(-2 * M_PI * r / 32), (float)sin(-2 * M_PI * r / 32));
    std::vector<int4> qyz(kQYZ);
    int qx[5][16][4];
    for (int k = 0; k < 5; k++)
        for (int x = 0; x < 16; x++) {
            const double w = rc_window(x, 16);
            const double a = -2.0 * M_PI * (k + 2) * x / 16.0;
            const double parts[2] = {w * cos(a), w * sin(a)};
            for (int c = 0; c < 2; c++) {
                const long long q = llround(parts[c] * 1152921504606846976.0);   // 2^60
                qx[k][x][2 * c] = (int)(q >> 30);                               // floor(q / 2^30)
                qx[k][x][2 * c + 1] = (int)(q & ((1LL << 30) - 1));
            }
        }
    for (int e = 0; e < kQYZ; e++) {
        const int z = e / (16 * 32), y = (e / 32) % 16, r = e % 32;
        const double w = rc_window(z, 8) * rc_window(y, 32), an = -2.0 * M_PI * r / 32;
        int w4[4];
        const double parts[2] = {w * cos(an), w * sin(an)};
        for (int c = 0; c < 2; c++) {
            const long long q = llround(parts[c] * 576460752303423488.0);   // 2^59
            w4[2 * c] = (int)(q >> 29);
            w4[2 * c + 1] = (int)(q & ((1LL << 29) - 1));
        }
        qyz[e] = make_int4(w4[0], w4[1], w4[2], w4[3]);
    }
#define TPAL_CPY(sym, src)                                                  \
    if (cudaMemcpyToSymbol(sym, src, sizeof(src)) != cudaSuccess) return -1;
    float2 xf[5][8], xi[5][8];
    for (int k = 0; k < 5; k++)
        for (int x = 0; x < 8; x++) {
            xf[k][x] = make_float2(cwx[k][x], -swx[k][x]);
            xi[k][x] = make_float2(cix[k][x], six[k][x]);
        }
    TPAL_CPY(c3_xf, xf);
    TPAL_CPY(c3_xi, xi);
    TPAL_CPY(c3_wy, wy);
    TPAL_CPY(c3_wx, wx);
    TPAL_CPY(c3_wz, wz);
    TPAL_CPY(c3_tw16, tw16);
    TPAL_CPY(c3_tw32, tw32);
    TPAL_CPY(c3_qx, qx);
    if (cudaMemcpyToSymbol(g3_qyz, qyz.data(), sizeof(int4) * kQYZ) != cudaSuccess) return -1;
#undef TPAL_CPY
    if (device >= 0 && device < 64) g_tp3_constants_ready[device] = true;
    return 0;
}

int tp3_launch(const T3Params &P, cudaStream_t stream, int max_blocks)
{
    const long long items = (long long)P.ntx * P.nty * P.nchunks;
    if (items <= 0) return 0;
    unsigned blocks = (unsigned)((items + kWarps3 - 1) / kWarps3);
    if (max_blocks > 0 && blocks > (unsigned)max_blocks) blocks = (unsigned)max_blocks;   // persistent grid
    const size_t smem = walk_smem(P.thr_table != nullptr);
    // function attributes are per device
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -1;
    if (!attr_set[dev]) {
        const int b = (int)walk_smem(true);
        const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (cudaFuncSetAttribute(tpal3d_kernel<0>, a, b) != cudaSuccess ||
            cudaFuncSetAttribute(tpal3d_kernel<1>, a, b) != cudaSuccess ||
            cudaFuncSetAttribute(tpal3d_kernel<2>, a, b) != cudaSuccess)
            return -1;
        attr_set[dev] = true;
    }
    if (P.unc_rec == nullptr || P.counters == nullptr || P.rerun == nullptr) return -1;
    const unsigned t = 32 * kWarps3;
    if (P.thr_table != nullptr) tpal3d_kernel<1><<<blocks, t, smem, stream>>>(P);
    else if (P.frame_t2 != nullptr) tpal3d_kernel<2><<<blocks, t, smem, stream>>>(P);
    else tpal3d_kernel<0><<<blocks, t, smem, stream>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int tp3_resolve_launch(const T3Params &P, cudaStream_t stream)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    // the record and item counts are only known on the device: fixed grids
    // walk them
    tp3_resolve_kernel<<<4 * sms, 32 * kWarps3, sizeof(int4) * kQYZ, stream>>>(P);
    const unsigned t = 32 * kWarpsX, blocks = 2u * (unsigned)sms;
    if (P.thr_table != nullptr) tpal3d_exact_kernel<1><<<blocks, t, 0, stream>>>(P);
    else if (P.frame_t2 != nullptr) tpal3d_exact_kernel<2><<<blocks, t, 0, stream>>>(P);
    else tpal3d_exact_kernel<0><<<blocks, t, 0, stream>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace tpal
