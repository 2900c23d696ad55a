// Texture window energies on larger windows, in three arithmetics, for the precision study (no counterpart in the
// reference, which sums FP32 box means on fixed 16 x 16 windows, src/kernels.cu:331-428).
//
// The box sums behind the figures (3 x 3 and 9 x 9 sums of luma, with the picture's edge pixels repeated) are made three
// ways: as exact integers from the pixels, and from a summed-area table of each picture in FP32 with two-sum
// compensation (a (hi, lo) pair per entry; Knuth's TwoSum) and in plain FP32. From them each pixel's fine detail y - S3/9, mid detail S3/9 - S9/81 and
// box-3 gradients are formed: as exact integer numerators in the exact form; in the compensated form as the same
// numerators in FP32 (9 y - S3, 9 S3 - S9 and differences of S3 are integers below 2^24, so exact) divided once; in the
// plain form as FP32 code usually does, from FP32 box means (y - S3/9, S3/9 - S9/81), which cancel. Their products are
// summed per 16 x 16 block (int64; FP32 with Neumaier's compensation; plain FP32). Windows of 16 k pixels sum k x k
// blocks in the same arithmetic and give the 8 figures of src/kernels.cu:340-341 as doubles.
#include <type_traits>

#include "es_kernels.h"

namespace es {
namespace {

constexpr int kQ = 12;  // per block: fine_r^2, mid_r^2, fine_d^2, mid_d^2, fine_r fine_d, mid_r mid_d, Jxx_r, Jyy_r, Jxy_r, Jxx_d, Jyy_d, Jxy_d

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Neumaier's compensated accumulator
struct Comp {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x)
    {
        float t, e;
        two_sum(s, x, t, e);
        s = t;
        c = __fadd_rn(c, e);
    }
    __device__ __forceinline__ float value() const { return __fadd_rn(s, c); }
};

// ---- tables ------------------------------------------------------------------------------------------------------------
// A table entry is the row prefix of column prefixes, each a chain of additions in a fixed order whose roundings are the
// point of the study. Down a column the sums are whole numbers below 2^24 for up to kExactRows rows of 10-bit values, so
// FP32 adds them exactly, compensated or not, in any order: band_sums_kernel / band_prefix_kernel make them per band of
// 32 rows as integers. sat_band_kernel then scans a band: one warp holds a row per lane and adds along x in order (the
// chain of additions that bounds it: about 20 cycles a column), while two warps make the next columns' prefixes in
// shared memory, their pixels read one chunk ahead, and five store the last columns' entries, a row at a time. The form
// this replaces had one thread per column, then one per row reading and writing rows w apart: 8.6 ms for two pictures of
// 3840 x 2160, against 0.16 ms.
constexpr int kBand = 32, kChunkX = 64, kSatThreads = 256;
constexpr int kExactRows = 16384;

struct SatJob {
    const uint16_t *y;
    unsigned *band;  // [bands][w]: first the bands' column sums, then the sums of all rows above the band
    float *shi, *slo, *sp;
};
struct SatPair {
    SatJob job[2];
    int w, h, up;
};

__global__ void __launch_bounds__(256) band_sums_kernel(const __grid_constant__ SatPair p)
{
    const int x = blockIdx.x * 256 + threadIdx.x, r0 = blockIdx.y * kBand;
    if (x >= p.w) return;
    const SatJob &J = p.job[blockIdx.z];
    unsigned a = 0;
#pragma unroll 8
    for (int r = r0; r < min(r0 + kBand, p.h); r++) a += (unsigned)__ldg(J.y + (size_t)r * p.w + x) << p.up;
    J.band[(size_t)blockIdx.y * p.w + x] = a;
}

__global__ void __launch_bounds__(64) band_prefix_kernel(const __grid_constant__ SatPair p, int bands)
{
    const int x = blockIdx.x * 64 + threadIdx.x;
    if (x >= p.w) return;
    unsigned *v = p.job[blockIdx.y].band + x;
    unsigned a = 0;
    int b = 0;
    for (; b + 8 <= bands; b += 8) {  // eight loads in flight
        unsigned q[8];
#pragma unroll
        for (int k = 0; k < 8; k++) q[k] = v[(size_t)(b + k) * p.w];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            v[(size_t)(b + k) * p.w] = a;
            a += q[k];
        }
    }
    for (; b < bands; b++) {
        const unsigned q = v[(size_t)b * p.w];
        v[(size_t)b * p.w] = a;
        a += q;
    }
}

struct SatSmem {
    float c[2][kChunkX][kBand + 1];       // column prefixes [column][row]
    float out[2][3][kChunkX][kBand + 1];  // entries: hi, lo, plain
};

__global__ void __launch_bounds__(kSatThreads) sat_band_kernel(const __grid_constant__ SatPair p)
{
    extern __shared__ __align__(16) unsigned char sat_dyn[];
    SatSmem &sm = *(SatSmem *)sat_dyn;
    const SatJob &J = p.job[blockIdx.y];
    const int w = p.w, r0 = blockIdx.x * kBand, rows = min(kBand, p.h - r0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = (w + kChunkX - 1) / kChunkX;
    float hi = 0.0f, lo = 0.0f, pl = 0.0f;
    // a loading lane's column of the next chunk: its pixels (0 below the picture) and its prefix above the band, read one
    // chunk ahead
    uint16_t raw[kBand];
    unsigned above = 0;
    auto fetch = [&](int chunk) {
        const int x = chunk * kChunkX + (warp - 1) * 32 + lane;
        if (x >= w) return;
        const uint16_t *src = J.y + (size_t)r0 * w + x;
        above = __ldg(J.band + (size_t)blockIdx.x * w + x);
        if (rows == kBand) {
#pragma unroll
            for (int r = 0; r < kBand; r++) raw[r] = __ldg(src + (size_t)r * w);
        } else {
#pragma unroll
            for (int r = 0; r < kBand; r++) raw[r] = r < rows ? __ldg(src + (size_t)r * w) : (uint16_t)0;
        }
    };
    if (warp == 1 || warp == 2) fetch(0);
    for (int it = 0; it < chunks + 2; it++) {  // chunk it is made, it - 1 scanned, it - 2 stored
        if (warp == 0) {
            if (it >= 1 && it <= chunks) {
                const int b = (it - 1) & 1, n = min(kChunkX, w - (it - 1) * kChunkX);
#pragma unroll 8
                for (int x = 0; x < n; x++) {
                    const float v = sm.c[b][x][lane];
                    float t, e;
                    two_sum(hi, v, t, e);
                    hi = t;
                    lo = __fadd_rn(lo, e);
                    pl = __fadd_rn(pl, v);
                    sm.out[b][0][x][lane] = hi;
                    sm.out[b][1][x][lane] = lo;
                    sm.out[b][2][x][lane] = pl;
                }
            }
        } else if (warp <= 2) {
            const int cx = (warp - 1) * 32 + lane;
            if (it < chunks) {
                unsigned a = above;
                float *dst = sm.c[it & 1][cx];
#pragma unroll
                for (int r = 0; r < kBand; r++) {
                    a += (unsigned)raw[r] << p.up;
                    dst[r] = __uint2float_rn(a);
                }
                if (it + 1 < chunks) fetch(it + 1);
            }
        } else if (it >= 2) {
            const int b = it & 1, x0 = (it - 2) * kChunkX;
            float *const dst[3] = {J.shi, J.slo, J.sp};
            for (int i = warp - 3; i < rows; i += kSatThreads / 32 - 3) {
#pragma unroll
                for (int q = 0; q < 3; q++)
#pragma unroll
                    for (int k = 0; k < kChunkX; k += 32)
                        if (x0 + k + lane < w) dst[q][(size_t)(r0 + i) * w + x0 + k + lane] = sm.out[b][q][k + lane][i];
            }
        }
        __syncthreads();
    }
}

// The tables of pictures with more than kExactRows rows: a thread per column, then a thread per row.
__global__ void sat_cols_kernel(const uint16_t *y, int w, int h, int up, float *shi, float *slo, float *sp)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= w) return;
    float hi = 0.0f, lo = 0.0f, p = 0.0f;
    for (int r = 0; r < h; r++) {
        const size_t k = (size_t)r * w + x;
        const int v = (int)y[k] << up;
        float t, e;
        two_sum(hi, (float)v, t, e);
        hi = t;
        lo = __fadd_rn(lo, e);
        p = __fadd_rn(p, (float)v);
        shi[k] = hi;
        slo[k] = lo;
        sp[k] = p;
    }
}

__global__ void sat_rows_kernel(int w, int h, float *shi, float *slo, float *sp)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= h) return;
    float hi = 0.0f, lo = 0.0f, p = 0.0f;
    for (int x = 0; x < w; x++) {
        const size_t k = (size_t)r * w + x;
        float t, e;
        two_sum(hi, shi[k], t, e);
        hi = t;
        lo = __fadd_rn(__fadd_rn(lo, e), slo[k]);
        p = __fadd_rn(p, sp[k]);
        shi[k] = hi;
        slo[k] = lo;
        sp[k] = p;
    }
}

// ---- block sums ----------------------------------------------------------------------------------------------------
struct SatView {
    const float *shi, *slo, *sp;
    const uint16_t *y;
};
struct BlockPair {
    SatView v[2];
    int w, h, up, bw;
};

// x / b correctly rounded, r = 1 / b rounded: the quotient's remainder is exact in a fused multiply-add and corrects it
// (Markstein 1990; checked against IEEE division over every 24-bit significand for b = 9 and 81, away from underflow).
__device__ __forceinline__ float div_by(float x, float b, float r)
{
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-b, q, x), r, q);
}
__device__ __forceinline__ float div9(float x) { return div_by(x, 9.0f, 1.0f / 9.0f); }
__device__ __forceinline__ float div81(float x) { return div_by(x, 81.0f, 1.0f / 81.0f); }

constexpr int kTS = 25;  // table entries per side around a block: columns x0 - 5 .. x0 + 19
struct BlockSmem {
    float t[3][kTS][kTS];  // hi, lo, plain; 0 outside the picture (left and above it the sums are 0)
    int y[24][24];         // pixels x0 - 4 .. x0 + 19, coordinates clamped
    int h3[20][18], h9[24][16];
    int s3[18][18];        // the box sums around x0 - 1 .. x0 + 16: exact, compensated, plain / 9
    float c3[18][18], p3[18][18];
};

struct PixelTerms {
    int f, m, gx, gy;        // exact numerators: fine x 9, mid x 81, gradients x 9
    float fc, mc, gxc, gyc;  // FP32 from the compensated table (gradients as their exact numerators, x 9)
    float fp, mp, gxp, gyp;  // FP32 from the plain table
};

// Box sum of side 2 r + 1 around block pixel (i, j) from the table: the 4-corner difference, in its order. An entry left
// of or above the picture is 0, which changes nothing.
__device__ __forceinline__ void corner_sum(const BlockSmem &sm, int i, int j, int r, float &c, float &p)
{
    const int x1 = i + 5 + r, y1 = j + 5 + r, x0 = x1 - 2 * r - 1, y0 = y1 - 2 * r - 1;
    float h = sm.t[0][y1][x1], l = sm.t[1][y1][x1];
    p = sm.t[2][y1][x1];
    auto add = [&](int yy, int xx, float sign) {
        float t, e;
        two_sum(h, sign * sm.t[0][yy][xx], t, e);
        h = t;
        l = __fadd_rn(__fadd_rn(l, e), sign * sm.t[1][yy][xx]);
        p = __fadd_rn(p, sign * sm.t[2][yy][xx]);
    };
    add(y1, x0, -1.0f);
    add(y0, x1, -1.0f);
    add(y0, x0, 1.0f);
    c = __fadd_rn(h, l);
}

// Fills both pictures' buffers for the block at (x0, y0), all loads in flight together: a warp per row. The box sums of
// the 18 x 18 pixels around are made once. Near the picture's edges the box is summed over clamped pixels: whole numbers
// below 2^24, so exact in every arithmetic.
__device__ __forceinline__ void fill_block(BlockSmem (&sm)[2], const BlockPair &P, int x0, int y0)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = P.w, h = P.h;
    const bool inside = x0 >= 5 && y0 >= 5 && x0 + 20 <= w && y0 + 20 <= h;
    const int xt = x0 - 5 + lane;
    float t[6][4];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const SatView &V = P.v[q / 3];
        const float *src = q % 3 == 0 ? V.shi : q % 3 == 1 ? V.slo : V.sp;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int r = warp + 8 * k, y = y0 - 5 + r;
            t[q][k] = (lane < kTS && r < kTS && (inside || (xt >= 0 && xt < w && y >= 0 && y < h))) ? __ldg(src + (size_t)y * w + xt) : 0.0f;
        }
    }
    const int xy = min(max(x0 - 4 + lane, 0), w - 1);
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int r = warp + 8 * k, y = min(max(y0 - 4 + r, 0), h - 1);
            if (lane < 24) sm[q].y[r][lane] = (int)__ldg(P.v[q].y + (size_t)y * w + xy) << P.up;
        }
#pragma unroll
    for (int q = 0; q < 6; q++)
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (lane < kTS && warp + 8 * k < kTS) sm[q / 3].t[q % 3][warp + 8 * k][lane] = t[q][k];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int r = warp + 8 * k;
            if (lane < 16) {
                int a = 0;
#pragma unroll
                for (int c = 0; c < 9; c++) a += sm[q].y[r][lane + c];
                sm[q].h9[r][lane] = a;
            }
            if (r >= 2 && r < 22 && lane < 18) sm[q].h3[r - 2][lane] = sm[q].y[r][lane + 2] + sm[q].y[r][lane + 3] + sm[q].y[r][lane + 4];
        }
    __syncthreads();
    for (int k = tid; k < 2 * 18 * 18; k += 256) {
        const int q = k >= 18 * 18, kk = k - q * 18 * 18, j = kk / 18, i = kk - j * 18, x = x0 - 1 + i, y = y0 - 1 + j;
        BlockSmem &B = sm[q];
        const int s3 = B.h3[j][i] + B.h3[j + 1][i] + B.h3[j + 2][i];
        float c = (float)s3, p = c;
        if (inside || (x >= 1 && y >= 1 && x + 1 < w && y + 1 < h)) corner_sum(B, i - 1, j - 1, 1, c, p);
        B.s3[j][i] = s3;
        B.c3[j][i] = c;
        B.p3[j][i] = div9(p);
    }
    __syncthreads();
}

__device__ __forceinline__ PixelTerms block_terms(const BlockSmem &sm, int w, int h, int x0, int y0)
{
    const int tid = threadIdx.x;
    const int i = tid & 15, j = tid >> 4, x = x0 + i, y = y0 + j;
    int s9 = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) s9 += sm.h9[j + k][i];
    float c9 = (float)s9, p9 = c9;
    if (x >= 4 && y >= 4 && x + 4 < w && y + 4 < h) corner_sum(sm, i, j, 4, c9, p9);
    const int v = sm.y[j + 4][i + 4], s3 = sm.s3[j + 1][i + 1];
    const float c3 = sm.c3[j + 1][i + 1], p3 = sm.p3[j + 1][i + 1];
    PixelTerms t;
    t.f = 9 * v - s3;
    t.m = 9 * s3 - s9;
    t.fc = div9(__fsub_rn(__fmul_rn(9.0f, (float)v), c3));
    t.mc = div81(__fsub_rn(__fmul_rn(9.0f, c3), c9));
    t.fp = __fsub_rn((float)v, p3);
    t.mp = __fsub_rn(p3, div81(p9));
    t.gx = t.gy = 0;
    t.gxc = t.gyc = t.gxp = t.gyp = 0.0f;
    if (x > 0 && x < w - 1) {
        t.gx = sm.s3[j + 1][i + 2] - sm.s3[j + 1][i];
        t.gxc = __fsub_rn(sm.c3[j + 1][i + 2], sm.c3[j + 1][i]);
        t.gxp = __fsub_rn(sm.p3[j + 1][i + 2], sm.p3[j + 1][i]);
    }
    if (y > 0 && y < h - 1) {
        t.gy = sm.s3[j + 2][i + 1] - sm.s3[j][i + 1];
        t.gyc = __fsub_rn(sm.c3[j + 2][i + 1], sm.c3[j][i + 1]);
        t.gyp = __fsub_rn(sm.p3[j + 2][i + 1], sm.p3[j][i + 1]);
    }
    return t;
}

// One block of 256 threads per 16 x 16 block: the 12 sums in the three arithmetics. The exact sums are in units of
// the numerators (fine and gradients x 9, mid x 81). Each quantity's 32 lanes are added as a butterfly would (lanes 16
// apart, then 8, 4, 2, 1), but a lane keeps only half of its quantities at each step: 13 exchanges instead of 60.
// Issue and shared-memory access bound it (1380 instructions per 32 pixels, 70 % of the issue slots); 906 us before, with
// the box sums gathered per pixel from the tables, against 430 us now for two 3840 x 2160 pictures (one picture's loads
// after the other's: 730 us).
__global__ void __launch_bounds__(256) block_sums_kernel(const __grid_constant__ BlockPair P, long long *qi, float *qc, float *qp)
{
    __shared__ BlockSmem sm[2];
    __shared__ long long si[kQ][8];
    __shared__ float sc[kQ][8], sp[kQ][8];
    const int b = blockIdx.x, bx = b % P.bw, by = b / P.bw;
    fill_block(sm, P, 16 * bx, 16 * by);
    const PixelTerms r = block_terms(sm[0], P.w, P.h, 16 * bx, 16 * by), d = block_terms(sm[1], P.w, P.h, 16 * bx, 16 * by);
    auto mul = [](int a, int c) { return (long long)a * c; };
    long long vi[kQ] = {mul(r.f, r.f), mul(r.m, r.m), mul(d.f, d.f), mul(d.m, d.m), mul(r.f, d.f), mul(r.m, d.m),
                        mul(r.gx, r.gx), mul(r.gy, r.gy), mul(r.gx, r.gy), mul(d.gx, d.gx), mul(d.gy, d.gy), mul(d.gx, d.gy)};
    // compensated form: the tensor's Jxx - Jyy summed per pixel as (gx - gy)(gx + gy) from the exact numerators, so
    // the cancellation of an isotropic texture happens before the sum; Jyy's slot is unused (0)
    auto dxy = [](float gx, float gy) { return div81(__fmul_rn(__fsub_rn(gx, gy), __fadd_rn(gx, gy))); };
    auto pxy = [](float gx, float gy) { return div81(__fmul_rn(gx, gy)); };
    float cs[kQ] = {r.fc * r.fc, r.mc * r.mc, d.fc * d.fc, d.mc * d.mc, r.fc * d.fc, r.mc * d.mc,
                    dxy(r.gxc, r.gyc), 0.0f, pxy(r.gxc, r.gyc), dxy(d.gxc, d.gyc), 0.0f, pxy(d.gxc, d.gyc)};
    float vp[kQ] = {r.fp * r.fp, r.mp * r.mp, d.fp * d.fp, d.mp * d.mp, r.fp * d.fp, r.mp * d.mp,
                    r.gxp * r.gxp, r.gyp * r.gyp, r.gxp * r.gyp, d.gxp * d.gxp, d.gyp * d.gyp, d.gxp * d.gyp};
    float ce[kQ];
#pragma unroll
    for (int q = 0; q < kQ; q++) ce[q] = 0.0f;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto combine = [&](int k, long long oi, float os, float oe, float op) {
        vi[k] += oi;
        float t, e;
        two_sum(cs[k], os, t, e);
        cs[k] = t;
        ce[k] = __fadd_rn(__fadd_rn(ce[k], oe), e);
        vp[k] = __fadd_rn(vp[k], op);
    };
    auto exchange = [&](auto kept_c, auto held_c, int off) {  // a lane keeps `kept` of `held` quantities
        constexpr int n = decltype(kept_c)::value, held = decltype(held_c)::value;
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < n; k++) {
            const int k2 = k + n < held ? k + n : k;  // a quantity without a partner is kept by both
            const long long si_ = upper ? vi[k] : vi[k2];
            const float ss = upper ? cs[k] : cs[k2], se = upper ? ce[k] : ce[k2], sv = upper ? vp[k] : vp[k2];
            vi[k] = upper ? vi[k2] : vi[k];
            cs[k] = upper ? cs[k2] : cs[k];
            ce[k] = upper ? ce[k2] : ce[k];
            vp[k] = upper ? vp[k2] : vp[k];
            combine(k, __shfl_xor_sync(0xffffffffu, si_, off), __shfl_xor_sync(0xffffffffu, ss, off), __shfl_xor_sync(0xffffffffu, se, off),
                    __shfl_xor_sync(0xffffffffu, sv, off));
        }
    };
    exchange(std::integral_constant<int, 6>{}, std::integral_constant<int, 12>{}, 16);
    exchange(std::integral_constant<int, 3>{}, std::integral_constant<int, 6>{}, 8);
    exchange(std::integral_constant<int, 2>{}, std::integral_constant<int, 3>{}, 4);
    exchange(std::integral_constant<int, 1>{}, std::integral_constant<int, 2>{}, 2);
    combine(0, __shfl_xor_sync(0xffffffffu, vi[0], 1), __shfl_xor_sync(0xffffffffu, cs[0], 1), __shfl_xor_sync(0xffffffffu, ce[0], 1),
            __shfl_xor_sync(0xffffffffu, vp[0], 1));
    const int third = ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1), q_of = (lane >> 4) * 6 + ((lane >> 3) & 1) * 3 + third;
    if ((lane & 1) == 0 && third < 3) {
        si[q_of][warp] = vi[0];
        sc[q_of][warp] = __fadd_rn(cs[0], ce[0]);
        sp[q_of][warp] = vp[0];
    }
    __syncthreads();
    if (threadIdx.x < kQ) {
        const int q = threadIdx.x;
        long long a = 0;
        Comp c;
        float p = 0.0f;
        for (int k = 0; k < 8; k++) {
            a += si[q][k];
            c.add(sc[q][k]);
            p = __fadd_rn(p, sp[q][k]);
        }
        qi[(size_t)b * kQ + q] = a;
        qc[(size_t)b * kQ + q] = c.value();
        qp[(size_t)b * kQ + q] = p;
    }
}

// Figures of each window of k x k blocks; mode 0 exact (int64, one rounding to double), 1 compensated FP32, 2 FP32. A
// thread per window and quantity adds the blocks in order, then a thread per window and figure.
constexpr int kFigWindows = 16;
__global__ void __launch_bounds__(kFigWindows *kQ) window_figures_kernel(const long long *qi, const float *qc, const float *qp, int bw, int bh,
                                                                        int k, int mode, double *out)
{
    __shared__ long long ti[kFigWindows][kQ];
    __shared__ float tf[kFigWindows][kQ];
    const int ww = bw / k, wh = bh / k, n = ww * wh;
    {
        const int l = threadIdx.x / kQ, q = threadIdx.x - l * kQ, i = blockIdx.x * kFigWindows + l;
        if (i < n) {
            const int wx = i % ww, wy = i / ww;
            long long a = 0;
            Comp c;
            float p = 0.0f;
            for (int by = wy * k; by < wy * k + k; by++) {
                const size_t at = ((size_t)by * bw + wx * k) * kQ + q;
#pragma unroll 8
                for (int bx = 0; bx < k; bx++) {
                    if (mode == 0) a += __ldg(qi + at + (size_t)bx * kQ);
                    else if (mode == 1) c.add(__ldg(qc + at + (size_t)bx * kQ));
                    else p = __fadd_rn(p, __ldg(qp + at + (size_t)bx * kQ));
                }
            }
            ti[l][q] = a;
            tf[l][q] = mode == 1 ? c.value() : p;
        }
    }
    __syncthreads();
    const int l = threadIdx.x >> 3, g = threadIdx.x & 7, i = blockIdx.x * kFigWindows + l;
    if (l >= kFigWindows || i >= n) return;
    double fig;
    if (mode == 0) {
        const long long *s = ti[l];
        if (g < 6) {
            fig = (double)s[g] / ((g & 1) ? 6561.0 : 81.0);
        } else {
            const int o = g == 6 ? 6 : 9;
            const double dd = (double)(s[o] - s[o + 1]), x = (double)s[o + 2];
            fig = sqrt(dd * dd + 4.0 * x * x) / 81.0;
        }
    } else {
        const float *s = tf[l];
        if (g < 6) {
            fig = (double)s[g];
        } else {
            // compensated form: slots 6 and 9 already hold Jxx - Jyy
            const int o = g == 6 ? 6 : 9;
            const float dd = mode == 1 ? s[o] : __fsub_rn(s[o], s[o + 1]);
            fig = (double)__fsqrt_rn(__fadd_rn(__fmul_rn(dd, dd), __fmul_rn(4.0f, __fmul_rn(s[o + 2], s[o + 2]))));
        }
    }
    out[(size_t)i * 8 + g] = fig;
}

}  // namespace

int precision_quantities() { return kQ; }

// Words of one picture's band sums.
size_t precision_band_words(int w, int h) { return h <= kExactRows ? (size_t)((h + kBand - 1) / kBand) * w : 1; }

cudaError_t launch_precision_sat(const uint16_t *const y[2], int w, int h, int up, unsigned *const band[2], float *const shi[2],
                                 float *const slo[2], float *const sp[2], cudaStream_t s)
{
    if (h > kExactRows) {
        for (int i = 0; i < 2; i++) {
            {
                LaunchTimer t("precision_sat", s);
                sat_cols_kernel<<<(w + 127) / 128, 128, 0, s>>>(y[i], w, h, up, shi[i], slo[i], sp[i]);
            }
            cudaError_t e = after_launch();
            if (e != cudaSuccess) return e;
            LaunchTimer t("precision_sat", s);
            sat_rows_kernel<<<(h + 127) / 128, 128, 0, s>>>(w, h, shi[i], slo[i], sp[i]);
            if ((e = after_launch()) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    SatPair p{};
    for (int i = 0; i < 2; i++) p.job[i] = SatJob{y[i], band[i], shi[i], slo[i], sp[i]};
    p.w = w;
    p.h = h;
    p.up = up;
    const int bands = (h + kBand - 1) / kBand;
    {
        LaunchTimer t("precision_sat", s);
        band_sums_kernel<<<dim3((w + 255) / 256, bands, 2), 256, 0, s>>>(p);
    }
    cudaError_t e = after_launch();
    if (e != cudaSuccess) return e;
    {
        LaunchTimer t("precision_sat", s);
        band_prefix_kernel<<<dim3((w + 63) / 64, 2), 64, 0, s>>>(p, bands);
    }
    if ((e = after_launch()) != cudaSuccess) return e;
    e = cudaFuncSetAttribute(sat_band_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SatSmem));
    if (e != cudaSuccess) return e;
    LaunchTimer t("precision_sat", s);
    sat_band_kernel<<<dim3(bands, 2), kSatThreads, sizeof(SatSmem), s>>>(p);
    return after_launch();
}

cudaError_t launch_precision_blocks(const uint16_t *const y[2], int w, int h, int up, const float *const shi[2], const float *const slo[2],
                                    const float *const sp[2], long long *qi, float *qc, float *qp, cudaStream_t s)
{
    const int bw = w / 16, bh = h / 16;
    if (bw <= 0 || bh <= 0) return cudaSuccess;
    BlockPair p{};
    for (int i = 0; i < 2; i++) p.v[i] = SatView{shi[i], slo[i], sp[i], y[i]};
    p.w = w;
    p.h = h;
    p.up = up;
    p.bw = bw;
    LaunchTimer t("precision_blocks", s);
    block_sums_kernel<<<bw * bh, 256, 0, s>>>(p, qi, qc, qp);
    return after_launch();
}

cudaError_t launch_precision_windows(const long long *qi, const float *qc, const float *qp, int bw, int bh, int k, int mode,
                                     double *out, cudaStream_t s)
{
    const int n = (bw / k) * (bh / k);
    if (n <= 0) return cudaSuccess;
    LaunchTimer t("precision_windows", s);
    window_figures_kernel<<<(n + kFigWindows - 1) / kFigWindows, kFigWindows * kQ, 0, s>>>(qi, qc, qp, bw, bh, k, mode, out);
    return after_launch();
}

}  // namespace es
