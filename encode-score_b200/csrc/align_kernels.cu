// Temporal alignment kernels for sm_100a: the thumbnails a source and its encodes are matched by, and the per-lag
// difference totals of the offset search.
//
// The reference (src/kernels.cu:502-520, src/main.cpp:301-353) launches tiny_luma once per decoded frame, copies
// each 64 x 36 thumbnail to the host with a stream synchronisation, and searches the lags on the CPU. Here one launch
// makes the thumbnails of a whole batch of frames (one block per cell and frame), each cell's sum is an exact integer
// divided once, and the lags are searched on the device with totals that equal the reference's in-order double sums bit
// for bit, so that the chosen lag is the same.
#include "es_kernels.h"

namespace es {
namespace {

__device__ __forceinline__ unsigned luma_at(const FrameViewDev &f, int x, int y)
{
    const unsigned char *row = (const unsigned char *)f.y + (size_t)y * f.ypitch;
    const unsigned v = f.bytes == 1 ? row[x] : ((const uint16_t *)row)[x];
    return v >> f.shift;
}

// Block (tx, ty, frame): the mean of cell (tx, ty) of that frame, for any crop and alignment. Threads walk the cell as
// 8 rows of 32 columns (one warp per row, consecutive columns per lane), summing 10-bit samples exactly.
__global__ void __launch_bounds__(256) thumb_kernel(const __grid_constant__ ThumbBatch b)
{
    const FrameViewDev &f = b.f[blockIdx.z];
    const int tx = blockIdx.x, ty = blockIdx.y;
    const int xa = b.x0 + tx * b.w / kThumbW, xb = b.x0 + (tx + 1) * b.w / kThumbW;
    const int ya = b.y0 + ty * b.h / kThumbH, yb = b.y0 + (ty + 1) * b.h / kThumbH;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5, up = 10 - f.depth;
    unsigned s = 0;  // at most a cell's share of a thread times 1023: far below 2^32 for any picture size in use
    for (int y = ya + row; y < yb; y += 8)
        for (int x = xa + lane; x < xb; x += 32) s += luma_at(f, x, y) << up;
    unsigned long long t = s;
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    __shared__ unsigned long long part[8];
    if (lane == 0) part[row] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int k = 0; k < 8; k++) total += part[k];
        const int n = (xb - xa) * (yb - ya);
        // a cell with no pixel gives 0 / 0 = NaN, as in the reference
        b.out[((size_t)blockIdx.z * kThumbH + ty) * kThumbW + tx] = __fdiv_rn((float)total, (float)n);
    }
}

// The same thumbnails by 8 samples at a time (16 bytes, 8 for 8-bit samples), for planes whose address and pitch are
// multiples of that and crops at least 512 columns wide (every cell at least 8, so 8 columns span at most two cells); the
// crop may start anywhere. Block (ty, frame) makes the 64 cells of thumbnail row ty from its band of rows: a thread takes
// one group of 8 columns down the band, adding 16 rows of samples in the 16-bit halves of 32-bit words before they go to
// its eight column sums (rows with a sample of 2^12 or more, beyond any depth here, are added one by one), and the block's
// cell sums meet in shared memory. A group that overlaps the crop's
// edge is read whole: it lies within the aligned 16 (8) bytes of a sample of the crop.
// Bound by HBM: 64 frames of 3840 x 2160 10-bit (1.06 GB) took 311 us with four rows in flight per thread and one sample
// added at a time, 182 us with eight in flight and packed sums.
constexpr int kThumbRowsInFlight = 8, kThumbPacked = 16;

template <int kBytes>
__device__ __forceinline__ void thumb_band(const FrameViewDev &f, int x, int ya, int yb, unsigned (&col)[8])
{
    const unsigned mask = kBytes == 2 ? (0xFFFFu >> f.shift) * 0x10001u : (0xFFu >> f.shift) * 0x10001u;
    const unsigned char *p = (const unsigned char *)f.y + (size_t)ya * f.ypitch + (size_t)x * kBytes;
    for (int y = ya; y < yb; y += kThumbPacked) {
        unsigned s[4] = {0, 0, 0, 0}, seen = 0;  // pairs of columns (2 bytes: 0 1, 2 3, ...; 1 byte: 0 2, 1 3, 4 6, 5 7)
#pragma unroll
        for (int g = 0; g < kThumbPacked; g += kThumbRowsInFlight) {
            uint4 q[kThumbRowsInFlight];
#pragma unroll
            for (int k = 0; k < kThumbRowsInFlight; k++) {
                q[k] = make_uint4(0, 0, 0, 0);
                if (y + g + k < yb) {
                    const unsigned char *r = p + (size_t)(g + k) * f.ypitch;
                    if (kBytes == 2) {
                        q[k] = __ldg((const uint4 *)r);
                    } else {
                        const uint2 v = __ldg((const uint2 *)r);
                        q[k].x = v.x;
                        q[k].y = v.y;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kThumbRowsInFlight; k++) {
                if (kBytes == 2) {
                    const unsigned t[4] = {(q[k].x >> f.shift) & mask, (q[k].y >> f.shift) & mask, (q[k].z >> f.shift) & mask,
                                           (q[k].w >> f.shift) & mask};
#pragma unroll
                    for (int i = 0; i < 4; i++) s[i] += t[i];
                    seen |= t[0] | t[1];
                    seen |= t[2] | t[3];
                } else {
                    s[0] += (q[k].x >> f.shift) & mask;
                    s[1] += (q[k].x >> (8 + f.shift)) & mask;
                    s[2] += (q[k].y >> f.shift) & mask;
                    s[3] += (q[k].y >> (8 + f.shift)) & mask;
                }
            }
        }
        if (kBytes == 2 && (seen & 0xF000F000u)) {  // the halves may have overflowed
            for (int k = 0; k < kThumbPacked && y + k < yb; k++)
#pragma unroll
                for (int i = 0; i < 8; i++) col[i] += (unsigned)((const uint16_t *)(p + (size_t)k * f.ypitch))[i] >> f.shift;
            p += (size_t)kThumbPacked * f.ypitch;
            continue;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int lo = kBytes == 2 ? 2 * k : 4 * (k >> 1) + (k & 1), hi = kBytes == 2 ? lo + 1 : lo + 2;
            col[lo] += s[k] & 0xFFFFu;
            col[hi] += s[k] >> 16;
        }
        p += (size_t)kThumbPacked * f.ypitch;
    }
}

__global__ void __launch_bounds__(256) thumb_rows_kernel(const __grid_constant__ ThumbBatch b)
{
    const FrameViewDev &f = b.f[blockIdx.y];
    const int ty = blockIdx.x;
    const int ya = b.y0 + ty * b.h / kThumbH, yb = b.y0 + (ty + 1) * b.h / kThumbH;
    __shared__ unsigned long long cell[kThumbW];
    if (threadIdx.x < kThumbW) cell[threadIdx.x] = 0;
    __syncthreads();
    const int up = 10 - f.depth, xs = b.x0 & ~7, groups = (b.x0 + b.w - xs + 7) / 8;
    for (int g = threadIdx.x; g < groups; g += 256) {
        const int c = xs + 8 * g - b.x0, c0 = max(c, 0);  // the group's first column, from x0; its first in the crop
        int ta = 64 * c0 / b.w;                           // its cell: 64 c0 / w or the next one
        if (ta < kThumbW - 1 && (ta + 1) * b.w / kThumbW <= c0) ta++;
        const int bound = (ta + 1) * b.w / kThumbW;       // first column of cell ta + 1
        unsigned col[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (f.bytes == 2) thumb_band<2>(f, xs + 8 * g, ya, yb, col);
        else thumb_band<1>(f, xs + 8 * g, ya, yb, col);
        unsigned long long sa = 0, sb = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (c + k < 0 || c + k >= b.w) continue;
            if (c + k < bound) sa += col[k];
            else sb += col[k];
        }
        atomicAdd(&cell[ta], sa << up);
        if (sb) atomicAdd(&cell[ta + 1], sb << up);  // columns past `bound` exist only when ta < 63
    }
    __syncthreads();
    if (threadIdx.x < kThumbW) {
        const int t = threadIdx.x, n = ((t + 1) * b.w / kThumbW - t * b.w / kThumbW) * (yb - ya);
        b.out[((size_t)blockIdx.y * kThumbH + ty) * kThumbW + t] = __fdiv_rn((float)cell[t], (float)n);
    }
}

// The total of lag l: the sum over probe frames i and pixels p (in that order) of |ref[l + i][p] - probe[i][p]|, the
// difference in float and the sum in double (src/main.cpp:342-346). Frames are stored one after another, so a lag
// reads two contiguous runs of n_probe x 2304 floats. One warp per lag, chunks of kChunk values, lane j holding values
// j*kLaneVals .. j*kLaneVals + kLaneVals - 1 of a chunk.
//
// The running total s is a double >= 0 and every value x is a float >= 0. While s stays in one binade [2^e, 2^(e+1)),
// s = m * u with u = 2^(e-52) and m an integer in [2^52, 2^53), and the rounded sum RN(s + x) is (m + n + r) * u where
// n = floor(x / u) and r is 1 when the remainder of x / u is above one half, 0 below, and on an exact half the value
// that makes m + n + r even (ties to even). x / u is exact (x has a 24-bit mantissa, u is a power of two), so n and the
// remainder's class come from integer shifts of x's mantissa. The only state one step passes to the next beyond the
// increment is the parity of m, so a run of values is a map from the parity coming in to (increment, parity going
// out): a pair of increments and a pair of parities. These maps compose in order, which makes the chunk an ordered
// warp reduction instead of a chain of kChunk dependent additions. If the chunk's end stays below 2^53 (m + the
// increment), every intermediate sum stayed in the binade (each exact sum is within one half of the next rounded
// one), so the result is exactly the in-order chain's. A chunk that crosses a binade, starts from s = 0, or holds a
// value the shifts cannot represent (an increment of 2^53 or more, an infinity or NaN) is added in order, one value at
// a time, from shared memory. Adding zeros leaves s as it is, so a chunk of zeros and the padding of the last chunk
// are skipped. The result equals the in-order double sum bit for bit.
// Thumbnails of ordinary pictures need none of that: means of 8 code values or more have no bits below 2^-20, so every
// difference is a whole number of those units below 2^30, and while the total stays below 2^53 of them every sum is
// exact in any order. offset_check_kernel finds the frames with a value that is no whole number of units (or outside
// [0, 1024), or NaN) and marks the lags that read them; offset_exact_kernel adds the differences of every lag as 64-bit
// integers: a block takes 16 lags x 16 probe frames x 768 pixels, a thread one pixel at a time, 47 values in registers
// for 256 differences (a float subtraction, a conversion and about one integer addition each). The loads bound it, 47
// from L2 per 256 differences (conversions spread over other pipes changed nothing, sums in double were slower: 84
// against 62 us); the in-order form issues about 40 instructions per difference and has one warp per lag. 483 lags of
// 192 frames: 1035 us in order, 76 us for the three launches; where no lag is exact (means below 8 code values) 1010 us, 1129
// when offset_exact_kernel added marked lags all the same.
constexpr double kFixed = 1048576.0;                     // units per code value
constexpr unsigned long long kInexact = 1ull << 63;      // mark in a lag's integer sum
constexpr int kExactMaxProbe = (1 << 23) / kThumbPixels;  // frames whose totals stay below 2^53 units
constexpr int kExLags = 16, kExFrames = 16, kExThreads = 256, kExPixels = 768;
static_assert(kThumbPixels % kExPixels == 0 && kExPixels % kExThreads == 0, "whole pixel chunks");

__global__ void __launch_bounds__(kExThreads) offset_check_kernel(const float *ref, int n_ref, const float *probe, int n_probe, int lags,
                                                                  unsigned long long *sums)
{
    const int f = blockIdx.x;
    const float *v = f < n_ref ? ref + (size_t)f * kThumbPixels : probe + (size_t)(f - n_ref) * kThumbPixels;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < kThumbPixels / kExThreads; i++) {
        const float x = __ldg(v + i * kExThreads + threadIdx.x), u = __fmul_rn(x, (float)kFixed);
        ok &= x >= 0.0f && x < 1024.0f && rintf(u) == u;
    }
    if (!__syncthreads_or(!ok)) return;
    const int first = f < n_ref ? max(f - n_probe + 1, 0) : 0, last = f < n_ref ? min(f, lags - 1) : lags - 1;
    for (int l = first + threadIdx.x; l <= last; l += kExThreads) atomicOr(sums + l, kInexact);
}

template <bool kWhole>
__device__ __forceinline__ void exact_pixel(const float *r0, const float *p0, int n_frames, int n_lags, unsigned long long (&acc)[kExLags])
{
    float r[kExLags + kExFrames - 1], p[kExFrames];
#pragma unroll
    for (int j = 0; j < kExLags + kExFrames - 1; j++)
        r[j] = kWhole || j < n_frames + n_lags - 1 ? __fmul_rn(__ldg(r0 + (size_t)j * kThumbPixels), (float)kFixed) : 0.0f;
#pragma unroll
    for (int i = 0; i < kExFrames; i++) p[i] = kWhole || i < n_frames ? __fmul_rn(__ldg(p0 + (size_t)i * kThumbPixels), (float)kFixed) : 0.0f;
#pragma unroll
    for (int l = 0; l < kExLags; l++) {
#pragma unroll
        for (int i = 0; i < kExFrames; i += 4) {
            unsigned t = 0;  // four differences below 1023 2^20 + 2^20 each: below 2^32
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned d = __float2uint_rz(fabsf(__fsub_rn(r[l + i + k], p[i + k])));
                if (kWhole || i + k < n_frames) t += d;
            }
            acc[l] += t;
        }
    }
}

__global__ void __launch_bounds__(kExThreads, 2) offset_exact_kernel(const float *ref, const float *probe, int n_probe, int lags,
                                                                     unsigned long long *sums)
{
    __shared__ unsigned long long total[kExLags];
    wait_for_previous();
    const int l0 = blockIdx.x * kExLags, i0 = blockIdx.y * kExFrames, lane = threadIdx.x & 31;
    const int n_lags = min(kExLags, lags - l0), n_frames = min(kExFrames, n_probe - i0);
    if (threadIdx.x < kExLags) total[threadIdx.x] = 0;
    // nothing to add where every lag is marked (other blocks' additions leave the marks as they are)
    if (__syncthreads_and((int)threadIdx.x >= n_lags || (__ldcg(sums + l0 + threadIdx.x) & kInexact))) return;
    unsigned long long acc[kExLags];
#pragma unroll
    for (int l = 0; l < kExLags; l++) acc[l] = 0;
    for (int c = 0; c < kExPixels; c += kExThreads) {
        const int px = blockIdx.z * kExPixels + c + threadIdx.x;
        const float *r0 = ref + (size_t)(l0 + i0) * kThumbPixels + px, *p0 = probe + (size_t)i0 * kThumbPixels + px;
        if (n_lags == kExLags && n_frames == kExFrames) exact_pixel<true>(r0, p0, n_frames, n_lags, acc);
        else exact_pixel<false>(r0, p0, n_frames, n_lags, acc);
    }
    // 16 sums over 32 lanes: each step halves the sums a lane holds and adds the other half lane's
#pragma unroll
    for (int n = kExLags / 2, off = 16; n >= 1; n >>= 1, off >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < n; k++) {
            const unsigned long long send = upper ? acc[k] : acc[k + n], keep = upper ? acc[k + n] : acc[k];
            acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    if ((lane & 1) == 0) atomicAdd(&total[lane >> 1], acc[0]);
    __syncthreads();
    if ((int)threadIdx.x < n_lags) atomicAdd(sums + l0 + threadIdx.x, total[threadIdx.x]);
}

constexpr int kLaneVals = 16, kChunk = 32 * kLaneVals, kLagWarps = 4;

struct ParityMap {
    unsigned long long inc0, inc1;  // increments of m for parity 0 / 1 coming in
    unsigned bits;                  // bit 0: parity out for 0 in, bit 1: for 1 in, bit 2: the chunk must be added in order
};

__device__ __forceinline__ ParityMap compose(const ParityMap &a, const ParityMap &b)
{
    const unsigned a0 = a.bits & 1u, a1 = (a.bits >> 1) & 1u, b0 = b.bits & 1u, b1 = (b.bits >> 1) & 1u;
    ParityMap r;
    r.inc0 = a.inc0 + (a0 ? b.inc1 : b.inc0);
    r.inc1 = a.inc1 + (a1 ? b.inc1 : b.inc0);
    r.bits = (a0 ? b1 : b0) | ((a1 ? b1 : b0) << 1) | ((a.bits | b.bits) & 4u);
    return r;
}

// With kSums, totals[] holds the exact kernels' integer sums: a lag they marked is added as above, any other becomes its
// sum's double.
template <bool kVec, bool kSums>
__global__ void __launch_bounds__(32 * kLagWarps) offset_totals_kernel(const float *ref, const float *probe, int n_probe, int lags,
                                                                      double *totals)
{
    __shared__ __align__(16) double serial[kLagWarps][kChunk];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, l = blockIdx.x * kLagWarps + w;
    if (l >= lags) return;  // whole warps: one lag per warp
    if (kSums) {
        wait_for_previous();
        const unsigned long long v = ((const unsigned long long *)totals)[l];
        if (!(v & kInexact)) {
            __syncwarp();
            if (lane == 0) totals[l] = (double)v * (1.0 / kFixed);  // both exact
            return;
        }
    }
    const float *r = ref + (size_t)l * kThumbPixels;
    const long long count = (long long)n_probe * kThumbPixels;
    const long long chunks = (count + kChunk - 1) / kChunk;
    constexpr int Q = kLaneVals / 4;
    float4 ra[Q], pa[Q];
    auto load = [&](long long c) {  // the next chunk's values, zeros past the end
        const long long v0 = c * kChunk + lane * kLaneVals;
#pragma unroll
        for (int t = 0; t < Q; t++) {
            const long long v = v0 + 4 * t;
            if (kVec) {
                if (v < count) {
                    ra[t] = __ldg((const float4 *)(r + v));
                    pa[t] = __ldg((const float4 *)(probe + v));
                } else {
                    ra[t] = pa[t] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else {
                float a[4], b[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    a[k] = v + k < count ? __ldg(r + v + k) : 0.f;
                    b[k] = v + k < count ? __ldg(probe + v + k) : 0.f;
                }
                ra[t] = make_float4(a[0], a[1], a[2], a[3]);
                pa[t] = make_float4(b[0], b[1], b[2], b[3]);
            }
        }
    };
    double s = 0.0;
    if (chunks > 0) load(0);
    for (long long c = 0; c < chunks; c++) {
        float x[kLaneVals];
#pragma unroll
        for (int t = 0; t < Q; t++) {
            x[4 * t + 0] = fabsf(__fsub_rn(ra[t].x, pa[t].x));
            x[4 * t + 1] = fabsf(__fsub_rn(ra[t].y, pa[t].y));
            x[4 * t + 2] = fabsf(__fsub_rn(ra[t].z, pa[t].z));
            x[4 * t + 3] = fabsf(__fsub_rn(ra[t].w, pa[t].w));
        }
        if (c + 1 < chunks) load(c + 1);
        const unsigned long long sbits = (unsigned long long)__double_as_longlong(s);
        const int E = (int)(sbits >> 52);  // s >= 0: the biased exponent
        const int ue = E - 1075;           // u = 2^ue
        ParityMap m;
        m.inc0 = m.inc1 = 0;
        m.bits = 2u | ((E == 0 || E == 0x7ff) ? 4u : 0u);
        bool nonzero = false;
#pragma unroll
        for (int j = 0; j < kLaneVals; j++) {
            const unsigned xb = __float_as_uint(x[j]);
            nonzero |= xb != 0;
            const int ex = (int)(xb >> 23);  // x >= 0
            const unsigned M = ex ? (xb & 0x7fffffu) | 0x800000u : xb;  // x = M * 2^(ex - 150), subnormals 2^-149
            const int sh = (ex ? ex - 150 : -149) - ue;                 // x / u = M * 2^sh
            const int left = max(sh, 0), right = min(max(-sh, 0), 25);  // M < 2^24: 25 right shifts leave 0 and a low remainder
            if (ex == 255 || left > 29) m.bits |= 4u;
            const unsigned long long n = ((unsigned long long)M << min(left, 29)) >> right;
            const unsigned twice_rem = (M & ((1u << right) - 1u)) << 1, one = 1u << right;
            const unsigned above = twice_rem > one, tie = twice_rem == one, nb = (unsigned)n & 1u;
            const unsigned p0 = m.bits & 1u, p1 = (m.bits >> 1) & 1u;
            const unsigned r0 = above | (tie & (p0 ^ nb)), r1 = above | (tie & (p1 ^ nb));
            m.inc0 += n + r0;
            m.inc1 += n + r1;
            m.bits = (m.bits & 4u) | ((p0 ^ nb ^ r0) & 1u) | (((p1 ^ nb ^ r1) & 1u) << 1);
        }
        if (!__any_sync(0xffffffffu, nonzero)) continue;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {  // ordered: lane j's run, then lane j + off's
            ParityMap o;
            o.inc0 = __shfl_down_sync(0xffffffffu, m.inc0, off);
            o.inc1 = __shfl_down_sync(0xffffffffu, m.inc1, off);
            o.bits = __shfl_down_sync(0xffffffffu, m.bits, off);
            if (lane + off < 32) m = compose(m, o);
        }
        const unsigned long long inc0 = __shfl_sync(0xffffffffu, m.inc0, 0), inc1 = __shfl_sync(0xffffffffu, m.inc1, 0);
        bool in_order = (__shfl_sync(0xffffffffu, m.bits, 0) & 4u) != 0;
        if (!in_order) {
            const unsigned long long mant = (sbits & 0xfffffffffffffull) | (1ull << 52);
            const unsigned long long end = mant + ((mant & 1ull) ? inc1 : inc0);
            if (end < (1ull << 53))
                s = __longlong_as_double((long long)(((unsigned long long)E << 52) | (end & 0xfffffffffffffull)));
            else
                in_order = true;
        }
        if (in_order) {
#pragma unroll
            for (int j = 0; j < kLaneVals; j++) serial[w][lane * kLaneVals + j] = (double)x[j];
            __syncwarp();
            if (lane == 0)
                for (int i = 0; i < kChunk; i++) s = __dadd_rn(s, serial[w][i]);
            s = __shfl_sync(0xffffffffu, s, 0);
            __syncwarp();
        }
    }
    if (lane == 0) totals[l] = s;
}

}  // namespace

cudaError_t launch_thumbnails(const ThumbBatch &b, cudaStream_t s)
{
    if (b.n <= 0) return cudaSuccess;
    bool rows = b.w >= 512;
    for (int i = 0; i < b.n && rows; i++) {
        const unsigned a = b.f[i].bytes == 2 ? 16u : 8u;
        rows = ((uintptr_t)b.f[i].y % a) == 0 && b.f[i].ypitch % a == 0 && (b.f[i].bytes == 2 || b.f[i].shift < 8);
    }
    LaunchTimer t("align_thumbnails", s);
    if (rows) thumb_rows_kernel<<<dim3(kThumbH, b.n), 256, 0, s>>>(b);
    else thumb_kernel<<<dim3(kThumbW, kThumbH, b.n), 256, 0, s>>>(b);
    return after_launch();
}

cudaError_t launch_offset_totals(const float *ref, int n_ref, const float *probe, int n_probe, double *totals, cudaStream_t s)
{
    const int lags = n_ref - n_probe + 1;
    if (lags <= 0) return cudaSuccess;
    const bool vec = (((uintptr_t)ref | (uintptr_t)probe) & 15) == 0;  // rows of 2304 floats keep the alignment
    const bool exact = n_probe <= kExactMaxProbe && (n_probe + kExFrames - 1) / kExFrames <= 65535;
    if (exact) {
        unsigned long long *sums = (unsigned long long *)totals;
        cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(double) * (size_t)lags, s);
        if (e != cudaSuccess) return e;
        {
            LaunchTimer t("align_offset_check", s);
            offset_check_kernel<<<n_ref + n_probe, kExThreads, 0, s>>>(ref, n_ref, probe, n_probe, lags, sums);
        }
        if ((e = after_launch()) != cudaSuccess) return e;
        {
            LaunchTimer t("align_offset_exact", s);
            const dim3 grid((lags + kExLags - 1) / kExLags, (n_probe + kExFrames - 1) / kExFrames, kThumbPixels / kExPixels);
            e = launch_kernel(true, offset_exact_kernel, grid, kExThreads, 0, s, ref, probe, n_probe, lags, sums);
        }
        if (e != cudaSuccess) return e;
    }
    LaunchTimer t("align_offset_totals", s);
    const auto kernel = vec ? exact ? offset_totals_kernel<true, true> : offset_totals_kernel<true, false>
                            : exact ? offset_totals_kernel<false, true> : offset_totals_kernel<false, false>;
    return launch_kernel(exact, kernel, dim3((lags + kLagWarps - 1) / kLagWarps), 32 * kLagWarps, 0, s, ref, probe, n_probe, lags, totals);
}

namespace {
constexpr int kTotalsLags = 2048, kTotalsSlots = 8;
static __device__ double g_totals[kTotalsSlots][kTotalsLags];
}  // namespace

int offset_totals_slots() { return kTotalsSlots; }
int offset_totals_slot_lags() { return kTotalsLags; }
cudaError_t offset_totals_slot(int slot, double **ptr)
{
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_totals);
    *ptr = (double *)p + (size_t)slot * kTotalsLags;
    return e;
}

}  // namespace es
