// Per-frame measures other than CAMBI, for sm_100a: frame unpacking, the detail / structure-tensor window energies,
// the lasting-texture statistics, PSNR squared errors, color sums and the per-frame reduction into segment figures.
//
// The reference (src/kernels.cu:297-484, src/main.cpp:518-643) computes the window energies in FP32 from exact box
// sums, writes two full FP32 mid-detail planes per encode, re-reads 13 of them per encode for the lasting texture and
// reduces the windows on the host. Here every figure is computed from integer numerators (fine x 9, mid x 81,
// gradients x 9) summed exactly in int64 and rounded once; the lasting texture keeps running integer sums of the
// source's luma over the even and odd frame offsets (mid detail is linear in luma), so a frame step reads a few
// 16-bit planes once for all encodes; and the per-frame reduction (structure threshold as an exact order statistic,
// masks, sums, histogram bins) runs on the device.
#include <type_traits>

#include "es_kernels.h"

namespace es {
namespace {

// ---------------------------------------------------------------------------------------------------------------
// Frame unpacking: src/kernels.cu:289-310.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned sample_at(const void *plane, int pitch, int x, int y, const FrameViewDev &f)
{
    const unsigned char *row = (const unsigned char *)plane + (size_t)y * pitch;
    const unsigned v = f.bytes == 1 ? row[x] : ((const uint16_t *)row)[x];
    return v >> f.shift;
}

// 8 samples from p as four words of two 16-bit samples: one load where the address allows, else four loads of two samples,
// else one by one.
__device__ __forceinline__ uint4 load8(const unsigned char *p, int bytes)
{
    const uintptr_t at = (uintptr_t)p;
    if (bytes == 2) {
        if ((at & 15) == 0) return __ldg((const uint4 *)p);
        const unsigned *q = (const unsigned *)p;
        if ((at & 3) == 0) return make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
        const uint16_t *r = (const uint16_t *)p;
        auto two = [&](int k) { return (unsigned)__ldg(r + k) | ((unsigned)__ldg(r + k + 1) << 16); };
        return make_uint4(two(0), two(2), two(4), two(6));
    }
    if ((at & 7) == 0) {
        const uint2 q = __ldg((const uint2 *)p);
        return make_uint4(__byte_perm(q.x, 0, 0x4140), __byte_perm(q.x, 0, 0x4342), __byte_perm(q.y, 0, 0x4140), __byte_perm(q.y, 0, 0x4342));
    }
    if ((at & 1) == 0) {
        const uint16_t *r = (const uint16_t *)p;
        auto two = [&](int k) { return __byte_perm((unsigned)__ldg(r + k), 0, 0x4140); };
        return make_uint4(two(0), two(1), two(2), two(3));
    }
    auto two = [&](int k) { return (unsigned)__ldg(p + k) | ((unsigned)__ldg(p + k + 1) << 16); };
    return make_uint4(two(0), two(2), two(4), two(6));
}

// 4 samples from p, likewise.
__device__ __forceinline__ uint2 load4(const unsigned char *p, int bytes)
{
    const uintptr_t at = (uintptr_t)p;
    if (bytes == 2) {
        if ((at & 7) == 0) return __ldg((const uint2 *)p);
        const uint16_t *r = (const uint16_t *)p;
        auto two = [&](int k) { return (unsigned)__ldg(r + k) | ((unsigned)__ldg(r + k + 1) << 16); };
        return make_uint2(two(0), two(2));
    }
    if ((at & 3) == 0) {
        const unsigned q = __ldg((const unsigned *)p);
        return make_uint2(__byte_perm(q, 0, 0x4140), __byte_perm(q, 0, 0x4342));
    }
    auto two = [&](int k) { return (unsigned)__ldg(p + k) | ((unsigned)__ldg(p + k + 1) << 16); };
    return make_uint2(two(0), two(2));
}

// 8 (4) samples to p, which is 4-byte (2-byte) aligned at least: rows of even widths.
__device__ __forceinline__ void store8(uint16_t *p, uint4 v)
{
    const uintptr_t at = (uintptr_t)p;
    if ((at & 15) == 0) {
        *(uint4 *)p = v;
    } else if ((at & 7) == 0) {
        *(uint2 *)p = make_uint2(v.x, v.y);
        *(uint2 *)(p + 4) = make_uint2(v.z, v.w);
    } else {
        unsigned *q = (unsigned *)p;
        q[0] = v.x;
        q[1] = v.y;
        q[2] = v.z;
        q[3] = v.w;
    }
}
__device__ __forceinline__ void store4(uint16_t *p, uint2 v)
{
    const uintptr_t at = (uintptr_t)p;
    if ((at & 7) == 0) {
        *(uint2 *)p = v;
    } else if ((at & 3) == 0) {
        ((unsigned *)p)[0] = v.x;
        ((unsigned *)p)[1] = v.y;
    } else {
        p[0] = (uint16_t)v.x;
        p[1] = (uint16_t)(v.x >> 16);
        p[2] = (uint16_t)v.y;
        p[3] = (uint16_t)(v.y >> 16);
    }
}

// Thread i takes 4 consecutive 2 x 2 groups of one chroma row (2 rows x 8 luma columns, 4 samples of U and of V), planar
// or semi-planar, with the widest loads and stores each address allows; the last columns of a chroma row that is no
// multiple of 4 go one sample at a time. Bound by HBM: two 3840 x 2160 P010 frames took 40 us one
// sample at a time, 20 us now.
__global__ void __launch_bounds__(256) unpack_kernel(const __grid_constant__ UnpackBatch b)
{
    const int j = find_job(b.njobs, (int)blockIdx.x, [&](int k) { return b.job[k].first_block; });
    const UnpackJob &J = b.job[j];
    const FrameViewDev f = b.views ? b.views[j].f : J.f;
    const int x0 = b.views ? b.views[j].x0 : J.x0, y0 = b.views ? b.views[j].y0 : J.y0;
    const int cw = J.w / 2, ch = J.h / 2, qw = (cw + 3) / 4;
    const int i = (blockIdx.x - J.first_block) * 256 + threadIdx.x;
    if (i >= qw * ch) return;
    const int cy = i / qw, cx0 = 4 * (i - cy * qw), up = J.pd - f.depth;
    if (cx0 + 4 <= cw) {
        const unsigned mask = ((f.bytes == 1 ? 0xFFu : 0xFFFFu) >> f.shift) * 0x10001u;
        auto put = [&](unsigned q) { return ((q >> f.shift) & mask) << up; };
        uint4 y[2];
#pragma unroll
        for (int dy = 0; dy < 2; dy++)
            y[dy] = load8((const unsigned char *)f.y + (size_t)(2 * cy + dy + y0) * f.ypitch + (size_t)(2 * cx0 + x0) * f.bytes, f.bytes);
        const size_t co = (size_t)(cy + y0 / 2) * f.cpitch;
        uint2 u, v;
        if (f.semi) {  // (U, V) pairs
            const uint4 q = load8((const unsigned char *)f.u + co + (size_t)(2 * cx0 + x0) * f.bytes, f.bytes);
            u = make_uint2(__byte_perm(q.x, q.y, 0x5410), __byte_perm(q.z, q.w, 0x5410));
            v = make_uint2(__byte_perm(q.x, q.y, 0x7632), __byte_perm(q.z, q.w, 0x7632));
        } else {
            u = load4((const unsigned char *)f.u + co + (size_t)(cx0 + x0 / 2) * f.bytes, f.bytes);
            v = load4((const unsigned char *)f.v + co + (size_t)(cx0 + x0 / 2) * f.bytes, f.bytes);
        }
#pragma unroll
        for (int dy = 0; dy < 2; dy++)
            store8(J.y16 + (size_t)(2 * cy + dy) * J.w + 2 * cx0, make_uint4(put(y[dy].x), put(y[dy].y), put(y[dy].z), put(y[dy].w)));
        store4(J.u16 + (size_t)cy * cw + cx0, make_uint2(put(u.x), put(u.y)));
        store4(J.v16 + (size_t)cy * cw + cx0, make_uint2(put(v.x), put(v.y)));
        return;
    }
    for (int cx = cx0; cx < cw; cx++) {
#pragma unroll
        for (int dy = 0; dy < 2; dy++) {
            const int y = 2 * cy + dy;
            const unsigned a = sample_at(f.y, f.ypitch, 2 * cx + x0, y + y0, f);
            const unsigned c = sample_at(f.y, f.ypitch, 2 * cx + 1 + x0, y + y0, f);
            *(uint32_t *)(J.y16 + (size_t)y * J.w + 2 * cx) = (a << up) | ((c << up) << 16);
        }
        const int sx = (2 * cx + x0) / 2, sy = (2 * cy + y0) / 2;
        const unsigned u = f.semi ? sample_at(f.u, f.cpitch, 2 * sx, sy, f) : sample_at(f.u, f.cpitch, sx, sy, f);
        const unsigned v = f.semi ? sample_at(f.u, f.cpitch, 2 * sx + 1, sy, f) : sample_at(f.v, f.cpitch, sx, sy, f);
        J.u16[(size_t)cy * cw + cx] = (uint16_t)(u << up);
        J.v16[(size_t)cy * cw + cx] = (uint16_t)(v << up);
    }
}

constexpr int kM = 4;  // margin of a staged region: the 9 x 9 box reaches 4 pixels

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float exact_ratio(long long num, double den) { return __double2float_rn(__ddiv_rn((double)num, den)); }

__device__ __forceinline__ float oriented_of(long long jxx, long long jyy, long long jxy)
{
    const double d = (double)(jxx - jyy), x = (double)jxy;
    const double s = __dadd_rn(__dmul_rn(d, d), __dmul_rn(4.0, __dmul_rn(x, x)));
    return __double2float_rn(__ddiv_rn(__dsqrt_rn(s), 81.0));
}

// ---------------------------------------------------------------------------------------------------------------
// Window statistics of one source frame against every encode: src/kernels.cu:346-428, exact.
//
// A block of 128 threads takes a 64 x 64 tile (4 x 4 windows) of every picture in turn. Per picture: the 72 x 72 region
// (4-pixel margin, coordinates clamped) is copied in asynchronously while the picture before is summed; the horizontal 3-
// and 9-sums of 8 columns of a region row are made from two 16-byte reads, two columns to a word (no sum leaves 16 bits);
// then thread (c, g) walks tile columns 2 c and 2 c + 1 down rows 16 g .. 16 g + 15 (two columns of one window) with
// running vertical sums, the 3 x 3 sums two to a word. The 8 lanes of a window reduce its sums with shuffles.
// Bound by integer issue. With one column per thread and one sum per word it took 121 us for a 3840 x 2160 source and
// three encodes and 247 us for 16 uneven pairs; now 88 and 171 us. (The dot-product form of add_half pays for the 9 x 9
// sums; used for the fine details and gradients too it made 102 and 203 us of these.)
// ---------------------------------------------------------------------------------------------------------------
constexpr int kWT = 64;             // tile side
constexpr int kWR = kWT + 2 * kM;   // region side, 72
constexpr int kWS = 72;             // row stride of the region planes (144 bytes, a multiple of 16)
constexpr int kWThreads = 128;

using Region = uint16_t[kWR][kWS];  // [r][j]: pixel (x0 - 4 + j, y0 - 4 + r) of a plane, coordinates clamped

struct WinSums {
    uint16_t h3[kWR][kWS];  // h3[r][k]: 3-sum of row r centred at x0 - 1 + k, k < 66
    uint16_t h9[kWR][kWT];  // h9[r][c]: 9-sum of row r centred at x0 + c
};

// h3 and h9 of every region row: item (r, s) covers columns 8 s .. 8 s + 7 from y[r][8 s .. 8 s + 15]; the sums are
// shifted left by `up`. Pairs of neighbouring columns: p[k] holds columns 2 k and 2 k + 1, the pair one column on is one
// byte permutation, and a pair of 9-sums is three pairs of 3-sums three columns apart.
__device__ __forceinline__ void window_horizontal_sums(WinSums &sm, const Region &y, int up)
{
    for (int i = threadIdx.x; i < kWR * 8; i += kWThreads) {
        const int r = i >> 3, c0 = 8 * (i & 7);
        const uint4 a = *(const uint4 *)&y[r][c0], b = *(const uint4 *)&y[r][c0 + 8];
        const unsigned p[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        auto next = [](unsigned lo, unsigned hi) { return __byte_perm(lo, hi, 0x5432); };
        unsigned t[7];  // t[k]: 3-sums from columns 2 k and 2 k + 1 on
#pragma unroll
        for (int k = 0; k < 7; k++) t[k] = p[k] + next(p[k], p[k + 1]) + p[k + 1];
        unsigned h9[4];
#pragma unroll
        for (int k = 0; k < 4; k++) h9[k] = (t[k] + next(t[k + 1], t[k + 2]) + t[k + 3]) << up;
        *(uint4 *)&sm.h9[r][c0] = make_uint4(h9[0], h9[1], h9[2], h9[3]);
        *(uint4 *)&sm.h3[r][c0] = make_uint4(t[1] << up, t[2] << up, t[3] << up, t[4] << up);
        if (c0 == 56) *(unsigned *)&sm.h3[r][64] = t[5] << up;
    }
}

// The sum over the 8 lanes of a window.
template <typename T>
__device__ __forceinline__ T window_sum(T v)
{
#pragma unroll
    for (int o = 4; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void cp_async8(void *dst_smem, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Queues the copy of `src`'s region at tile (x0, y0) into raw (unshifted; rows clamped): 8-byte asynchronous copies
// where the columns lie inside the picture and the rows are 8-byte aligned, else plain loads and stores now. Every
// thread commits one group of copies (possibly empty). kUnroll: a tile without a row to clamp takes its copies without a
// loop, 5 % of persist_kernel's time (window_stats has no registers left for their addresses: 174 against 171 us).
template <bool kUnroll>
__device__ __forceinline__ void stage_raw_async(Region &raw, const uint16_t *src, int w, int h, int x0, int y0)
{
    const bool vec = x0 >= kM && x0 + kWT + kM <= w && (w & 3) == 0 && ((uintptr_t)src & 7) == 0;
    if (kUnroll && vec && y0 >= kM && y0 + kWT + kM <= h) {
        // no row to clamp: thread (q, r) copies group q of rows r, r + 7, ...
        const int r = threadIdx.x / 18, q = threadIdx.x - 18 * r;
        if (r < 7) {
            const uint16_t *p = src + (size_t)(y0 - kM + r) * w + (x0 - kM) + 4 * q;
            uint16_t *to = &raw[r][4 * q];
#pragma unroll
            for (int k = 0; k < kWR / 7; k++) cp_async8(to + 7 * k * kWS, p + (size_t)(7 * k) * w);
            if (r < kWR % 7) cp_async8(to + kWR / 7 * 7 * kWS, p + (size_t)(kWR / 7 * 7) * w);
        }
    } else if (vec) {
        for (int i = threadIdx.x; i < kWR * 18; i += kWThreads) {
            const int r = i / 18, q = i - r * 18;
            const int y = min(max(y0 - kM + r, 0), h - 1);
            cp_async8(&raw[r][4 * q], src + (size_t)y * w + (x0 - kM) + 4 * q);
        }
    } else {
        for (int i = threadIdx.x; i < kWR * kWR; i += kWThreads) {
            const int r = i / kWR, j = i - r * kWR;
            const int x = min(max(x0 - kM + j, 0), w - 1), y = min(max(y0 - kM + r, 0), h - 1);
            raw[r][j] = src[(size_t)y * w + x];
        }
    }
    cp_async_commit();
}

// c + K times half `Hi` of a pair of unsigned 16-bit values: one instruction, beside the pipe of the additions and shifts.
template <int K, int Hi>
__device__ __forceinline__ int add_half(unsigned pair, int c)
{
    static_assert(K >= -128 && K < 128, "a signed byte");
    int d;
    asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(pair), "r"((K & 0xFF) << 8 * Hi), "r"(c));
    return d;
}

// Vertical running sums of two neighbouring columns (tile columns c, c + 1, c even) down a window's 16 rows: start at row
// r0 - 1's successor state, then next() once per row.
struct ColumnPair {
    const WinSums &sm;
    int c, row;            // tile row the sums are at
    unsigned a1, a2, b1, b2;  // h3 words (columns left of and at c; right of c and of c + 1) of rows row, row + 1
    unsigned l, r;            // 3 x 3 sums left of the pair's columns, right of them
    int n9[2];                // minus the 9 x 9 sums
    __device__ __forceinline__ unsigned h3(int t, int k) const { return *(const unsigned *)&sm.h3[t + kM][c + 2 * k]; }
    __device__ __forceinline__ unsigned h9(int t) const { return *(const unsigned *)&sm.h9[t + kM][c]; }
    __device__ __forceinline__ unsigned centre() const { return __byte_perm(l, r, 0x5432); }
    __device__ __forceinline__ ColumnPair(const WinSums &s, int c_, int r0) : sm(s), c(c_), row(r0)
    {
        a1 = h3(r0, 0);
        b1 = h3(r0, 1);
        a2 = h3(r0 + 1, 0);
        b2 = h3(r0 + 1, 1);
        l = h3(r0 - 1, 0) + a1 + a2;
        r = h3(r0 - 1, 1) + b1 + b2;
        n9[0] = n9[1] = 0;
#pragma unroll
        for (int k = -4; k <= 4; k++) add9<-1>(h9(r0 + k));
    }
    // the 3 x 3 sums of the row above the current one
    __device__ __forceinline__ unsigned centre_above() const
    {
        const unsigned a = h3(row - 2, 0) + h3(row - 1, 0) + a1, b = h3(row - 2, 1) + h3(row - 1, 1) + b1;
        return __byte_perm(a, b, 0x5432);
    }
    // the 3 x 3 sums on to the next row (first half), the 9 x 9 sums (second half)
    __device__ __forceinline__ void next3()
    {
        const unsigned a3 = h3(row + 2, 0), b3 = h3(row + 2, 1);
        l = a1 + a2 + a3;
        r = b1 + b2 + b3;
        a1 = a2;
        a2 = a3;
        b1 = b2;
        b2 = b3;
    }
    __device__ __forceinline__ void next9()
    {
        add9<-1>(h9(row + 5));
        add9<1>(h9(row - 4));
        row++;
    }
    template <int K>
    __device__ __forceinline__ void add9(unsigned v)
    {
        n9[0] = add_half<K, 0>(v, n9[0]);
        n9[1] = add_half<K, 1>(v, n9[1]);
    }
    // mid-detail numerator 9 S3 - S9 of the pair's column k
    template <int Hi>
    __device__ __forceinline__ int mid(unsigned here) const
    {
        return add_half<9, Hi>(here, n9[Hi]);
    }
};

struct WinStatsSmem {
    WinSums sm;
    Region raw[2];  // the next picture's region is copied in while the current one is summed
};

__global__ void __launch_bounds__(kWThreads, 4) window_stats_kernel(const __grid_constant__ WindowBatch B)
{
    extern __shared__ __align__(16) unsigned char win_dyn[];
    WinStatsSmem &ws = *(WinStatsSmem *)win_dyn;
    const int jb = find_job(B.njobs, (int)blockIdx.x, [&](int k) { return B.job[k].first_block; });
    const WindowJob &J = B.job[jb];
    const int bid = blockIdx.x - J.first_block;
    const int w = J.w, h = J.h, ww = w / kWin, wh = h / kWin;
    const int tiles_x = (ww + 3) / 4;
    const int x0 = (bid % tiles_x) * kWT, y0 = (bid / tiles_x) * kWT;
    const int tid = threadIdx.x, lane = tid & 31;
    const int c = 2 * lane, r0 = (tid >> 5) * kWin;  // tile columns c and c + 1, first tile row
    const int wx = (x0 + c) / kWin, wy = (y0 + r0) / kWin;
    const bool inside = wx < ww && wy < wh;
    const int x = x0 + c, up = J.up;
    const bool gx_on[2] = {x > 0 && x < w - 1, x + 1 < w - 1};
    unsigned long long src_f = 0, src_m = 0, src_xx = 0, src_yy = 0;
    long long src_xy = 0;
    unsigned fr[kWin] = {};  // the source's fine numerators of the thread's pixels (|f| <= 9 x 1023: 16 bits each)
    int mr[kWin][2] = {};    // and its mid numerators, for the encodes' cross products
    auto walk = [&](auto first, const Region &raw, int p) {
        constexpr bool kFirst = decltype(first)::value;
        ColumnPair s(ws.sm, c, r0);
        unsigned above = s.centre_above(), here = s.centre();
        unsigned fine_sq = 0, jxx = 0, jyy = 0;
        int jxy[2] = {0, 0}, fine_x[2] = {0, 0};  // 16 products each stay below 2^31
        unsigned long long mid_sq = 0;
        long long mid_x = 0;
#pragma unroll
        for (int i = 0; i < kWin; i++) {
            const int y = y0 + r0 + i;
            const bool gy_on = y > 0 && y < h - 1;
            const unsigned v = *(const unsigned *)&raw[r0 + i + kM][c + kM] << up, left = s.l, right = s.r;
            s.next3();  // the next row's 3 x 3 sums, for the vertical gradient
            const unsigned below = s.centre();
            // differences of pairs, 0x8000 added to each half so that nothing is borrowed between them
            const unsigned dx = right + 0x80008000u - left, dy = below + 0x80008000u - above;
            unsigned f16[2];
            auto column = [&](auto which) {
                constexpr int k = decltype(which)::value;
                auto half = [&](unsigned q) { return (int)(k ? q >> 16 : q & 0xFFFFu); };
                const int s3 = half(here), f = 9 * half(v) - s3, m = 9 * s3 + s.n9[k];
                const int gx = gx_on[k] ? half(dx) - 0x8000 : 0, gy = gy_on ? half(dy) - 0x8000 : 0;
                f16[k] = (unsigned)f;
                if (kFirst) {
                    mr[i][k] = m;
                } else {
                    fine_x[k] += f * (k ? (int)fr[i] >> 16 : (int)(short)fr[i]);
                    mid_x += (long long)m * mr[i][k];
                }
                fine_sq += (unsigned)(f * f);
                mid_sq += (unsigned long long)((long long)m * m);
                jxx += (unsigned)(gx * gx);
                jyy += (unsigned)(gy * gy);
                jxy[k] += gx * gy;
            };
            column(std::integral_constant<int, 0>{});
            column(std::integral_constant<int, 1>{});
            if (kFirst) fr[i] = __byte_perm(f16[0], f16[1], 0x5410);
            above = here;
            here = below;
            if (i + 1 < kWin) s.next9();
        }
        const unsigned long long sf = window_sum((unsigned long long)fine_sq), sm2 = window_sum(mid_sq),
                                 sxx = window_sum((unsigned long long)jxx), syy = window_sum((unsigned long long)jyy);
        const long long sxy = window_sum((long long)jxy[0] + jxy[1]);
        if (kFirst) {
            src_f = sf;
            src_m = sm2;
            src_xx = sxx;
            src_yy = syy;
            src_xy = sxy;
            return;
        }
        const long long cf = window_sum((long long)fine_x[0] + fine_x[1]), cm = window_sum(mid_x);
        if (inside && (lane & 7) == 0) {
            float *o = J.stats + (((size_t)(p - 1) * wh + wy) * ww + wx) * 8;
            o[0] = exact_ratio((long long)src_f, 81.0);
            o[1] = exact_ratio((long long)src_m, 6561.0);
            o[2] = exact_ratio((long long)sf, 81.0);
            o[3] = exact_ratio((long long)sm2, 6561.0);
            o[4] = exact_ratio(cf, 81.0);
            o[5] = exact_ratio(cm, 6561.0);
            o[6] = oriented_of((long long)src_xx, (long long)src_yy, src_xy);
            o[7] = oriented_of((long long)sxx, (long long)syy, sxy);
        }
    };
    wait_for_previous();
    stage_raw_async<false>(ws.raw[0], J.yr, w, h, x0, y0);
    for (int p = 0; p <= J.nenc; p++) {
        const Region &raw = ws.raw[p & 1];
        __syncthreads();  // the walk of picture p - 1 is done with the buffer picture p + 1 goes to
        if (p < J.nenc) {
            stage_raw_async<false>(ws.raw[(p + 1) & 1], J.yd[p], w, h, x0, y0);
            cp_async_wait<1>();  // picture p's copies are in; p + 1's may still be in flight
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        window_horizontal_sums(ws.sm, raw, up);
        __syncthreads();
        if (p == 0) walk(std::true_type{}, raw, p);
        else walk(std::false_type{}, raw, p);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Lasting texture: src/kernels.cu:435-451, exact, from running luma sums (see PersistJob).
//
// advance_kernel moves the running sums E and O on by a frame, 8 pixels per thread with 16-byte accesses: a pass over six
// planes in and two out, bound by memory. persist_kernel then treats E, O, the centre frame and the encodes' pictures as
// window_stats treats its pictures: regions copied in asynchronously, horizontal sums, and thread (c, g) walks tile
// columns 2 c and 2 c + 1 down window row g with running vertical sums of the mid-detail numerators. When each tile
// advanced its own region of the sums first, the scattered 8-byte loads of that part alone took 59 of 98 us for a 3840 x
// 2160 pair at 20 % of the memory's rate. One kernel with a column per thread took 82 us for that pair, 107 us with three
// encodes and 317 us for 16 uneven pairs; the two now take 75, 99 and 280 us, of which 26, 26 and 93 us advance.
// ---------------------------------------------------------------------------------------------------------------
struct AdvanceJob {
    const uint16_t *e_old, *o_old, *y_m13, *y_m7, *y_c, *y_f;
    uint16_t *e_new, *o_new;
    size_t n;
    int up, first_block;
};
struct AdvanceBatch {
    AdvanceJob job[kMaxSources];
    int njobs;
};
constexpr int kAdvThreads = 256;
constexpr int kAdvPixels = 8 * kAdvThreads;  // per block

__global__ void __launch_bounds__(kAdvThreads) advance_kernel(const __grid_constant__ AdvanceBatch B)
{
    wait_for_previous();
    const int jb = find_job(B.njobs, (int)blockIdx.x, [&](int k) { return B.job[k].first_block; });
    const AdvanceJob &J = B.job[jb];
    const size_t at = (size_t)(blockIdx.x - J.first_block) * kAdvPixels + 8 * threadIdx.x;
    if (at >= J.n) return;
    const int up = J.up;
    // E(c) = O(c-1) - y(c) + y(c+6), O(c) = E(c-1) - y(c-7) + y(c-1); a missing frame is 0
    uintptr_t align = (uintptr_t)J.e_old | (uintptr_t)J.o_old | (uintptr_t)J.e_new | (uintptr_t)J.o_new;
    align |= (uintptr_t)J.y_m13 | (uintptr_t)J.y_m7 | (uintptr_t)J.y_c | (uintptr_t)J.y_f;
    if (at + 8 <= J.n && (align & 15) == 0) {
        auto load = [&](const uint16_t *p) { return p ? __ldg((const uint4 *)(p + at)) : make_uint4(0, 0, 0, 0); };
        const uint4 a = load(J.o_old), b = load(J.y_c), c = load(J.y_f), d = load(J.e_old), e = load(J.y_m13), f = load(J.y_m7);
        // no element leaves 0 .. 65535 (the leaving frame is part of the old sum), so 32-bit arithmetic on the pairs
        // carries and borrows nothing between the halves
        *(uint4 *)(J.e_new + at) = make_uint4(a.x - (b.x << up) + (c.x << up), a.y - (b.y << up) + (c.y << up),
                                              a.z - (b.z << up) + (c.z << up), a.w - (b.w << up) + (c.w << up));
        *(uint4 *)(J.o_new + at) = make_uint4(d.x - (e.x << up) + (f.x << up), d.y - (e.y << up) + (f.y << up),
                                              d.z - (e.z << up) + (f.z << up), d.w - (e.w << up) + (f.w << up));
        return;
    }
    const size_t end = J.n < at + 8 ? J.n : at + 8;
    for (size_t k = at; k < end; k++) {
        auto value = [&](const uint16_t *p) { return p ? (int)(p[k] << up) : 0; };
        J.e_new[k] = (uint16_t)((int)J.o_old[k] - value(J.y_c) + value(J.y_f));
        J.o_new[k] = (uint16_t)((int)J.e_old[k] - value(J.y_m13) + value(J.y_m7));
    }
}

// put(i, k, m): the mid-detail numerator 9 S3 - S9 of row r0 + i, column c + k, from the horizontal sums
template <typename Put>
__device__ __forceinline__ void window_mids(const WinSums &sm, int c, int r0, Put put)
{
    ColumnPair s(sm, c, r0);
#pragma unroll
    for (int i = 0; i < kWin; i++) {
        const unsigned here = s.centre();
        put(i, 0, s.mid<0>(here));
        put(i, 1, s.mid<1>(here));
        if (i + 1 < kWin) {
            s.next3();
            s.next9();
        }
    }
}

// Dynamic shared memory of persist_kernel: the region's horizontal sums and two buffers of raw regions.
struct PersistSmem {
    WinSums sm;
    Region raw[2];
};

__global__ void __launch_bounds__(kWThreads, 4) persist_kernel(const __grid_constant__ PersistBatch B)
{
    extern __shared__ __align__(16) unsigned char persist_dyn[];
    PersistSmem &ps = *(PersistSmem *)persist_dyn;
    const int jb = find_job(B.njobs, (int)blockIdx.x, [&](int k) { return B.job[k].first_block; });
    const PersistJob &J = B.job[jb];
    const int bid = blockIdx.x - J.first_block;
    const int w = J.w, h = J.h, ww = w / kWin, wh = h / kWin;
    const int tiles_x = (ww + 3) / 4;
    const int x0 = (bid % tiles_x) * kWT, y0 = (bid / tiles_x) * kWT;
    const int tid = threadIdx.x, lane = tid & 31;
    const int c = 2 * lane, r0 = (tid >> 5) * kWin;
    const int wx = (x0 + c) / kWin, wy = (y0 + r0) / kWin;
    const bool inside = wx < ww && wy < wh;
    // pictures in turn: E, O, the centre frame, the encodes at the centre frame
    const int last = J.nenc + 2;
    wait_for_previous();
    auto stage = [&](int p) {
        const uint16_t *src = p == 0 ? J.e_new : p == 1 ? J.o_new : p == 2 ? J.y_c : J.yd[p - 3];
        stage_raw_async<true>(ps.raw[p & 1], src, w, h, x0, y0);
    };
    auto sums = [&](int p) {  // horizontal sums of picture p; picture p + 1's copies go on meanwhile
        __syncthreads();      // the sums of picture p - 1 are read, and its buffer takes picture p + 1
        if (p < last) {
            stage(p + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        window_horizontal_sums(ps.sm, ps.raw[p & 1], p < 2 ? 0 : J.up);
        __syncthreads();
    };
    int t[kWin][2] = {};  // A x 486 = mid x 81 of E, then T = A + B, x 972
    stage(0);
    sums(0);
    window_mids(ps.sm, c, r0, [&](int i, int k, int m) { t[i][k] = m; });
    long long sab = 0, saa = 0, sbb = 0;
    sums(1);
    window_mids(ps.sm, c, r0, [&](int i, int k, int m) {  // B x 486
        const int a = t[i][k];
        t[i][k] = a + m;
        sab += (long long)a * m;
        saa += (long long)a * a;
        sbb += (long long)m * m;
    });
    sab = window_sum(sab);
    saa = window_sum(saa);
    sbb = window_sum(sbb);
    long long own = 0;
    for (int p = 2; p <= last; p++) {
        sums(p);
        long long sp = 0;
        window_mids(ps.sm, c, r0, [&](int i, int k, int m) { sp += (long long)m * t[i][k]; });
        sp = window_sum(sp);
        if (p == 2) {
            own = sp;
            continue;
        }
        if (inside && (lane & 7) == 0) {
            float *o = J.out + (((size_t)(p - 3) * wh + wy) * ww + wx) * 5;
            o[0] = exact_ratio(own, 78732.0);
            o[1] = exact_ratio(sp, 78732.0);
            o[2] = exact_ratio(sab, 236196.0);
            o[3] = exact_ratio(saa, 236196.0);
            o[4] = exact_ratio(sbb, 236196.0);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// PSNR squared errors (src/kernels.cu:454-464) and color sums (470-484), exact integers; the color strength of each
// sample sqrt(du^2 + dv^2) is rounded to units of 2^-30 so its sum is exact too. The pictures of a job:
// 0 .. nenc-1 the encodes (squared errors against the source, and their colors), nenc the source's colors.
//
// A block takes kSumPixels neighbouring pixels of a picture, their luma and chroma. Bound by the latency of its loads and of
// the square roots. With 148 blocks a picture striding over all of it, two an SM of which every second (the source's) had a
// third of the work, it took 32 us for a 3840 x 2160 pair and 79 us for 16 uneven pairs; now 21 and 67 us (8192 pixels a
// block: 23 and 78 us; 32768: 21 and 64 us, but 15 against 12 us for a 1920 x 1080 pair).
// ---------------------------------------------------------------------------------------------------------------
constexpr int kSumPixels = 16384;

__global__ void __launch_bounds__(256, 4) pair_sums_kernel(const __grid_constant__ PairSumsBatch B)
{
    __shared__ unsigned long long part[8][6];
    const int jb = find_job(B.njobs, (int)blockIdx.x, [&](int k) { return B.job[k].first_block; });
    const PairSumsJob &J = B.job[jb];
    const size_t n = (size_t)J.w * J.h, cn = n / 4;
    const int blocks = (int)((n + kSumPixels - 1) / kSumPixels), chunk = (int)(blockIdx.x - J.first_block) % blocks;
    const int p = (int)(blockIdx.x - J.first_block) / blocks, tid = threadIdx.x;
    const bool src_only = p == J.nenc;
    const size_t k0 = (size_t)chunk * kSumPixels, k1 = min(k0 + kSumPixels, n), c0 = k0 / 4, c1 = min(c0 + kSumPixels / 4, cn);
    unsigned long long sy = 0, su = 0, sv = 0, cu = 0, cv = 0, cs = 0;
    // 8 samples per 16-byte load (the planes are allocated aligned); the remainder one at a time
    auto sq = [](unsigned a, unsigned b) -> unsigned {  // squared differences of two pairs of 16-bit samples
        const int d0 = (int)(a & 0xFFFFu) - (int)(b & 0xFFFFu), d1 = (int)(a >> 16) - (int)(b >> 16);
        return (unsigned)(d0 * d0 + d1 * d1);
    };
    if (!src_only) {
        const uint16_t *a = J.ry, *b = J.dy[p];
        const size_t kv = (((uintptr_t)a | (uintptr_t)b) & 15) ? k0 : k0 + (k1 - k0) / 8 * 8;
#pragma unroll 4
        for (size_t i = k0 / 8 + tid; i < kv / 8; i += 256) {
            const uint4 x = __ldg((const uint4 *)a + i), y = __ldg((const uint4 *)b + i);
            sy += sq(x.x, y.x) + sq(x.y, y.y) + sq(x.z, y.z) + sq(x.w, y.w);
        }
        for (size_t i = kv + tid; i < k1; i += 256) {
            const long long d = (long long)a[i] - (long long)b[i];
            sy += (unsigned long long)(d * d);
        }
    }
    const uint16_t *u = src_only ? J.ru : J.du[p], *v = src_only ? J.rv : J.dv[p];
    auto color = [&](unsigned uu, unsigned vv) {
        uu <<= J.up;
        vv <<= J.up;
        const int eu = (int)uu - 512, ev = (int)vv - 512;
        cu += uu;
        cv += vv;
        cs += (unsigned long long)__double2ll_rn(__dmul_rn(__dsqrt_rn((double)(eu * eu + ev * ev)), 1073741824.0));
    };
    const size_t cw = (((uintptr_t)u | (uintptr_t)v | (uintptr_t)J.ru | (uintptr_t)J.rv) & 15) ? c0 : c0 + (c1 - c0) / 8 * 8;
#pragma unroll 2
    for (size_t i = c0 / 8 + tid; i < cw / 8; i += 256) {
        const uint4 uq = __ldg((const uint4 *)u + i), vq = __ldg((const uint4 *)v + i);
        if (!src_only) {
            const uint4 ru = __ldg((const uint4 *)J.ru + i), rv = __ldg((const uint4 *)J.rv + i);
            su += sq(ru.x, uq.x) + sq(ru.y, uq.y) + sq(ru.z, uq.z) + sq(ru.w, uq.w);
            sv += sq(rv.x, vq.x) + sq(rv.y, vq.y) + sq(rv.z, vq.z) + sq(rv.w, vq.w);
        }
        const unsigned us[4] = {uq.x, uq.y, uq.z, uq.w}, vs[4] = {vq.x, vq.y, vq.z, vq.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            color(us[k] & 0xFFFFu, vs[k] & 0xFFFFu);
            color(us[k] >> 16, vs[k] >> 16);
        }
    }
    for (size_t i = cw + tid; i < c1; i += 256) {
        if (!src_only) {
            const long long du = (long long)J.ru[i] - (long long)u[i], dv = (long long)J.rv[i] - (long long)v[i];
            su += (unsigned long long)(du * du);
            sv += (unsigned long long)(dv * dv);
        }
        color(u[i], v[i]);
    }
    sy = warp_sum(sy); su = warp_sum(su); sv = warp_sum(sv);
    cu = warp_sum(cu); cv = warp_sum(cv); cs = warp_sum(cs);
    if ((tid & 31) == 0) {
        const unsigned long long mine[6] = {sy, su, sv, cu, cv, cs};
#pragma unroll
        for (int k = 0; k < 6; k++) part[tid >> 5][k] = mine[k];
    }
    __syncthreads();
    if (tid < 6) {
        unsigned long long sum = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) sum += part[k][tid];
        if (tid >= 3) atomicAdd(&J.color[p * 3 + tid - 3], sum);
        else if (!src_only) atomicAdd(&J.sse[p * 3 + tid], sum);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Per-frame reduction, src/main.cpp:606-641 with quantile() of 280-289 and Histogram::add's binning of
// src/stats.hpp:14-19, in three launches: (1) the structure threshold, an exact order statistic of the source's
// oriented figures by a 3-round radix select, and the frame's structure mask; (2) every window of every encode: its
// bins and the block's sums, added in a fixed order; (3) per encode the blocks' sums, in a fixed order -- so the
// figures are the same on every run.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kCT = 1024;  // threshold block
constexpr int kCW = 256;   // windows per block
constexpr int kThreshStage = 40960;  // oriented figures a threshold block stages in shared memory (160 KB)
__host__ __device__ inline int collect_blocks_dev(int windows) { return (windows + kCW - 1) / kCW; }

__device__ __forceinline__ uint16_t hist_bin(double pct)
{
    const double c = pct < -500.0 ? -500.0 : pct > 500.0 ? 500.0 : pct;
    return (uint16_t)llround(__ddiv_rn(__dadd_rn(c, 500.0), 0.05));
}

// The rank-th smallest (0-based) of the non-negative floats v[i * stride] (their bit patterns order as the values), by
// three radix rounds of 11, 11 and 10 bits; each warp adds the lanes that share a digit with one atomic.
__device__ unsigned select_kth(const float *v, int n, int stride, unsigned rank, unsigned *hist)
{
    __shared__ unsigned s_prefix, s_mask, s_rem;
    __shared__ unsigned warp_tot[kCT / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { s_prefix = 0; s_mask = 0; s_rem = rank; }
    for (int round = 0; round < 3; round++) {
        const int shift = round == 0 ? 21 : round == 1 ? 10 : 0, nb = round == 2 ? 1024 : 2048;
        for (int i = tid; i < 2048; i += kCT) hist[i] = 0;
        __syncthreads();
        const unsigned prefix = s_prefix, mask = s_mask;
        for (int i0 = tid - lane; i0 < n; i0 += kCT) {  // the same trip count for every lane of a warp
            const int i = i0 + lane;
            const unsigned bits = i < n ? __float_as_uint(v[(size_t)i * stride]) : 0u;
            const bool in = i < n && (bits & mask) == prefix;
            if (!__any_sync(0xffffffffu, in)) continue;  // after the first round most warps hold no candidate
            const unsigned d = in ? (bits >> shift) & (unsigned)(nb - 1) : 0xFFFFFFFFu;
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            if (in && lane == __ffs(peers) - 1) atomicAdd(&hist[d], (unsigned)__popc(peers));
        }
        __syncthreads();
        // the digit holding the rem-th smallest: thread t sums digits [t per, t per + per), a block scan places it
        const int per = nb / kCT;
        unsigned local = 0;
        for (int k = 0; k < per; k++) local += hist[tid * per + k];
        unsigned incl = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v2 = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v2;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        unsigned before = 0;
        for (int k = 0; k < warp; k++) before += warp_tot[k];
        incl += before;
        const unsigned rem = s_rem, excl = incl - local;
        __syncthreads();
        if (excl <= rem && rem < incl) {
            unsigned below = excl;
            int d = tid * per;
            while (below + hist[d] <= rem) below += hist[d++];
            s_rem = rem - below;
            s_prefix = prefix | ((unsigned)d << shift);
            s_mask = mask | ((unsigned)(nb - 1) << shift);
        }
        __syncthreads();
    }
    return s_prefix;
}

// The (rank + 1)-th smallest of the same floats, given bits a of the rank-th: a again when more than rank + 1 values
// are at most a, otherwise the least value above a (one pass instead of three radix rounds).
__device__ unsigned select_next(const float *v, int n, int stride, unsigned rank, unsigned a)
{
    __shared__ unsigned s_le, s_min;
    if (threadIdx.x == 0) { s_le = 0; s_min = 0xFFFFFFFFu; }
    __syncthreads();
    unsigned le = 0, mn = 0xFFFFFFFFu;
    for (int i = threadIdx.x; i < n; i += kCT) {
        const unsigned bits = __float_as_uint(v[(size_t)i * stride]);
        if (bits <= a) le++;
        else mn = min(mn, bits);
    }
    le = __reduce_add_sync(0xffffffffu, le);
    mn = __reduce_min_sync(0xffffffffu, mn);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_le, le);
        atomicMin(&s_min, mn);
    }
    __syncthreads();
    return s_le >= rank + 2 ? a : s_min;
}

// One block per source. With `staged` (every job has at most kThreshStage windows) the oriented figures, which sit
// 8 floats apart in the figure array, are first gathered into dynamic shared memory, so the radix rounds and the
// mask read them there.
__global__ void __launch_bounds__(kCT) collect_threshold_kernel(const __grid_constant__ CollectBatch B, int staged)
{
    __shared__ unsigned hist[2048];
    extern __shared__ float stage[];
    const CollectJob &J = B.job[blockIdx.x];
    const float *st = J.stats;  // the source's oriented figures are the same in every encode's array
    const int n = J.windows;
    const float *v = st + 6;
    int stride = 8;
    if (staged) {
#pragma unroll 8
        for (int i = threadIdx.x; i < n; i += kCT) stage[i] = __ldg(st + (size_t)i * 8 + 6);
        __syncthreads();
        v = stage;
        stride = 1;
    }
    // numpy's linear quantile at 0.8 of exact order statistics, in the reference's float / double arithmetic
    const double pos = 0.8 * (double)(n - 1);
    const unsigned lo = (unsigned)pos;
    const unsigned a_bits = select_kth(v, n, stride, lo, hist);
    const float a = __uint_as_float(a_bits);
    float q = a;
    if (lo + 1 < (unsigned)n) {
        const float b = __uint_as_float(select_next(v, n, stride, lo, a_bits));
        const float diff = __fsub_rn(b, a);
        q = __double2float_rn(__dadd_rn((double)a, __dmul_rn((double)diff, __dsub_rn(pos, (double)lo))));
    }
    if (threadIdx.x == 0) *J.threshold = q;
    for (int i = threadIdx.x; i < n; i += kCT) {
        const float o = v[(size_t)i * stride];
        J.mask[i] = o >= q && o > 0.0f;
    }
}

__global__ void __launch_bounds__(kCW) collect_windows_kernel(const __grid_constant__ CollectBatch B)
{
    __shared__ double part[kCW / 32][kCollectSums];
    int jb = 0;
    while (jb + 1 < B.njobs && (int)blockIdx.y >= B.job[jb + 1].first_enc) jb++;
    const CollectJob &J = B.job[jb];
    const int nb = collect_blocks_dev(J.windows);
    if ((int)blockIdx.x >= nb) return;  // the grid covers the job with the most windows
    const int e = blockIdx.y - J.first_enc, n = J.windows, i = blockIdx.x * kCW + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // sums: all_r[3] all_d[3] st_r[3] st_d[3] sh_all_x[2] sh_st_x[2] own mine n_structure n_lasting
    double v[kCollectSums];
#pragma unroll
    for (int k = 0; k < kCollectSums; k++) v[k] = 0.0;
    uint16_t bin[6];  // amount 0-2, matching 0-1 (valid on structure windows), lasting (valid where v[19] is 1)
    bool structure = false, lasting = false;
    if (i < n) {
        const float q = *J.threshold;
        const float *s = J.stats + ((size_t)e * n + i) * 8;
        const bool m = s[6] >= q && s[6] > 0.0f;
        structure = m;
        const double er[3] = {(double)s[0], (double)s[1], (double)s[6]}, ed[3] = {(double)s[2], (double)s[3], (double)s[7]};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k] = er[k];
            v[3 + k] = ed[k];
            if (m) {
                v[6 + k] = er[k];
                v[9 + k] = ed[k];
                bin[k] = hist_bin(__dmul_rn(100.0, __dsqrt_rn(__ddiv_rn(ed[k], fmax(er[k], 1e-9)))));
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const double x = (double)s[4 + k];
            v[12 + k] = x;
            if (m) {
                v[14 + k] = x;
                bin[3 + k] = hist_bin(__ddiv_rn(__dmul_rn(100.0, x), fmax(er[k], 1e-9)));
            }
        }
        v[18] = m ? 1.0 : 0.0;
        if (J.persist) {
            const float *ps = J.persist + ((size_t)e * n + i) * 5;
            const double agree = __ddiv_rn((double)ps[2], __dsqrt_rn(fmax(__dmul_rn((double)ps[3], (double)ps[4]), 1e-9)));
            if (J.centre_mask[i] && agree > 0.5 && ps[0] > 0.0f) {
                v[16] = (double)ps[0];
                v[17] = (double)ps[1];
                v[19] = 1.0;
                lasting = true;
                bin[5] = hist_bin(__ddiv_rn(__dmul_rn(100.0, (double)ps[1]), (double)ps[0]));
            }
        }
    }
    // the bins that count, compacted (a histogram does not depend on their order), straight to the host's memory: the
    // five structure arrays share one position per window, the lasting array has its own; a warp reserves its places with
    // one atomic each
    {
        uint16_t *bins = J.host_bins + (size_t)e * 6 * n;
        const unsigned below = (1u << lane) - 1u;
        const unsigned sm = __ballot_sync(0xffffffffu, structure), lm = __ballot_sync(0xffffffffu, lasting);
        unsigned sb = 0, lb = 0;
        if (sm && lane == 0) sb = atomicAdd(&J.bin_n[2 * e], (unsigned)__popc(sm));
        if (lm && lane == 0) lb = atomicAdd(&J.bin_n[2 * e + 1], (unsigned)__popc(lm));
        sb = __shfl_sync(0xffffffffu, sb, 0);
        lb = __shfl_sync(0xffffffffu, lb, 0);
        if (structure) {
            const unsigned at = sb + __popc(sm & below);
#pragma unroll
            for (int k = 0; k < 5; k++) bins[(size_t)k * n + at] = bin[k];
        }
        if (lasting) bins[(size_t)5 * n + lb + __popc(lm & below)] = bin[5];
    }
#pragma unroll
    for (int k = 0; k < kCollectSums; k++) {
        const double x = warp_sum(v[k]);
        if (lane == 0) part[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < kCollectSums) {
        double s = 0.0;
        for (int k = 0; k < kCW / 32; k++) s += part[k][threadIdx.x];
        J.partials[((size_t)e * nb + blockIdx.x) * kCollectSums + threadIdx.x] = s;
    }
}

// Warp k of an encode's block makes sum k: lane l adds the partials of blocks l, l + 32, ... in order, then a fixed
// shuffle tree adds the 32 lane sums (the same order on every run). The figures, the encode's squared errors and colors
// (the first block: also the source's colors) and its bin counts go to the host's memory; the copied sums and counts are
// cleared. (As three copies and two memory clears per source they cost the step 15 us of waiting on one another.)
__global__ void __launch_bounds__(32 * kCollectSums) collect_final_kernel(const __grid_constant__ CollectBatch B)
{
    wait_for_previous();
    int jb = 0;
    while (jb + 1 < B.njobs && (int)blockIdx.x >= B.job[jb + 1].first_enc) jb++;
    const CollectJob &J = B.job[jb];
    const int e = blockIdx.x - J.first_enc, k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto move = [&](unsigned long long *from, unsigned long long *to) {
        *to = *from;
        *from = 0;
    };
    const int t = threadIdx.x, c0 = 3 * J.nenc;  // the sums: squared errors, then the encodes' colors, then the source's
    if (t < 3) move(J.sums + 3 * e + t, J.host_sums + 3 * e + t);
    else if (t < 6) move(J.sums + c0 + 3 * e + t - 3, J.host_sums + c0 + 3 * e + t - 3);
    else if (t < 9 && e == 0) move(J.sums + 2 * c0 + t - 6, J.host_sums + 2 * c0 + t - 6);
    else if (t >= 32 && t < 34) {
        J.host_bin_n[2 * e + t - 32] = J.bin_n[2 * e + t - 32];
        J.bin_n[2 * e + t - 32] = 0;
    }
    const int nblocks = collect_blocks_dev(J.windows);
    double s = 0.0;
    for (int b = lane; b < nblocks; b += 32) s += J.partials[((size_t)e * nblocks + b) * kCollectSums + k];
    s = warp_sum(s);
    if (lane != 0) return;
    FrameFigures *f = J.host_fig + e;
    if (k < 3) f->all_r[k] = s;
    else if (k < 6) f->all_d[k - 3] = s;
    else if (k < 9) f->st_r[k - 6] = s;
    else if (k < 12) f->st_d[k - 9] = s;
    else if (k < 14) f->sh_all_x[k - 12] = s;
    else if (k < 16) f->sh_st_x[k - 14] = s;
    else if (k == 16) f->own = s;
    else if (k == 17) f->mine = s;
    else if (k == 18) f->n_structure = (unsigned)s;
    else f->n_lasting = (unsigned)s;
    if (k == 0) f->threshold = *J.threshold;
}

}  // namespace

cudaError_t launch_unpack(const UnpackBatch &b, cudaStream_t s)
{
    if (b.total_blocks <= 0) return cudaSuccess;
    LaunchTimer t("frame_unpack", s);
    unpack_kernel<<<b.total_blocks, 256, 0, s>>>(b);
    return after_launch();
}

cudaError_t launch_window_stats(WindowBatch &b, cudaStream_t s)
{
    int blocks = 0;
    for (int j = 0; j < b.njobs; j++) {
        WindowJob &J = b.job[j];
        J.first_block = blocks;
        const int ww = J.w / kWin, wh = J.h / kWin;
        if (ww > 0 && wh > 0 && J.nenc > 0) blocks += ((ww + 3) / 4) * ((wh + 3) / 4);
    }
    if (blocks == 0) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(window_stats_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(WinStatsSmem));
    if (e != cudaSuccess) return e;
    LaunchTimer t("window_stats", s);
    return launch_kernel(true, window_stats_kernel, dim3(blocks), kWThreads, sizeof(WinStatsSmem), s, b);
}

cudaError_t launch_persist(PersistBatch &b, cudaStream_t s)
{
    AdvanceBatch ab{};
    size_t advance = 0;
    int blocks = 0;
    for (int j = 0; j < b.njobs; j++) {
        PersistJob &J = b.job[j];
        const size_t n = (size_t)J.w * J.h;
        ab.job[ab.njobs++] = AdvanceJob{J.e_old, J.o_old, J.y_m13, J.y_m7, J.y_c, J.y_f, J.e_new, J.o_new, n, J.up, (int)advance};
        advance += (n + kAdvPixels - 1) / kAdvPixels;
        J.first_block = blocks;
        if (J.stats) blocks += ((J.w / kWin + 3) / 4) * ((J.h / kWin + 3) / 4);
    }
    if (advance == 0) return cudaSuccess;
    LaunchTimer t("persist_stats", s);
    cudaError_t e = launch_kernel(true, advance_kernel, dim3((unsigned)advance), kAdvThreads, 0, s, ab);
    if (e != cudaSuccess || blocks == 0) return e;
    e = cudaFuncSetAttribute(persist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PersistSmem));
    if (e != cudaSuccess) return e;
    return launch_kernel(true, persist_kernel, dim3(blocks), kWThreads, sizeof(PersistSmem), s, b);
}

cudaError_t launch_pair_sums(PairSumsBatch &b, cudaStream_t s)
{
    size_t blocks = 0;
    for (int j = 0; j < b.njobs; j++) {
        b.job[j].first_block = (int)blocks;
        blocks += (((size_t)b.job[j].w * b.job[j].h + kSumPixels - 1) / kSumPixels) * (b.job[j].nenc + 1);
    }
    if (blocks == 0) return cudaSuccess;
    LaunchTimer t("pair_sums", s);
    pair_sums_kernel<<<(unsigned)blocks, 256, 0, s>>>(b);
    return after_launch();
}

int collect_blocks(int windows) { return collect_blocks_dev(windows); }

// Grid rows of each job's encodes, and the most collect blocks of a job; an error for a job without encodes or windows.
static cudaError_t collect_shape(CollectBatch &b, int &encs, int &nb, int &max_windows)
{
    encs = nb = max_windows = 0;
    for (int j = 0; j < b.njobs; j++) {
        if (b.job[j].nenc <= 0 || b.job[j].windows <= 0) return cudaErrorInvalidValue;
        b.job[j].first_enc = encs;
        encs += b.job[j].nenc;
        nb = nb > collect_blocks(b.job[j].windows) ? nb : collect_blocks(b.job[j].windows);
        max_windows = max_windows > b.job[j].windows ? max_windows : b.job[j].windows;
    }
    return cudaSuccess;
}

cudaError_t launch_collect_threshold(CollectBatch &b, cudaStream_t s)
{
    int encs, nb, max_windows;
    cudaError_t e = collect_shape(b, encs, nb, max_windows);
    if (e != cudaSuccess || encs == 0) return e;
    const int staged = max_windows <= kThreshStage;
    e = cudaFuncSetAttribute(collect_threshold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kThreshStage * (int)sizeof(float));
    if (e != cudaSuccess) return e;
    LaunchTimer t("frame_collect_threshold", s);
    collect_threshold_kernel<<<b.njobs, kCT, staged ? (size_t)max_windows * sizeof(float) : 0, s>>>(b, staged);
    return after_launch();
}

cudaError_t launch_collect_sums(CollectBatch &b, cudaStream_t s)
{
    int encs, nb, max_windows;
    cudaError_t e = collect_shape(b, encs, nb, max_windows);
    if (e != cudaSuccess || encs == 0) return e;
    {
        LaunchTimer t("frame_collect_windows", s);
        collect_windows_kernel<<<dim3(nb, encs), kCW, 0, s>>>(b);
    }
    e = after_launch();
    if (e != cudaSuccess) return e;
    LaunchTimer t("frame_collect_final", s);
    return launch_kernel(true, collect_final_kernel, dim3(encs), 32 * kCollectSums, 0, s, b);
}

// ---------------------------------------------------------------------------------------------------------------
// The VMAF picture feed: src/kernels.cu:537-545 (to_picture), one launch for every plane of a step. A thread moves 8
// samples of a row: one 16-byte load of the 16-bit values, and one 8-byte (8-bit picture) or 16-byte store where the
// destination row allows, else sample by sample. An 8-bit picture keeps the low byte of each value, as the reference.
// ---------------------------------------------------------------------------------------------------------------
namespace {
constexpr int kPicThreads = 256;

__global__ void __launch_bounds__(kPicThreads) to_pictures_kernel(const __grid_constant__ PictureBatch b)
{
    const int j = find_job(b.njobs, (int)blockIdx.x, [&](int k) { return b.job[k].first_block; });
    const PictureJob &J = b.job[j];
    const int groups = (J.w + 7) / 8;  // 8-sample groups per row
    const long long i = (long long)(blockIdx.x - J.first_block) * kPicThreads + threadIdx.x;
    if (i >= (long long)groups * J.h) return;
    const int y = (int)(i / groups), x = (int)(i - (long long)y * groups) * 8;
    const uint16_t *src = J.src + (size_t)y * J.w + x;
    char *row = (char *)J.dst + (size_t)y * J.pitch;
    const bool src_vec = (J.w & 7) == 0 && (((uintptr_t)J.src) & 15) == 0;
    if (src_vec && x + 8 <= J.w) {
        const uint4 q = __ldg((const uint4 *)src);
        if (J.bytes == 1) {
            uint8_t *d = (uint8_t *)row + x;
            const uint2 v = make_uint2(__byte_perm(q.x, q.y, 0x6420), __byte_perm(q.z, q.w, 0x6420));
            if ((((uintptr_t)d) & 7) == 0) {
                *(uint2 *)d = v;
            } else {
                for (int k = 0; k < 4; k++) d[k] = (uint8_t)(v.x >> (8 * k));
                for (int k = 0; k < 4; k++) d[4 + k] = (uint8_t)(v.y >> (8 * k));
            }
        } else {
            uint16_t *d = (uint16_t *)row + x;
            if ((((uintptr_t)d) & 15) == 0) {
                *(uint4 *)d = q;
            } else {
                const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
                for (int k = 0; k < 8; k++) d[k] = (uint16_t)(w4[k >> 1] >> (16 * (k & 1)));
            }
        }
        return;
    }
    for (int k = 0; k < 8 && x + k < J.w; k++) {
        const uint16_t v = src[k];
        if (J.bytes == 1) ((uint8_t *)row)[x + k] = (uint8_t)v;
        else ((uint16_t *)row)[x + k] = v;
    }
}

}  // namespace

cudaError_t launch_to_pictures(PictureBatch &b, cudaStream_t s)
{
    int blocks = 0;
    for (int j = 0; j < b.njobs; j++) {
        PictureJob &J = b.job[j];
        J.first_block = blocks;
        blocks += (int)(((long long)((J.w + 7) / 8) * J.h + kPicThreads - 1) / kPicThreads);
    }
    if (blocks <= 0) return cudaSuccess;
    LaunchTimer t("to_pictures", s);
    to_pictures_kernel<<<blocks, kPicThreads, 0, s>>>(b);
    return after_launch();
}

const void *kernel_entry_unpack() { return (const void *)unpack_kernel; }
const void *kernel_entry_window_stats() { return (const void *)window_stats_kernel; }
const void *kernel_entry_persist() { return (const void *)persist_kernel; }
const void *kernel_entry_pair_sums() { return (const void *)pair_sums_kernel; }
const void *kernel_entry_collect() { return (const void *)collect_windows_kernel; }

}  // namespace es
