// CAMBI (Contrast Aware Multiscale Banding Index) kernels for sm_100a.
//
// Per picture the reference (src/kernels.cu:14-278, src/cambi.cpp:88-184) copies or converts the plane, builds the
// zero-derivative mask, runs decimation and a mode filter per scale, counts windowed histograms into a full float
// c-value buffer that it clears every frame, and pools the top 60% with host-driven radix rounds. Here:
//
//  * prep0_kernel fuses the 8-to-10-bit conversion (or copy), the 7x7 flat-pixel count and the 3x3 mode filter of
//    scale 0 in one pass over a shared-memory tile, and packs each pixel as value | mask << 15, so every later step
//    reads one 16-bit word per pixel;
//  * the same kernel makes scale 1 and clears the counters; decimate_mode_kernel builds scales 2-4 from scale 1's words;
//  * the c-values themselves are in cvalues_kernels.cu;
//  * two launches of select_kernel and the score kernel find the exact k-th largest value, and the sum above it, on the
//    device when more than k values are positive (no host round trips; the first radix digit is counted by the c-value
//    kernel); the score kernel also pools and weights the scales and writes the score to the host's memory.
// A picture is six launches: scales 0 and 1, scales 2-4, the c-values, two top-k rounds, the score. They were twelve and a
// copy: a launch takes 2.5 to 5 us of host time and 3 to 5 us on the GPU here, as long as the work of most of them.
#include "cambi_codes.h"
#include "es_kernels.h"

namespace es {
namespace {

// The mode of three values (the smallest when all differ), as selects rather than branches: neighbouring pixels of a
// warp take different cases.
__device__ __forceinline__ uint16_t mode3(uint16_t a, uint16_t b, uint16_t c)
{
    const unsigned mn = min((unsigned)a, min((unsigned)b, (unsigned)c));
    const unsigned bc = b == c ? (unsigned)b : mn;
    return (uint16_t)((a == b || a == c) ? (unsigned)a : bc);
}

// ---------------------------------------------------------------------------------------------------------------
// Scales 0 and 1: src/kernels.cu:524-535 (from8), 14-40 (mask), 488-500 (mode), 43-53 (decimation), in one pass over a
// 64 x 64 tile of scale 0 and the 32 x 32 tile of scale 1 beneath it.
//
//  1. The plane is staged with its margins, 8 pixels per load, coordinates clamped to the picture. An 8-bit plane becomes
//     10-bit anti-dithered values in place: ((4 a + 4 b + 4 c + 4 d) >> 2) of a pixel and its right, lower and lower
//     right neighbours is a + b + c + d, and on the last row and column the clamped copies give the reference's pairs.
//  2. Flat pixels (equal to the right and lower neighbours; a clamped copy is equal) become bits, 8 per thread and step.
//  3. The 7 x 7 counts of flat pixels are made 32 columns at a time in bit-sliced form: the counts of 7 columns as three
//     bit planes (four full adders of three-input logic), then 7 rows of those as six planes, compared with mask_index.
//  4. Each warp walks 8 rows of the tile, a lane taking two neighbouring columns as the two halves of 32-bit words: the
//     3 x 3 mode filter reads both columns' neighbours with 32-bit loads.
//  5. The scale-0 words at even positions, with a ring of them one step outside the tile (made on their own), give the
//     tile's scale-1 words (decimation and mode filter of the decimated values) without another read of scale 0.
// Bound by integer issue (11 thousand warp instructions a tile, the ALU pipe 71 % busy). With counts by population count
// per pixel pair, flat bits by ballot and a longer mode filter it took 54 us for a 3840 x 2160 10-bit picture and 31 us
// for a 1920 x 1080 8-bit one; now 40 and 22 us.
// Staged region: columns x0-8 .. x0+71 (index x - (x0-8)), rows y0-5 .. y0+69 (index y - (y0-5)).
// ---------------------------------------------------------------------------------------------------------------
constexpr int kP0T = 64;                 // scale-0 tile side
constexpr int kP0C = 80, kP0R = 75;      // staged columns and rows
constexpr int kP0X = 8, kP0Y = 5;        // staged index of x0, y0
constexpr int kP0FR = 74;                // rows of flat bits (staged rows 0 .. 73); bit i of a row is staged column i
constexpr int kP0M = 66;                 // rows of mask bits: y0 - 2, y0 .. y0 + 63, y0 + 64
constexpr int kP0D = 34;                 // scale-0 words (x0-2+2X, y0-2+2Y), X, Y in 0 .. 33

__device__ __forceinline__ uint32_t vmin_u16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t vmax_u16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Bit 15 of each half, over the half.
__device__ __forceinline__ uint32_t sign_x2(uint32_t a)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(r) : "r"(a));
    return r;
}
// The mode of three values below 2^15 per 16-bit half (the smallest when all three differ): with two or three equal
// values the repeated one is the median, and it equals the largest unless the pair is the two smallest, when it equals
// the smallest; with three different values the mode is the smallest. So the mode is the largest where the median equals
// it, else the smallest. The halves' differences are never negative, so 32-bit subtraction keeps them apart.
__device__ __forceinline__ uint32_t mode3x2(uint32_t a, uint32_t b, uint32_t c)
{
    const uint32_t lo = vmin_u16x2(a, b), hi = vmax_u16x2(a, b);
    const uint32_t mn = vmin_u16x2(lo, c), mx = vmax_u16x2(hi, c), md = vmax_u16x2(lo, vmin_u16x2(hi, c));
    const uint32_t differ = sign_x2(mx - md + 0x7FFF7FFFu);
    return (mx & ~differ) | (mn & differ);
}

// One full adder on 32 columns: a + b + c = sum + 2 carry.
struct Planes3 {
    uint32_t p0, p1, p2;
};
__device__ __forceinline__ void full_add(uint32_t a, uint32_t b, uint32_t c, uint32_t &sum, uint32_t &carry)
{
    sum = a ^ b ^ c;
    carry = (a & b) | (a & c) | (b & c);
}
// The number of set bits among seven words, per column.
__device__ __forceinline__ Planes3 count7(const uint32_t (&v)[7])
{
    uint32_t s0, s1, c0, c1, c2;
    Planes3 r;
    full_add(v[0], v[1], v[2], s0, c0);
    full_add(v[3], v[4], v[5], s1, c1);
    full_add(s0, s1, v[6], r.p0, c2);
    full_add(c0, c1, c2, r.p1, r.p2);
    return r;
}

// 8 pixels of row y (inside the picture) from column x, clamped to 0 .. w - 1.
__device__ __forceinline__ uint4 plane8(const uint16_t *img, int pitch, int w, int y, int x, int align)
{
    const uint16_t *row = img + (size_t)y * pitch;
    if (x >= 0 && x + 8 <= w && align < 2) {
        if (align == 0) return __ldg((const uint4 *)(row + x));
        const uint32_t *q = (const uint32_t *)(row + x);
        return make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
    }
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = __ldg(row + min(max(x + k, 0), w - 1));
    return make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
}

// kStrips: every job has strips (a branch on them instead cost 12 of 267 us for 16 uneven pairs without any).
template <bool kStrips>
__global__ void __launch_bounds__(256, 5) prep0_kernel(const __grid_constant__ Prep0Batch b)
{
    wait_for_previous();
    if ((int)blockIdx.x >= b.total_tiles) {  // the blocks after the tiles clear the counters, a slot each
        const int i = blockIdx.x - b.total_tiles;
        CvSlot &S = b.slots[i];
        for (int k = threadIdx.x; k < 2048 / 4; k += 256) ((uint4 *)S.hist)[k] = make_uint4(0, 0, 0, 0);
        if (threadIdx.x == 0) {
            S.sum_fx = S.count = S.list_n = 0;
            S.n = b.slot_n[i];
            S.k = b.slot_k[i];
            S.above_fx = S.above_n = 0;
            if (i == 0 && b.clear) b.clear[0] = b.clear[1] = 0;
        }
        return;
    }
    __shared__ __align__(16) uint16_t buf[kP0R][kP0C];     // the staged plane at 10 bits
    __shared__ __align__(16) uint32_t flatbits[kP0FR][4];  // 80 bits a row, then zeros
    __shared__ uint32_t seven[kP0FR][9];                   // flat pixels among 7 columns: 3 planes of 3 words
    __shared__ uint32_t maskbits[kP0M][3];
    __shared__ __align__(4) uint16_t dw[kP0D][kP0D + 2];   // scale-0 words at even positions, for scale 1: word X at X + 1
    __shared__ uint32_t needbits[32];
    const int j = find_job(b.njobs, (int)blockIdx.x, [&](int k) { return b.job[k].first_tile; });
    const Prep0Job &J = b.job[j];
    const int t = blockIdx.x - J.first_tile, w = J.w, h = J.h, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int x0 = (t % J.tiles_x) * kP0T, y0 = (t / J.tiles_x) * kP0T;
    const int xs = x0 - kP0X, ys = y0 - kP0Y;
    if (J.feat && b.need_span < 0) {  // the codes that need c-values when they are no single range: bit c of word
                                      // c / 32 (warp w makes words w, w + 8, ...)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int code = (warp + 8 * k) * 32 + lane;
            const unsigned m = __ballot_sync(0xffffffffu, code < b.band.band_size && needs_cvalue(code, b.band));
            if (lane == 0) needbits[warp + 8 * k] = m;
        }
    }
    const int align = (J.pitch & 7) == 0 && (((uintptr_t)J.img) & 15) == 0 ? 0 : (J.pitch & 1) == 0 && (((uintptr_t)J.img) & 3) == 0 ? 1 : 2;
    constexpr int kQ = kP0C / 8;  // 8-pixel groups of a staged row
    for (int i = tid; i < kP0R * kQ; i += 256) {
        const int r = i / kQ, q = i - r * kQ;
        *(uint4 *)&buf[r][8 * q] = plane8(J.img, J.pitch, w, min(max(ys + r, 0), h - 1), xs + 8 * q, align);
    }
    if (tid < kP0FR) ((uint4 *)flatbits)[tid] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    // the pixels right of a group of 8, as a group
    auto right = [](uint4 v, uint32_t next) {
        return make_uint4(__byte_perm(v.x, v.y, 0x5432), __byte_perm(v.y, v.z, 0x5432), __byte_perm(v.z, v.w, 0x5432),
                          __byte_perm(v.w, next, 0x5432));
    };
    if (J.depth == 8) {
        uint4 sum[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {  // rows 0 .. 73; the last staged row is only read
            const int i = tid + 256 * k, r = i / kQ, q = i - r * kQ;
            sum[k] = make_uint4(0, 0, 0, 0);
            if (i < kP0FR * kQ) {
                const uint4 a = *(const uint4 *)&buf[r][8 * q], c = *(const uint4 *)&buf[r + 1][8 * q];
                // (the staged region's last column has no right neighbour and is not used)
                const uint4 ar = right(a, q < kQ - 1 ? buf[r][8 * q + 8] : 0u), cr = right(c, q < kQ - 1 ? buf[r + 1][8 * q + 8] : 0u);
                sum[k] = make_uint4(a.x + ar.x + c.x + cr.x, a.y + ar.y + c.y + cr.y, a.z + ar.z + c.z + cr.z, a.w + ar.w + c.w + cr.w);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int i = tid + 256 * k, r = i / kQ, q = i - r * kQ;
            if (i < kP0FR * kQ) *(uint4 *)&buf[r][8 * q] = sum[k];
        }
        __syncthreads();
    }
    // flat bits: rows of the picture 0 .. h - 1 and columns 0 .. w - 1 only. (The values of an 8-bit plane's last staged
    // row are not made; its flat row, 73, is not used.)
    for (int i = tid; i < kP0FR * kQ; i += 256) {
        const int r = i / kQ, q = i - r * kQ, x = xs + 8 * q, y = ys + r;
        if (y < 0 || y >= h || x < 0 || x >= w) continue;  // groups start at multiples of 8
        const uint4 a = *(const uint4 *)&buf[r][8 * q], ar = right(a, q < kQ - 1 ? buf[r][8 * q + 8] : 0u);
        uint4 c = *(const uint4 *)&buf[r + 1][8 * q];
        if (y == h - 1) c = a;  // (an 8-bit plane's values past the last row are sums of other copies)
        // per half: 0 when flat; values are below 2^15, so adding 0x7FFF sets bit 15 for every other one
        const uint32_t v[4] = {((a.x ^ ar.x) | (a.x ^ c.x)) + 0x7FFF7FFFu, ((a.y ^ ar.y) | (a.y ^ c.y)) + 0x7FFF7FFFu,
                               ((a.z ^ ar.z) | (a.z ^ c.z)) + 0x7FFF7FFFu, ((a.w ^ ar.w) | (a.w ^ c.w)) + 0x7FFF7FFFu};
        const uint32_t lo = ~__byte_perm(v[0], v[1], 0x7531) & 0x80808080u, hi = ~__byte_perm(v[2], v[3], 0x7531) & 0x80808080u;
        uint32_t bits = (((lo >> 7) * 0x10204080u) >> 28) | ((((hi >> 7) * 0x10204080u) >> 28) << 4);  // byte k's bit to bit k
        if (x + 8 >= w) {  // the last columns: column w - 1 has no right neighbour, nothing is flat past it
            const int n = w - x;  // 1 .. 8
            const uint32_t last = (n & 1) ? 0x0000FFFFu : 0xFFFF0000u, e = n <= 2 ? a.x ^ c.x : n <= 4 ? a.y ^ c.y : n <= 6 ? a.z ^ c.z : a.w ^ c.w;
            bits = (bits & ((1u << (n - 1)) - 1u)) | ((e & last) == 0 ? 1u << (n - 1) : 0u);
        }
        ((uint8_t *)flatbits[r])[q] = (uint8_t)bits;
    }
    __syncthreads();
    // flat pixels among the 7 columns around each column
    if (tid < kP0FR * 3) {
        const int r = tid / 3, k = tid - 3 * r;
        const uint32_t c = flatbits[r][k], l = k ? flatbits[r][k - 1] : 0u, n = flatbits[r][k + 1];
        const uint32_t v[7] = {__funnelshift_l(l, c, 3), __funnelshift_l(l, c, 2), __funnelshift_l(l, c, 1), c,
                               __funnelshift_r(c, n, 1), __funnelshift_r(c, n, 2), __funnelshift_r(c, n, 3)};
        const Planes3 p = count7(v);
        seven[r][k] = p.p0;
        seven[r][3 + k] = p.p1;
        seven[r][6 + k] = p.p2;
    }
    __syncthreads();
    // the mask: more than mask_index of the 49
    if (tid < kP0M * 3) {
        const int m = tid / 3, k = tid - 3 * m, r0 = (m == 0 ? 0 : m == kP0M - 1 ? 66 : m + 1);  // flat rows y - 3 .. y + 3
        Planes3 p[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            uint32_t v[7];
#pragma unroll
            for (int i = 0; i < 7; i++) v[i] = seven[r0 + i][3 * q + k];
            p[q] = count7(v);
        }
        // p[0] + 2 p[1] + 4 p[2], bit by bit
        uint32_t bit[6], c1, c2, c3, c4, c5, s;
        bit[0] = p[0].p0;
        bit[1] = p[0].p1 ^ p[1].p0;
        c1 = p[0].p1 & p[1].p0;
        full_add(p[0].p2, p[1].p1, p[2].p0, s, c2);
        bit[2] = s ^ c1;
        c3 = s & c1;
        full_add(p[1].p2, p[2].p1, c2, s, c4);
        bit[3] = s ^ c3;
        c5 = s & c3;
        full_add(p[2].p2, c4, c5, bit[4], bit[5]);
        uint32_t more = J.mask_index < 0 ? 0xFFFFFFFFu : 0u, equal = J.mask_index < 0 || J.mask_index > 63 ? 0u : 0xFFFFFFFFu;
#pragma unroll
        for (int q = 5; q >= 0; q--) {
            const uint32_t limit = (J.mask_index >> q) & 1 ? 0xFFFFFFFFu : 0u;
            more |= equal & bit[q] & ~limit;
            equal &= ~(bit[q] ^ limit);
        }
        maskbits[m][k] = more;
    }
    __syncthreads();

    // the walk: warp g makes rows y0 + 8 g .. + 7, lane l columns x0 + 2 l and + 1
    const int x = x0 + 2 * lane, g = warp;
    const int mw = (kP0X + 2 * lane) >> 5, ms = (kP0X + 2 * lane) & 31;  // the mask bit of column x
    // columns x and x + 1 at a picture edge keep their own value in the horizontal mode
    const uint32_t edge = ((x == 0 || x == w - 1) ? 0x0000FFFFu : 0u) | ((x + 1 == w - 1) ? 0xFFFF0000u : 0u);
    const int c = x - xs;  // staged column of x (even)
    auto pair = [&](int r, int cc) -> uint32_t { return *(const uint32_t *)&buf[r][cc]; };
    auto hmode = [&](int y) -> uint32_t {  // horizontal modes of x and x + 1 in picture row y
        const int r = y - ys;
        const uint32_t l2 = pair(r, c - 2), m2 = pair(r, c), r2 = pair(r, c + 2);
        const uint32_t left = __byte_perm(l2, m2, 0x5432), right = __byte_perm(m2, r2, 0x5432);
        return (m2 & edge) | (mode3x2(left, m2, right) & ~edge);
    };
    const bool feat = J.feat != nullptr;  // the same for the whole block
    const bool vec_store = (w & 1) == 0 && (((uintptr_t)J.word) & 3) == 0;
    const bool need_range = b.need_span >= 0;
    const int yb = y0 + 8 * g;
    uint32_t m0 = hmode(yb - 1), m1 = hmode(yb);
    // features of this lane's two columns over the current 4 rows, as 16-bit pairs (a pair holds 2 rows of sums of
    // values below 2^15, then it is folded into fsum; counts up to 4)
    uint32_t fsum = 0, fsum2 = 0, fmask2 = 0, fn2 = 0;
    // the smallest (value - need_lo) of the lane's masked pixels per half, wrapping for values below need_lo: a pixel
    // needs a c-value when it is at most need_span (unmasked pixels count as 0x8000, above any span)
    const uint32_t lo2 = (uint32_t)(b.need_lo & 0x7FFF) * 0x10001u;
    uint32_t dmin = 0xFFFFFFFFu;
    bool need = false;
    // the strip, per half: the least masked value (unmasked words count as 0x8000 and more) and the greatest (with the mask
    // bit; without it for none)
    uint32_t smin = 0xFFFFFFFFu, smax = 0;
    auto strip_word = [&](uint32_t word) {
        smin = vmin_u16x2(smin, word ^ 0x80008000u);
        smax = vmax_u16x2(smax, word);
    };
    // the warp's strip, from the halves of columns inside the picture
    auto strip_out = [&](unsigned *to, bool in0, bool in1) {
        const unsigned lo = min(in0 ? smin & 0xFFFFu : 0xFFFFu, in1 ? smin >> 16 : 0xFFFFu);
        const unsigned hi = max(in0 ? smax & 0xFFFFu : 0u, in1 ? smax >> 16 : 0u);
        const unsigned wlo = __reduce_min_sync(0xffffffffu, lo), whi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) *to = wlo | (whi & 0x7FFFu) << 16;
        smin = 0xFFFFFFFFu;
        smax = 0;
    };
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int y = yb + i;
        const uint32_t m2 = hmode(y + 1);
        uint32_t v2 = mode3x2(m0, m1, m2);
        if (y == 0 || y == h - 1) v2 = pair(y - ys, c);  // (the same for the whole warp)
        const uint32_t mb = maskbits[8 * g + i + 1][mw] >> ms;
        const uint32_t mk = ((mb << 15) & 0x8000u) | ((mb << 30) & 0x80000000u);
        const uint32_t word2 = v2 | mk;
        if (y < h) {
            if (kStrips) strip_word(word2);
            if (vec_store && x + 1 < w) {
                *(uint32_t *)(J.word + (size_t)y * w + x) = word2;
            } else {
                if (x < w) J.word[(size_t)y * w + x] = (uint16_t)word2;
                if (x + 1 < w) J.word[(size_t)y * w + x + 1] = (uint16_t)(word2 >> 16);
            }
            if ((i & 1) == 0 && x < w) dw[4 * g + i / 2 + 1][lane + 2] = (uint16_t)word2;
            if (feat) {
                const uint32_t ok = (x + 1 < w) ? 0xFFFFFFFFu : (x < w ? 0x0000FFFFu : 0u);
                const uint32_t mm = (mk >> 15) & ok & 0x10001u;
                fsum2 += v2 & ok;
                if (i & 1) {
                    fsum += (fsum2 & 0xFFFFu) + (fsum2 >> 16);
                    fsum2 = 0;
                }
                fmask2 += mm;
                fn2 += ok & 0x10001u;
                uint32_t hit = 0;
                if (need_range) {
                    // per half (value | 0x8000) - need_lo never borrows; flipping bit 15 leaves value - need_lo
                    // modulo 2^16, which is at most need_span exactly when the value is in the range
                    const uint32_t d = ((((v2 | 0x80008000u) - lo2) & (mm * 0xFFFFu)) ^ 0x80008000u);
                    dmin = vmin_u16x2(dmin, d);
                } else {
                    for (int k = 0; k < 2; k++) {
                        const uint16_t code = code_of((uint16_t)(word2 >> (16 * k)), b.band);
                        if (((ok >> (16 * k)) & 1u) && code != kNone && ((needbits[code >> 5] >> (code & 31)) & 1u)) hit = 1;
                    }
                }
                need |= hit != 0;
            }
        }
        m0 = m1;
        m1 = m2;
        if (feat && (i & 3) == 3) {
            // the 4 x 4 block of columns x - 2 l % 4 .. + 3: this lane's pair and its neighbour's
            fsum += (fsum2 & 0xFFFFu) + (fsum2 >> 16);  // a last row past the picture leaves a pair unfolded
            uint32_t fmask = (fmask2 & 0xFFFFu) + (fmask2 >> 16), fn = (fn2 & 0xFFFFu) + (fn2 >> 16);
            fsum += __shfl_xor_sync(0xffffffffu, fsum, 1);
            fmask += __shfl_xor_sync(0xffffffffu, fmask, 1);
            fn += __shfl_xor_sync(0xffffffffu, fn, 1);
            const int fw = (w + 3) / 4, fh = (h + 3) / 4, u = x >> 2, v4 = (y - 3) >> 2;
            if ((lane & 1) == 0 && u < fw && v4 < fh) {
                // (sum / n - 512) / 256 rounded once to float; for a whole block (n = 16) every step is exact in
                // float, so the double path is needed only at the picture's edges
                const float f0 = fn == 16 ? __fmul_rn(__fsub_rn(__fmul_rn((float)fsum, 0.0625f), 512.0f), 0.00390625f)
                                          : fn ? (float)(((double)fsum / (double)fn - 512.0) / 256.0) : 0.0f;
                J.feat[(size_t)v4 * fw + u] = make_float2(f0, __fmul_rn((float)fmask, 0.0625f));
            }
            fsum = fsum2 = fmask2 = fn2 = 0;
        }
    }
    if (feat) {
        if (need_range) need = (dmin & 0xFFFFu) <= (unsigned)b.need_span || (dmin >> 16) <= (unsigned)b.need_span;
        need = __syncthreads_or(need);
        if (tid == 0) J.need[t] = need ? 1u : 0u;
    }
    if (!J.word1) return;  // the same for the whole block
    if (kStrips) strip_out(J.strips + 8 * t + g, x < w, x + 1 < w);

    // the ring of scale-0 words one step outside the tile that scale 1 reads: rows y0-2 and y0+64 (X = 0 .. 33), then
    // columns x0-2 and x0+64 (Y = 1 .. 32)
    if (tid < 2 * kP0D + 2 * (kP0D - 2)) {
        int X, Y;
        if (tid < 2 * kP0D) {
            X = tid % kP0D;
            Y = tid < kP0D ? 0 : kP0D - 1;
        } else {
            Y = 1 + (tid - 2 * kP0D) % (kP0D - 2);
            X = tid - 2 * kP0D < kP0D - 2 ? 0 : kP0D - 1;
        }
        const int px = x0 - 2 + 2 * X, py = y0 - 2 + 2 * Y;
        if (px >= 0 && px < w && py >= 0 && py < h) {
            const int pc = px - xs, m = Y == 0 ? 0 : Y == kP0D - 1 ? kP0M - 1 : 2 * Y - 1;  // mask row of y0 - 2 + 2 Y
            const bool masked = (maskbits[m][pc >> 5] >> (pc & 31)) & 1u;
            auto hm1 = [&](int yy) -> uint16_t {
                const uint16_t *row = buf[yy - ys];
                return (px == 0 || px == w - 1) ? row[pc] : (uint16_t)(mode3x2(row[pc - 1], row[pc], row[pc + 1]) & 0xFFFFu);
            };
            const uint16_t v = (py == 0 || py == h - 1) ? buf[py - ys][pc]
                                                        : (uint16_t)(mode3x2(hm1(py - 1), hm1(py), hm1(py + 1)) & 0xFFFFu);
            dw[Y][X + 1] = (uint16_t)(v | (masked ? kMaskBit : 0));
        }
    }
    __syncthreads();
    // scale 1: the decimated words dw, mode-filtered (rows and columns at the picture's edges keep their value); thread
    // (p, q) makes columns 2 p and 2 p + 1 of rows 2 q and 2 q + 1 of the 32 x 32 tile
    {
        const int w1 = J.w1, h1 = J.h1, p = tid & 15, q = tid >> 4, X1 = (x0 >> 1) + 2 * p, Y0 = (y0 >> 1) + 2 * q;
        if (X1 < w1) {
            const uint32_t edge1 = ((X1 == 0 || X1 == w1 - 1) ? 0x0000FFFFu : 0u) | ((X1 + 1 == w1 - 1) ? 0xFFFF0000u : 0u);
            auto pair1 = [&](int Y, int X) -> uint32_t { return *(const uint32_t *)&dw[Y][X] & 0x7FFF7FFFu; };
            uint32_t hm[4];  // rows Y0 - 1 .. Y0 + 2 (dw rows 2 q .. 2 q + 3; rows outside the picture are not used)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t l2 = pair1(2 * q + k, 2 * p), m2 = pair1(2 * q + k, 2 * p + 2), r2 = pair1(2 * q + k, 2 * p + 4);
                const uint32_t v = mode3x2(__byte_perm(l2, m2, 0x5432), m2, __byte_perm(m2, r2, 0x5432));
                hm[k] = (m2 & edge1) | (v & ~edge1);
            }
            const bool vec1 = (w1 & 1) == 0 && (((uintptr_t)J.word1) & 3) == 0;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int Y1 = Y0 + i;
                if (Y1 >= h1) break;
                const uint32_t word = *(const uint32_t *)&dw[2 * q + i + 1][2 * p + 2];
                const uint32_t v = (Y1 == 0 || Y1 == h1 - 1) ? word & 0x7FFF7FFFu : mode3x2(hm[i], hm[i + 1], hm[i + 2]);
                const uint32_t out = v | (word & 0x80008000u);
                if (kStrips) strip_word(out);
                uint16_t *dst = J.word1 + (size_t)Y1 * w1 + X1;
                if (vec1) {
                    *(uint32_t *)dst = out;
                } else {
                    dst[0] = (uint16_t)out;
                    if (X1 + 1 < w1) dst[1] = (uint16_t)(out >> 16);
                }
            }
        }
        if (kStrips) strip_out(J.strips + 8 * (J.tiles_x * ((h + kP0T - 1) / kP0T) + t) + warp, X1 < w1, X1 + 1 < w1);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Scales 2-4: src/kernels.cu:43-53 (decimate) and 488-500 (mode) on the decimated picture, mask decimated alongside, all
// three in one launch: a block of 256 threads makes a 64 x 32 tile of scale 2 and the 32 x 16 and 16 x 8 tiles of scales
// 3 and 4 beneath it. A scale's 3 x 3 filter reads its decimated neighbours, so the tile grows by 2 words a side per
// scale above; the block makes those margins itself (a word of scale 2 in 1.5 is made twice; the three scales are a
// twelfth of scale 0). Bound by latency: one launch of 10 us for two 4K pictures instead of three of 9.5.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kDTW = 64, kDTH = 32;                        // scale-2 tile
constexpr int kD2W = kDTW + 12, kD2H = kDTH + 12;          // scale 2's decimated words from (x - 6 - 1, y - 6 - 1), 1 more
constexpr int kF2W = kD2W - 2, kF2H = kD2H - 2;            // scale 2 filtered, from (x - 6, y - 6)
constexpr int kF3W = kDTW / 2 + 3, kF3H = kDTH / 2 + 3;    // scale 3 filtered, from (x / 2 - 2, y / 2 - 2)

// The 3 x 3 mode filter of N rows of one column: d points at the column's word in the row above the first, rows `stride`
// apart; (x, y) is the first row's place in a w x h picture. Columns and rows on the picture's edge keep their value in
// their direction, and a word keeps its mask. put(i, word) gets row i's word.
template <int N, typename Put>
__device__ __forceinline__ void mode_column(const uint16_t *d, int stride, int x, int y, int w, int h, Put put)
{
    const bool edge = x == 0 || x == w - 1;
    auto hm = [&](const uint16_t *r) -> uint16_t {
        const uint16_t m = r[0] & 0x7FFF;
        return edge ? m : mode3(r[-1] & 0x7FFF, m, r[1] & 0x7FFF);
    };
    uint16_t m0 = hm(d), m1 = hm(d + stride);
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint16_t c = d[(i + 1) * stride], m2 = hm(d + (i + 2) * stride);
        const bool keep = y + i == 0 || y + i == h - 1;
        put(i, (uint16_t)((keep ? c & 0x7FFF : mode3(m0, m1, m2)) | (c & kMaskBit)));
        m0 = m1;
        m1 = m2;
    }
}

__global__ void __launch_bounds__(256) decimate_mode_kernel(const __grid_constant__ DecBatch b)
{
    wait_for_previous();
    if (b.early) let_next_start();
    __shared__ uint16_t d2[kD2H][kD2W], f2[kF2H][kF2W], d3[kF3H + 2][kF3W + 2], f3[kF3H][kF3W], d4[kDTH / 4 + 2][kDTW / 4 + 2];
    const int j = find_job(b.njobs, (int)blockIdx.x, [&](int k) { return b.job[k].first_block; });
    const DecJob &J = b.job[j];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles_x = (J.w[0] + kDTW - 1) / kDTW, t = blockIdx.x - J.first_block;
    const int x0 = (t % tiles_x) * kDTW, y0 = (t / tiles_x) * kDTH;
    for (int r = warp; r < kD2H; r += 8) {
        const int Y = y0 - 7 + r;
        const uint16_t *row = J.src + (size_t)(2 * Y) * J.sw;
#pragma unroll
        for (int c = lane; c < kD2W; c += 32) {
            const int X = x0 - 7 + c;  // word (2 X, 2 Y) of scale 1
            d2[r][c] = (X >= 0 && X < J.w[0] && Y >= 0 && Y < J.h[0]) ? __ldg(row + 2 * X) : (uint16_t)0;
        }
    }
    __syncthreads();
    // scale 2: a thread per column and 14 rows. Its words at even positions are scale 3's decimated words: (X, Y) is
    // f2[2 (Y - y0 / 2) + 6][2 (X - x0 / 2) + 6]
    static_assert(kF2H == 3 * 14 && kF2W * 3 <= 256, "three threads per column");
    if (tid < kF2W * 3) {
        const int seg = tid / kF2W, c = tid - seg * kF2W, r0 = 14 * seg, X = x0 - 6 + c, Y = y0 - 6 + r0;
        if (X >= 0 && X < J.w[0])
            mode_column<14>(&d2[r0][c + 1], kD2W, X, Y, J.w[0], J.h[0], [&](int i, uint16_t v) {
                f2[r0 + i][c] = v;
                if (X >= x0 && X < x0 + kDTW && Y + i >= y0 && Y + i < y0 + kDTH && Y + i < J.h[0]) J.dst[0][(size_t)(Y + i) * J.w[0] + X] = v;
            });
    }
    __syncthreads();
    static_assert(2 * (kF3W + 1) < kF2W && 2 * (kF3H + 1) < kF2H, "scale 3's margins lie in scale 2's");
    for (int r = warp; r < kF3H + 2; r += 8)
        for (int c = lane; c < kF3W + 2; c += 32) d3[r][c] = f2[2 * r][2 * c];  // from (x / 2 - 3, y / 2 - 3)
    __syncthreads();
    static_assert(kF3H == 19 && kF3W * 7 <= 256, "seven threads per column of scale 3, 3 rows each");
    if (tid < kF3W * 7) {
        const int seg = tid / kF3W, c = tid - seg * kF3W, r0 = min(3 * seg, kF3H - 3), X = x0 / 2 - 2 + c, Y = y0 / 2 - 2 + r0;
        if (X >= 0 && X < J.w[1])
            mode_column<3>(&d3[r0][c + 1], kF3W + 2, X, Y, J.w[1], J.h[1], [&](int i, uint16_t v) {
                const int r = r0 + i;
                f3[r][c] = v;
                if (c >= 2 && c < 2 + kDTW / 2 && r >= 2 && r < 2 + kDTH / 2 && Y + i < J.h[1]) J.dst[1][(size_t)(Y + i) * J.w[1] + X] = v;
            });
    }
    __syncthreads();
    for (int i = tid; i < (kDTH / 4 + 2) * (kDTW / 4 + 2); i += 256) {
        const int r = i / (kDTW / 4 + 2), c = i - r * (kDTW / 4 + 2);
        d4[r][c] = f3[2 * r][2 * c];  // from (x / 4 - 1, y / 4 - 1)
    }
    __syncthreads();
    if (tid < (kDTW / 4) * (kDTH / 4)) {
        const int r = tid / (kDTW / 4), c = tid % (kDTW / 4), X = x0 / 4 + c, Y = y0 / 4 + r;
        if (X < J.w[2] && Y < J.h[2])
            mode_column<1>(&d4[r][c + 1], kDTW / 4 + 2, X, Y, J.w[2], J.h[2], [&](int, uint16_t v) { J.dst[2][(size_t)Y * J.w[2] + X] = v; });
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Pooling: src/cambi.cpp:137-184 with the radix rounds on the device.
// ---------------------------------------------------------------------------------------------------------------
// A positive c-value in units of 2^-24 (exact: c-values are multiples of 2^-24).
__device__ __forceinline__ unsigned long long fx_of(unsigned bits) { return __float2ull_rn(__fmul_rn(__uint_as_float(bits), 16777216.0f)); }

constexpr int kSelThreads = 1024, kSelBlocks = 148;

// The digit of the `remaining`-th largest value from the counts of nb = 2 kSelThreads digits, and the values above that
// digit (called by a whole block; every block of a launch finds the same).
struct Picked {
    unsigned digit;
    unsigned long long above;
};
__device__ Picked pick_digit(const unsigned *hist, unsigned long long remaining, unsigned long long (&warp_tot)[32], Picked &found)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int top = 2 * kSelThreads - 1 - 2 * tid;  // this thread: digits top and top - 1
    const unsigned long long c0 = hist[top], c1 = hist[top - 1];
    unsigned long long incl = c0 + c1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    unsigned long long before = incl - c0 - c1;
    for (int k = 0; k < warp; k++) before += warp_tot[k];
    if (before < remaining && before + c0 + c1 >= remaining) {
        const bool second = before + c0 < remaining;
        found.digit = (unsigned)(second ? top - 1 : top);
        found.above = before + (second ? c0 : 0);
    }
    __syncthreads();
    return found;
}

// A radix round over every slot whose positive count exceeds k: a block picks the digit of the round before (round 1:
// the c-value kernel's counts, 11 bits; round 2: 11 bits), then counts the next one (round 1: 11 bits, round 2: 10) over
// its share of the slot's list. Round 2 also sums the values whose prefix is greater than the selected one (all of them lie
// above the k-th value). What is written of the state (by the block with the list's start) is read by the next launch only.
// One block of kSelThreads per SM: each merges one shared histogram per slot into the slot's, so fewer, larger blocks mean
// fewer global atomics for the same reads. The lists are shared out as if they were one after the other, so that a block
// has one or two slots: picking a digit and merging take 4 us of latency a slot, whatever its list's length. When every
// block took a share of every slot, one slot after the other, and counted runs of equal digits (which costs more
// instructions than one atomic per matching value) a round took 29 us for a dense 3840 x 2160 picture and for four of them
// with fewer values; now 19 us.
template <int kRound>
__global__ void __launch_bounds__(kSelThreads) select_kernel(CvSlot *slots, int nslots, bool early)
{
    constexpr bool last = kRound == 2;
    constexpr int shift = last ? 0 : 10, nb = last ? 1024 : 2048;
    __shared__ unsigned hist[nb];
    __shared__ unsigned long long warp_tot[32];
    __shared__ Picked found;
    __shared__ int todo[kMaxJobs];
    __shared__ unsigned long long groups[kMaxJobs];  // of 4 values, in the slot's list
    __shared__ int warp_n[kSelThreads / 32];
    static_assert(kMaxJobs <= kSelThreads, "a thread per slot");
    wait_for_previous();
    if (early) let_next_start();
    const int tid = threadIdx.x;
    const bool mine = tid < nslots && slots[tid].count > slots[tid].k;
    if (!__syncthreads_or(mine)) return;
    const unsigned set = __ballot_sync(0xffffffffu, mine);
    if ((tid & 31) == 0) warp_n[tid >> 5] = __popc(set);
    __syncthreads();
    int ntodo = 0, rank = __popc(set & ((1u << (tid & 31)) - 1u));
    for (int k = 0; k < kSelThreads / 32; k++) {
        if (k < tid >> 5) rank += warp_n[k];
        ntodo += warp_n[k];
    }
    if (mine) {
        todo[rank] = tid;
        groups[rank] = (slots[tid].list_n + 3) / 4;
    }
    __syncthreads();
    unsigned long long total = 0;
    for (int it = 0; it < ntodo; it++) total += groups[it];
    const unsigned long long share = (total + gridDim.x - 1) / gridDim.x, g0 = blockIdx.x * share, g1 = min(g0 + share, total);
    unsigned long long start = 0;  // of the slot's list among all
    for (int it = 0; it < ntodo && start < g1; start += groups[it], it++) {
        if (start + groups[it] <= g0) continue;
        CvSlot &S = slots[todo[it]];
        const unsigned long long remaining = last ? S.remaining1 : S.k;
        const Picked p = pick_digit(last ? S.hist1 : S.hist, remaining, warp_tot, found);
        const unsigned prefix = last ? S.prefix1 | (p.digit << 10) : p.digit << 21, mask = last ? 0xFFFFFC00u : 0xFFE00000u;
        if (start >= g0 && tid == 0) {
            if (last) {
                S.prefix2 = prefix;
                S.remaining2 = remaining - p.above;
            } else {
                S.prefix1 = prefix;
                S.remaining1 = remaining - p.above;
            }
        }
        for (int i = tid; i < nb; i += kSelThreads) hist[i] = 0;
        __syncthreads();
        const unsigned *v = (const unsigned *)S.list;
        // the block's groups of this list: from .. to - 1, whole ones up to n4
        const unsigned long long n = S.list_n, n4 = n / 4, from = max(g0, start) - start, to = min(g1 - start, groups[it]);
        // the sum is exact: a thread's share of a list is far below the 2^14 values (each below 2^15, in 2^-24) that could
        // leave 53 bits
        double above = 0.0;
        unsigned above_n = 0;
        auto add = [&](unsigned bits) {
            const unsigned top = bits & mask;
            if (top == prefix) atomicAdd(&hist[(bits >> shift) & (unsigned)(nb - 1)], 1u);
            if (last && top > prefix) {
                above += (double)__uint_as_float(bits);
                above_n++;
            }
        };
        // four 16-byte loads in flight per thread, then the rest one by one
        const unsigned long long whole = min(to, n4);
        unsigned long long i = from + tid;
        for (; i + 3 * kSelThreads < whole; i += 4 * kSelThreads) {
            uint4 q[4];
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = __ldg((const uint4 *)v + i + u * kSelThreads);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                add(q[u].x);
                add(q[u].y);
                add(q[u].z);
                add(q[u].w);
            }
        }
        for (; i < whole; i += kSelThreads) {
            const uint4 q = __ldg((const uint4 *)v + i);
            add(q.x);
            add(q.y);
            add(q.z);
            add(q.w);
        }
        if (to > n4 && tid < (int)(n & 3)) add(v[4 * n4 + tid]);
        if (last) {
            unsigned long long above_fx = __double2ull_rn(above * 16777216.0);
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                above_fx += __shfl_down_sync(0xffffffffu, above_fx, o);
                above_n += __shfl_down_sync(0xffffffffu, above_n, o);
            }
            if ((tid & 31) == 0 && above_n) {
                atomicAdd(&S.above_fx, above_fx);
                atomicAdd(&S.above_n, (unsigned long long)above_n);
            }
        }
        __syncthreads();
        for (int i = tid; i < nb; i += kSelThreads)
            if (hist[i]) atomicAdd(last ? &S.hist2[i] : &S.hist1[i], hist[i]);
        __syncthreads();
    }
}

// A block per picture, a warp per scale: the last digit of a slot with more than k positive values, from round 2's counts,
// and the sum above it (the counters of both rounds are left clear); then the scales' pooled values and the score, to
// device memory and, where the job has a place, to the host's.
__global__ void __launch_bounds__(32 * kScales) score_kernel(const __grid_constant__ ScoreBatch b)
{
    __shared__ double part[kScales];
    wait_for_previous();
    const ScoreJob &J = b.job[blockIdx.x];
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    CvSlot &S = b.slots[J.first_slot + s];
    const unsigned long long count = S.count, k = S.k;
    double pooled;
    if (count <= k) {
        pooled = __ddiv_rn(__dmul_rn(__ull2double_rn(S.sum_fx), 1.0 / 16777216.0), __ull2double_rn(k));
    } else {
        const unsigned long long remaining = S.remaining2;
        // lane l: digits 1023 - 32 l down to 992 - 32 l
        const int top = 1023 - 32 * lane;
        unsigned long long mine = 0, fx = 0;
#pragma unroll 8
        for (int d = 0; d < 32; d++) {
            const unsigned c = S.hist2[top - d];  // values equal to the digit's
            mine += c;
            fx += c * fx_of(S.prefix2 | (unsigned)(top - d));
        }
        unsigned long long cincl = mine, fincl = fx;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long c = __shfl_up_sync(0xffffffffu, cincl, o), f = __shfl_up_sync(0xffffffffu, fincl, o);
            if (lane >= o) {
                cincl += c;
                fincl += f;
            }
        }
        unsigned long long above_n = cincl - mine, above_fx = fincl - fx;
        const bool here = above_n < remaining && cincl >= remaining;
        int digit = top;
        if (here) {
            for (int d = 0; d < 31; d++, digit--) {
                const unsigned c = S.hist2[digit];
                if (above_n + c >= remaining) break;
                above_n += c;
                above_fx += c * fx_of(S.prefix2 | (unsigned)digit);
            }
        }
        const unsigned who = __ballot_sync(0xffffffffu, here);
        const int src = __ffs(who) - 1;
        digit = __shfl_sync(0xffffffffu, digit, src);
        above_n = __shfl_sync(0xffffffffu, above_n, src) + S.above_n;
        above_fx = __shfl_sync(0xffffffffu, above_fx, src) + S.above_fx;
        const unsigned kth = S.prefix2 | (unsigned)digit;
        const double above = __dmul_rn(__ull2double_rn(above_fx), 1.0 / 16777216.0);
        const double rest = __dmul_rn(__ull2double_rn(k - above_n), (double)__uint_as_float(kth));
        pooled = __ddiv_rn(__dadd_rn(above, rest), __ull2double_rn(k));
        __syncwarp();
        for (int i = lane; i < 2048 / 4; i += 32) ((uint4 *)S.hist1)[i] = make_uint4(0, 0, 0, 0);
        for (int i = lane; i < 1024 / 4; i += 32) ((uint4 *)S.hist2)[i] = make_uint4(0, 0, 0, 0);
    }
    if (lane == 0) {
        part[s] = pooled;
        J.score[1 + s] = pooled;
        if (J.host) J.host[1 + s] = pooled;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double total = 0.0;
    const double kScaleWeight[kScales] = {16.0, 8.0, 4.0, 2.0, 1.0};
    for (int q = 0; q < kScales; q++) total = __dadd_rn(total, __dmul_rn(part[q], kScaleWeight[q]));
    const int odd = 2 * (J.window >> 1) + 1;
    const double score = __ddiv_rn(total, (double)(odd * odd));
    J.score[0] = score < 1000.0 ? score : 1000.0;
    if (J.host) J.host[0] = J.score[0];
}

}  // namespace

cudaError_t launch_prep0(Prep0Batch &b, cudaStream_t s)
{
    int tiles = 0;
    for (int j = 0; j < b.njobs; j++) {
        Prep0Job &J = b.job[j];
        J.tiles_x = (J.w + kP0T - 1) / kP0T;
        J.first_tile = tiles;
        tiles += J.tiles_x * ((J.h + kP0T - 1) / kP0T);
    }
    b.total_tiles = tiles;
    if (b.total_tiles <= 0) return cudaSuccess;
    // the values whose codes need c-values, as one range when they are one (they are for CAMBI's thresholds)
    int lo = -1, hi = -2;
    bool one_range = true;
    for (int code = 0; code < b.band.band_size; code++) {
        if (!cvalue_dists(code, b.band)) continue;
        if (lo < 0) lo = code;
        else if (code != hi + 1) one_range = false;
        hi = code;
    }
    b.need_lo = lo < 0 ? 0 : lo + b.band.band_base;
    b.need_span = !one_range ? -1 : lo < 0 ? -1 : hi - lo;
    LaunchTimer t("cambi_prep0", s);
    bool strips = true;
    for (int j = 0; j < b.njobs; j++) strips = strips && b.job[j].strips && b.job[j].word1;
    return launch_kernel(b.chained, strips ? prep0_kernel<true> : prep0_kernel<false>, dim3(b.total_tiles + b.nslots), 256, 0, s, b);
}

cudaError_t launch_decimate_mode(DecBatch &b, cudaStream_t s)
{
    int blocks = 0;
    for (int j = 0; j < b.njobs; j++) {
        b.job[j].first_block = blocks;
        blocks += ((b.job[j].w[0] + kDTW - 1) / kDTW) * ((b.job[j].h[0] + kDTH - 1) / kDTH);
    }
    if (blocks <= 0) return cudaSuccess;
    LaunchTimer t("cambi_decimate_mode", s);
    return launch_kernel(b.chained, decimate_mode_kernel, dim3(blocks), 256, 0, s, b);
}

cudaError_t launch_topk(CvSlot *slots, int nslots, cudaStream_t s, bool early)
{
    if (nslots <= 0) return cudaSuccess;
    {
        LaunchTimer t("cambi_select", s);
        const cudaError_t e = launch_kernel(true, select_kernel<1>, dim3(kSelBlocks), kSelThreads, 0, s, slots, nslots, early);
        if (e != cudaSuccess) return e;
    }
    LaunchTimer t("cambi_select", s);
    return launch_kernel(true, select_kernel<2>, dim3(kSelBlocks), kSelThreads, 0, s, slots, nslots, early);
}

cudaError_t launch_score(const ScoreBatch &b, cudaStream_t s)
{
    if (b.njobs <= 0) return cudaSuccess;
    LaunchTimer t("cambi_score", s);
    return launch_kernel(true, score_kernel, dim3(b.njobs), 32 * kScales, 0, s, b);
}

const void *kernel_entry_prep0() { return (const void *)prep0_kernel<false>; }
const void *kernel_entry_decimate_mode() { return (const void *)decimate_mode_kernel; }

}  // namespace es
