// CAMBI c-values for sm_100a: src/kernels.cu:113-278 (cambi.c's c_value_pixel over the (2 pad + 1)^2 window of every
// masked pixel in the band, histogram windows clipped at the picture's edges), bit-exact, with a different algorithm.
//
// One 256-thread block per tile of 64 columns by 64, 32 or 16 rows of any scale of any picture (a table of jobs):
//  1. the tile's own pixels give the range of band codes (value - band_base of a masked pixel in the band) whose
//     c-value is needed; tiles without one -- most tiles of most pictures -- leave after reading them. (A launch of many
//     tiles has a kernel list the others first, and blocks that stay take tiles from the list);
//  2. the tile and its window margins are staged as one byte per pixel (the code relative to that range), and every
//     code seen sets a byte flag; the codes that can matter -- occurring within kDiffs of a code whose c-value is not
//     trivially 0 -- are ranked in order. The plane holds ranks: as it is when the codes are consecutive, else through
//     a 256-byte table. A range over kSegSpan codes is taken in segments, each staged anew;
//  3. per pass over 32 ranks, each warp takes 8 neighbouring rows of the tile by itself: its column counts (8 bits per
//     column and rank: pixels of the 2 pad + 1 window rows) are a 32 x region-width byte matrix in shared memory that
//     slides down the warp's rows; a row's window counts are an exact integer matrix product on the tensor cores
//     (mma.sync u8, counts x a band of ones 2 pad + 1 wide), 32 columns at a time into a small buffer of the warp's
//     own, from which each lane makes one pixel's c-value. Nothing in the row loop waits for another warp.
//     The 8 warps' first column counts come from one sum over the rows of the first window and one over each warp's
//     own changes, both made by all warps in parallel and added up in a prefix over the warps.
// Positive c-values are summed exactly (they are multiples of 2^-24) and counted, and the rows that have served pixels
// are written to the scale's list (for the top-k selection), zeros where a pixel has no positive c-value; nothing else per pixel
// is written unless the caller asks for the c-value planes.
//
// What bounds it: instruction issue and, on pictures with few busy tiles, one block's latency. The block-wide form this
// replaces (two block barriers per row, every warp stepping through every row) issued 130 thousand warp instructions per
// busy 4K tile, this one 60 thousand; three blocks per SM (80 registers) against two (128): 245 against 270 us on the
// dense 4K picture. C-values of one picture, before / now: 3840x2160 10-bit dense 520 / 225 us, the same size bright with
// steps of 8 codes 557 / 105 us, 1920x1080 8-bit 176 / 55 us, 640x360 8-bit 90 / 24 us. (Of the 225, 23 fewer since the
// counts move by atomics without a result and the four differences are computed without branches.)
#include "cambi_codes.h"
#include "es_kernels.h"

namespace es {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = kCvThreads / 32;
constexpr int kSegSpan = 240;      // own codes of one staging: with kDiffs on both sides below the byte plane's 255
constexpr unsigned kNoRank = 0xFFu;
constexpr int kWStride = 64;       // window-count row: 32 u16 columns
constexpr int kWRows = kCvBins + 1;  // row 0 stays zero (absent neighbours), rank k is row k + 1
constexpr int kWBytes = kWRows * kWStride;
// A window-count row's byte offset with its swizzle: the row's four 16-byte chunks are permuted by bits 1 and 2 of the
// row, so the 8 rows of a store phase fall on different banks; column x is at (cv_row(row) ^ 2 x).
__host__ __device__ constexpr int cv_row(int row) { return row * kWStride | ((row << 3) & 0x30); }
constexpr uint32_t kBias = 0x08080808u;  // per byte: a warp's rows take at most 8 pixels out of a column

// k-steps of 32 region columns that 32 output columns with a pad reach (the staged region starts at the multiple of 8
// at or left of x0 - pad, ox columns further left), and what follows from it: staged columns, the column counts' row
// (16 bytes more, so the 8 rows an ldmatrix phase reads fall on different banks).
__host__ __device__ constexpr int cv_ox(int pad) { return (8 - pad % 8) % 8; }
__host__ __device__ constexpr int cv_ksteps(int pad) { return (31 + cv_ox(pad) + 2 * pad) / 32 + 1 < 2 ? 2 : (31 + cv_ox(pad) + 2 * pad) / 32 + 1; }
__host__ __device__ constexpr int cv_cols(int n) { return 32 * (n + 1); }
__host__ __device__ constexpr int cv_cstr(int n) { return cv_cols(n) + 16; }

// Shared memory. The window counts come first: their addresses fit 16 bits, two to a word in the neighbour table.
struct CvLayout {
    int counts, colc, plane, seen, served, nbr, tab, band, total;
};
__host__ __device__ inline CvLayout cv_layout(int pad)
{
    const int n = cv_ksteps(pad);
    CvLayout l;
    l.counts = 0;
    l.colc = l.counts + kWarps * kWBytes;
    l.plane = l.colc + kWarps * kCvBins * cv_cstr(n);
    l.seen = l.plane + (kCvTY + 2 * pad) * cv_cols(n);
    l.served = l.seen + 512;
    l.nbr = l.served + 256;
    l.tab = l.nbr + 1024;
    l.band = l.tab + kCvBins * 16;
    l.total = l.band + (4 * n + 2) * 128;
    return l;
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3)
{
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
                 : "memory");
}
__device__ __forceinline__ unsigned lds_u16(uint32_t addr)
{
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(addr) : "memory");
    return v;
}

// d = (kAdd: d +) a (16 x 32 u8, row-major) x b (32 x 8 u8, column-major), exact in 32-bit integers.
template <bool kAdd>
__device__ __forceinline__ void mma_u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    if (kAdd)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// per 16-bit half, modulo 2^16 and unsigned
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("add.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// The words of row y, pixels x .. x + 7 (x a multiple of 8), 0 (unmasked) outside the picture: one 16-byte load, or 4-
// or 2-byte loads where the rows are not 16-byte aligned (align: 0, 1, 2).
__device__ __forceinline__ uint4 load8(const CvJob &J, int align, int y, int x)
{
    if (y < 0 || y >= J.h || x < 0 || x >= J.w) return make_uint4(0, 0, 0, 0);
    const uint16_t *p = J.word + (size_t)y * J.w + x;
    if (align == 0) return __ldg((const uint4 *)p);
    if (align == 1 && x + 8 <= J.w) {
        const uint32_t *q = (const uint32_t *)p;
        return make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
    }
    uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (x + k < J.w) v[k >> 1] |= (uint32_t)__ldg(p + k) << (16 * (k & 1));
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Bits c - 4 .. c + 4 (c = 32 word + lane) of a 256-bit set.
__device__ __forceinline__ unsigned around(const uint32_t *set, int word, int lane)
{
    const uint32_t mid = set[word], lo = word > 0 ? set[word - 1] : 0u, hi = word < 7 ? set[word + 1] : 0u;
    const uint32_t v = lane >= kDiffs ? __funnelshift_r(mid, hi, lane - kDiffs) : __funnelshift_l(lo, mid, kDiffs - lane);
    return v & 0x1FFu;
}

struct CvShared {
    uint32_t occ[8], srv[8], rel[8], needbits[32];
    unsigned redlo[kWarps], redhi[kWarps], rowcnt[kWarps];
    unsigned long long red_sum[kWarps];
    unsigned red_cnt[kWarps];
    unsigned hist1[kCvDigits];  // the tile's positive c-values by their first radix digit
    unsigned long long list_base;
    unsigned next_tile;
};

// How a job's rows may be read: load8's align.
__device__ __forceinline__ int row_align(const CvJob &J)
{
    return (J.w & 7) == 0 && (((uintptr_t)J.word) & 15) == 0 ? 0 : (J.w & 1) == 0 && (((uintptr_t)J.word) & 3) == 0 ? 1 : 2;
}

constexpr unsigned kNoRange = 0xFFFFFFFFu;  // a tile whose code range is not known

// One tile, gt its global number; all threads return together. N: k-steps of the job's pad. known: a range of band codes
// that holds the tile's needed ones, or kNoRange.
template <int N>
__device__ __forceinline__ void tile_cvalues(const CvBatch &b, const CvJob &J, const int gt, const unsigned known, unsigned char *smem, CvShared &sh)
{
    constexpr int kCols = cv_cols(N), kCstr = cv_cstr(N), kWords = kCols / 4, kVecs = kCols / 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Band &bd = b.band;
    const int tile = gt - J.first_tile;
    const int th = J.tile_rows ? J.tile_rows : kCvTY;
    const int x0 = (tile % J.tiles_x) * kCvTX, y0 = (tile / J.tiles_x) * th;
    const int w = J.w, h = J.h, P = J.pad;
    const int rows = min(th, h - y0), cols = min(kCvTX, w - x0);
    const int align = row_align(J);
    const CvLayout L = cv_layout(P);
    uint8_t *plane = smem + L.plane;           // [RH][kCols]: code or rank of pixel (xs + j, y0 - P + r)
    uint8_t *seen = smem + L.seen;             // byte flags: [0, 256) codes in the margins, [256, 512) in the tile itself
    uint8_t *served = smem + L.served;         // by plane byte: its c-values are wanted and not trivially 0
    uint32_t *nbr = (uint32_t *)(smem + L.nbr);  // by rank: rank offsets of the neighbours its c-value reads

    // 1. the range of needed codes among the tile's pixels
    unsigned mlo = 0xFFFFu, mhi = 0xFFFFu;
    const bool range = b.need_span >= 0;
    if (known == kNoRange) {
        const uint32_t clo = (uint32_t)((0x10000 - 0x8000 - b.need_lo) & 0xFFFF) * 0x10001u;
        const uint32_t chi = (uint32_t)((0x8000 + b.need_lo + b.need_span + 1) & 0xFFFF) * 0x10001u;
        uint32_t lo2 = 0xFFFFFFFFu, hi2 = 0xFFFFFFFFu;
        for (int i = tid; i < rows * (kCvTX / 8); i += kCvThreads) {
            const uint4 q = load8(J, align, y0 + (i >> 3), x0 + 8 * (i & 7));
            const uint32_t v[4] = {q.x, q.y, q.z, q.w};
            if (range) {
                // per half: masked value - need_lo and need_hi - masked value; above the span for every other word
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    lo2 = min2(lo2, add2(v[k], clo));
                    hi2 = min2(hi2, add2(~v[k], chi));
                }
            } else {
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint16_t code = code_of((v[k >> 1] >> (16 * (k & 1))) & 0xFFFFu, bd);
                    if (code != kNone && ((sh.needbits[code >> 5] >> (code & 31)) & 1u)) {
                        mlo = min(mlo, (unsigned)code);
                        mhi = min(mhi, 0xFFFEu - code);
                    }
                }
            }
        }
        if (range) {
            mlo = min(lo2 & 0xFFFFu, lo2 >> 16);
            mhi = min(hi2 & 0xFFFFu, hi2 >> 16);
        }
    }
    mlo = __reduce_min_sync(kFull, mlo);
    mhi = __reduce_min_sync(kFull, mhi);
    if (lane == 0) {
        sh.redlo[warp] = mlo;
        sh.redhi[warp] = mhi;
    }
    if (tid < 32) ((uint4 *)seen)[tid] = make_uint4(0, 0, 0, 0);
    if (tid < kCvDigits) sh.hist1[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kWarps; k++) {
        mlo = min(mlo, sh.redlo[k]);
        mhi = min(mhi, sh.redhi[k]);
    }
    if (known == kNoRange && (mlo == 0xFFFFu || (range && mlo > (unsigned)b.need_span))) {
        if (b.tile_mass && tid == 0) b.tile_mass[gt] = 0;
        return;
    }
    const int own_lo = known != kNoRange ? (int)(known & 0xFFFFu) : range ? b.need_lo + (int)mlo - bd.band_base : (int)mlo;
    const int own_hi = known != kNoRange ? (int)(known >> 16) : range ? b.need_lo + b.need_span - (int)mhi - bd.band_base : 0xFFFE - (int)mhi;

    const int RH = rows + 2 * P, xs = x0 - P - cv_ox(P), px = P + cv_ox(P);  // plane column of tile column 0
    const int rpw = th / kWarps;  // rows of a warp: 8, 4 or 2
    uint8_t *cw = smem + L.colc + warp * (kCvBins * kCstr);  // this warp's column counts [rank][kCstr]
    unsigned char *ww = smem + L.counts + warp * kWBytes;    // this warp's window counts [1 + rank][32]
    // the products' B operands, by lane: band[m] holds the band of ones at region columns 8 (m - 3) + 4 t + i from output
    // column g (+ ox), t = lane % 4, g = lane / 4
    uint32_t *band = (uint32_t *)(smem + L.band);
    for (int i = tid; i < (4 * N + 2) * 32; i += kCvThreads) {
        const int d0 = 8 * ((i >> 5) - 3) + 4 * (i & 3) - ((i & 31) >> 2) - cv_ox(P);
        uint32_t word = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) word |= (uint32_t)((unsigned)(d0 + k) <= 2u * P) << (8 * k);
        band[i] = word;
    }

    CvSlot &SL = b.slots[J.slot];
    double my_sum = 0.0;  // exact: at most 16 pixels per lane and pass, multiples of 2^-24 below 2^15
    unsigned my_cnt = 0;
    unsigned run[2] = {0, 0};  // per half row: the run of equal first digits down the column, digit << 16 | length

    // a first digit's run of equal ones, into the tile's counts (larger digits exist only for weights beyond CAMBI's)
    auto count_run = [&](int half) {
        const unsigned n = run[half] & 0xFFFFu, dg = run[half] >> 16;
        if (!n) return;
        if (dg < kCvDigits) atomicAdd(&sh.hist1[dg], n);
        else atomicAdd(&SL.hist[(dg + kCvDigit0) & 2047u], n);
    };

    // a tile of several segments takes list places for all its rows at once (its segments share rows), zeros first
    const bool segments = own_hi - own_lo >= kSegSpan;
    if (segments) {
        if (tid == 0) sh.list_base = atomicAdd(&SL.list_n, (unsigned long long)rows * cols);
        __syncthreads();
        for (int i = tid; i < rows * cols; i += kCvThreads) SL.list[sh.list_base + i] = 0.0f;
    }
    for (int seg_lo = own_lo; seg_lo <= own_hi; seg_lo += kSegSpan) {
        const int seg_hi = min(own_hi, seg_lo + kSegSpan - 1);
        const int base = max(seg_lo - kDiffs, 0), len = min(seg_hi + kDiffs, bd.band_size - 1) - base + 1;  // len <= 248
        if (seg_lo != own_lo) {
            __syncthreads();
            if (tid < 32) ((uint4 *)seen)[tid] = make_uint4(0, 0, 0, 0);
            __syncthreads();
        }
        // 2. the region as bytes: code - base, or len for every other pixel
        {
            constexpr int kPer = 32 / kVecs > 0 ? 32 / kVecs : 1;  // region rows a warp stages at once
            const int lr = lane / kVecs, lv = lane % kVecs;
            const uint32_t cbase = (uint32_t)((0x10000 - 0x8000 - bd.band_base - base) & 0xFFFF) * 0x10001u, len2 = (uint32_t)len * 0x10001u;
            const int xv = xs + 8 * lv;
            const bool mid = xv >= x0 && xv < x0 + kCvTX;
            if (lr < kPer) {
#pragma unroll 2
                for (int r = warp * kPer + lr; r < RH; r += kWarps * kPer) {
                    const uint4 q = load8(J, align, y0 - P + r, xv);
                    const uint32_t z0 = min2(add2(q.x, cbase), len2), z1 = min2(add2(q.y, cbase), len2);
                    const uint32_t z2 = min2(add2(q.z, cbase), len2), z3 = min2(add2(q.w, cbase), len2);
                    const uint32_t lo = __byte_perm(z0, z1, 0x6420), hi = __byte_perm(z2, z3, 0x6420);
                    *(uint2 *)(plane + r * kCols + 8 * lv) = make_uint2(lo, hi);
                    uint8_t *flag = seen + (mid && r >= P && r < P + rows ? 256 : 0);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        flag[(lo >> (8 * e)) & 0xFFu] = 1;  // racing writers store the same 1
                        flag[(hi >> (8 * e)) & 0xFFu] = 1;
                    }
                }
            }
        }
        __syncthreads();
        // thread c: code base + c
        const int c = tid, code = base + c;
        const unsigned dists = c < len ? cvalue_dists(code, bd) : 0u;
        const bool in_tile = c < len && seen[256 + c] != 0, in_region = c < len && (in_tile || seen[c] != 0);
        const bool own = in_tile && dists && code >= seg_lo && code <= seg_hi;
        const unsigned occ_w = __ballot_sync(kFull, in_region);
        if (lane == 0) sh.occ[warp] = occ_w;
        __syncthreads();
        // the neighbours its c-value reads: occurring, at a distance d + 1 its thresholds switch on (an absent one gives
        // the same c-value as one with no pixels); a code without any has c-value 0 everywhere and is not served
        unsigned allowed = 0;
#pragma unroll
        for (int d = 0; d < kDiffs; d++)
            if ((dists >> d) & 1u) allowed |= (1u << (kDiffs + 1 + d)) | (1u << (kDiffs - 1 - d));
        const unsigned nb = around(sh.occ, warp, lane) & allowed;
        const bool serve = own && nb != 0;
        const unsigned srv_w = __ballot_sync(kFull, serve);
        if (lane == 0) sh.srv[warp] = srv_w;
        if (!__syncthreads_or(serve)) continue;
        const bool relevant = in_region && around(sh.srv, warp, lane) != 0;
        const unsigned rel_w = __ballot_sync(kFull, relevant);
        if (lane == 0) sh.rel[warp] = rel_w;
        __syncthreads();
        int R = 0, rank = 0, first = -1, last = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t word = sh.rel[k];
            if (k == warp) rank = R + __popc(word & ((1u << lane) - 1u));
            if (word) {
                if (first < 0) first = 32 * k + __ffs(word) - 1;
                last = 32 * k + 31 - __clz(word);
            }
            R += __popc(word);
        }
        const bool identity = last - first + 1 == R;  // consecutive codes: a code's byte is first + its rank
        seen[c] = relevant ? (uint8_t)rank : (uint8_t)kNoRank;  // the flags are read: [0, 256) becomes the rank table
        if (identity) {
            served[c] = serve;
        } else {
            if (relevant) served[rank] = serve;
            if (c >= R) served[c] = 0;
        }
        if (relevant) {
            const unsigned rm = around(sh.rel, warp, lane);
            uint32_t packed = 0;  // nibble d: the neighbour d + 1 above, 4 + d: below; rank offset + 4, or 15
#pragma unroll
            for (int d = 0; d < kDiffs; d++) {
                const unsigned below = (2u << d) - 1u;
                const unsigned up = (nb >> (kDiffs + 1 + d)) & 1u ? kDiffs + __popc((rm >> (kDiffs + 1)) & below) : 15u;
                const unsigned dn = (nb >> (kDiffs - 1 - d)) & 1u ? kDiffs - __popc((rm >> (kDiffs - 1 - d)) & below) : 15u;
                packed |= (up << (4 * d)) | (dn << (4 * (kDiffs + d)));
            }
            nbr[rank] = serve ? packed : 0xFFFFFFFFu;
        }
        __syncthreads();
        if (!identity) {
            for (int i = tid; i < RH * (kCols / 16); i += kCvThreads) {
                uint4 q = ((const uint4 *)plane)[i];
                auto ranks4 = [&](uint32_t v) -> uint32_t {
                    return (uint32_t)seen[v & 0xFFu] | ((uint32_t)seen[(v >> 8) & 0xFFu] << 8) | ((uint32_t)seen[(v >> 16) & 0xFFu] << 16) |
                           ((uint32_t)seen[v >> 24] << 24);
                };
                q.x = ranks4(q.x);
                q.y = ranks4(q.y);
                q.z = ranks4(q.z);
                q.w = ranks4(q.w);
                ((uint4 *)plane)[i] = q;
            }
            __syncthreads();
        }
        // the rows of this warp that have served pixels: they get places in the scale's list
        unsigned rowbits = 0;
        for (int i = 0; i < rpw; i++) {
            const int r = warp * rpw + i;
            if (r >= rows) break;
            const uint8_t *p = plane + (r + P) * kCols + px + lane;
            const bool any = (lane < cols && served[p[0]]) || (lane + 32 < cols && served[p[32]]);
            if (__any_sync(kFull, any)) rowbits |= 1u << i;
        }
        unsigned list_row = warp * rpw;  // of the warp's first row in the tile's places
        if (!segments) {
            if (lane == 0) sh.rowcnt[warp] = __popc(rowbits);
            __syncthreads();
            unsigned list_rows = 0;
            list_row = 0;
#pragma unroll
            for (int k = 0; k < kWarps; k++) {
                if (k < warp) list_row += sh.rowcnt[k];
                list_rows += sh.rowcnt[k];
            }
            if (tid == 0) sh.list_base = atomicAdd(&SL.list_n, (unsigned long long)list_rows * cols);  // read after the barriers below
        }

        // 3. passes over 32 ranks; a pass serves ranks lo .. hi - 1 (all of them read ranks of the pass only)
        for (int b0 = 0;;) {
            const int lo = b0 ? b0 + kDiffs : 0, hi = b0 + kCvBins >= R ? R : b0 + kCvBins - kDiffs;
            const int off = (identity ? first : 0) + b0;  // plane byte of pass rank 0
            const int npos = min(kCvBins, R - b0), nrows = npos <= 16 ? 16 : 32;  // ranks in the pass; count rows used
            const int nvec = nrows * kCstr / 16;
            // per pass rank, 8 halves: the window-count row of each neighbour as a byte offset (0: the zero row)
            {
                const int kk = tid >> 3, i = tid & 7;
                const unsigned nib = b0 + kk < R ? (nbr[b0 + kk] >> (4 * i)) & 15u : 15u;
                const int row = kk + (int)nib - kDiffs;
                ((uint16_t *)(smem + L.tab))[tid] = (nib == 15u || row < 0 || row >= kCvBins) ? 0 : (uint16_t)cv_row(row + 1);
            }
            // a count on or off, as an addition to the word of its four columns (a lane's own): no byte ends below 0 or
            // above 255, so the carries between the bytes cancel. An atomic without a result is one instruction that
            // nothing waits for, where the byte's load, addition and store made a chain of eight per word.
            const uint32_t cw_at = (uint32_t)__cvta_generic_to_shared(cw);
            auto count_rank = [&](uint32_t word, int wi, int e, int delta) {
                const unsigned k = ((word >> (8 * e)) & 0xFFu) - off;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %0, %1;\n\t@p red.shared.add.u32 [%2], %3;\n\t}\n" ::"r"(k), "r"(npos),
                             "r"(cw_at + k * kCstr + 4 * wi), "r"((unsigned)delta << (8 * e))
                             : "memory");
            };
            // moves counts on from tile row r to r + 1: region row r leaves, r + 2 P + 1 enters
            auto slide = [&](int r) {
                const int enter = r + 2 * P + 1;
#pragma unroll
                for (int s = 0; s < (kWords + 31) / 32; s++) {
                    const int wi = lane + 32 * s;
                    if (kWords % 32 && wi >= kWords) break;
                    const uint32_t wl = *(const uint32_t *)(plane + r * kCols + 4 * wi);
                    const uint32_t we = enter < RH ? *(const uint32_t *)(plane + enter * kCols + 4 * wi) : 0xFFFFFFFFu;
                    if (wl == we) continue;
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        count_rank(wl, wi, e, -1);
                        count_rank(we, wi, e, 1);
                    }
                }
            };
            for (int i = lane; i < nvec; i += 32) ((uint4 *)cw)[i] = make_uint4(0, 0, 0, 0);
            for (int i = lane; i < kWBytes / 16; i += 32) ((uint4 *)ww)[i] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            // the first window's rows, shared out over the warps
            for (int r = warp; r <= min(2 * P, RH - 1); r += kWarps) {
#pragma unroll
                for (int s = 0; s < (kWords + 31) / 32; s++) {
                    const int wi = lane + 32 * s;
                    if (kWords % 32 && wi >= kWords) break;
                    const uint32_t word = *(const uint32_t *)(plane + r * kCols + 4 * wi);
#pragma unroll
                    for (int e = 0; e < 4; e++) count_rank(word, wi, e, 1);
                }
            }
            __syncthreads();
            auto add4 = [](uint4 &a, const uint4 &v) {  // bytes of counts: no carry leaves a byte
                a.x += v.x;
                a.y += v.y;
                a.z += v.z;
                a.w += v.w;
            };
            uint4 sum[2];
#pragma unroll
            for (int s = 0; s < 2; s++) {
                sum[s] = make_uint4(0, 0, 0, 0);
                const int i = tid + kCvThreads * s;
                if (i < nvec)
#pragma unroll
                    for (int k = 0; k < kWarps; k++) add4(sum[s], ((const uint4 *)(smem + L.colc + k * (kCvBins * kCstr)))[i]);
            }
            __syncthreads();
            // each warp's own changes (plus the bias, so that no byte goes below 0), then the prefix over the warps
            for (int i = lane; i < nvec; i += 32) ((uint4 *)cw)[i] = make_uint4(kBias, kBias, kBias, kBias);
            __syncwarp();
            if (warp < kWarps - 1)
                for (int i = 0; i < rpw && warp * rpw + i < rows; i++) slide(warp * rpw + i);
            __syncthreads();
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const int i = tid + kCvThreads * s;
                if (i < nvec) {
#pragma unroll
                    for (int k = 0; k < kWarps; k++) {
                        uint4 *p = (uint4 *)(smem + L.colc + k * (kCvBins * kCstr)) + i;
                        const uint4 v = *p;
                        *p = sum[s];
                        add4(sum[s], v);
                        sum[s].x -= kBias;
                        sum[s].y -= kBias;
                        sum[s].z -= kBias;
                        sum[s].w -= kBias;
                    }
                }
            }
            __syncthreads();

            const uint32_t cw_s = (uint32_t)__cvta_generic_to_shared(cw), ww_s = (uint32_t)__cvta_generic_to_shared(ww);
            const uint32_t lane2 = 2 * lane * 0x10001u, ww2 = ww_s * 0x10001u;  // below 2^16 (the layout starts with them)
            const uint32_t tab_s = (uint32_t)__cvta_generic_to_shared(smem + L.tab);
            const uint32_t ldm_s = cw_s + (((lane >> 3) & 1) * 8 + (lane & 7)) * kCstr + (lane >> 4) * 16;  // + 16 mt kCstr + 32 k-step
            // this lane's store row: chunks 0 / 1 and 2 / 3 of the row's 32 columns (+ 16 mt rows; the swizzle is of the
            // offset, whatever the buffer's address)
            const int stm_o = cv_row(1 + ((lane >> 3) & 1) * 8 + (lane & 7)) ^ ((lane >> 4) * 16);
            const uint32_t stm_s[2] = {ww_s + stm_o, ww_s + (stm_o ^ 32)};
            uint32_t bfrag[4 * N + 2];
#pragma unroll
            for (int m = 0; m < 4 * N + 2; m++) bfrag[m] = band[32 * m + lane];
            const int klo = lo - b0, kspan = hi - lo;
            const unsigned long long list_base = sh.list_base;
            for (int i = 0; (rowbits >> i) != 0; i++) {
                const int r = warp * rpw + i;
                if ((rowbits >> i) & 1u) {
                    const uint8_t *prow = plane + (r + P) * kCols + px + lane;
                    const int nth = segments ? i : __popc(rowbits & ((1u << i) - 1u));
                    float *lrow = SL.list + list_base + (size_t)(list_row + nth) * cols + lane;
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        const bool inside = lane + 32 * half < cols;
                        const unsigned v = prow[32 * half];
                        const int k = (int)v - off;
                        const bool sv = inside && (unsigned)(k - klo) < (unsigned)kspan && served[v];
                        float cval = 0.0f;
                        if (__any_sync(kFull, sv)) {
                            // window counts of the ranks the half row reads (a pixel of rank k: k - 4 .. k + 4)
                            const bool need_m[2] = {__any_sync(kFull, sv && k < 16 + kDiffs) != 0,
                                                    nrows > 16 && __any_sync(kFull, sv && k >= 16 - kDiffs)};
#pragma unroll
                            for (int mt = 0; mt < 2; mt++) {
                                if (!need_m[mt]) continue;
                                int acc[4][4];
#pragma unroll
                                for (int q = 0; q < N; q++) {
                                    uint32_t a[4];
                                    ldmatrix_x4(ldm_s + 16 * mt * kCstr + 32 * (half + q), a);
#pragma unroll
                                    for (int n = 0; n < 4; n++) {
                                        if (q == 0) mma_u8<false>(acc[n], a, bfrag[3 - n], bfrag[5 - n]);
                                        else mma_u8<true>(acc[n], a, bfrag[4 * q + 3 - n], bfrag[4 * q + 5 - n]);
                                    }
                                }
                                // counts below 2^16: the low halves of the accumulators
#pragma unroll
                                for (int n = 0; n < 4; n += 2)
                                    stmatrix_x4(stm_s[n / 2] + 16 * mt * kWStride, __byte_perm((uint32_t)acc[n][0], (uint32_t)acc[n][1], 0x5410),
                                                __byte_perm((uint32_t)acc[n][2], (uint32_t)acc[n][3], 0x5410),
                                                __byte_perm((uint32_t)acc[n + 1][0], (uint32_t)acc[n + 1][1], 0x5410),
                                                __byte_perm((uint32_t)acc[n + 1][2], (uint32_t)acc[n + 1][3], 0x5410));
                            }
                            __syncwarp();
                            if (sv) {
                                uint4 T;
                                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                                             : "=r"(T.x), "=r"(T.y), "=r"(T.z), "=r"(T.w)
                                             : "r"(tab_s + 16 * k)
                                             : "memory");
                                const unsigned p0 = lds_u16(ww_s + (cv_row(k + 1) ^ (2 * lane)));
                                const uint32_t up[2] = {(T.x ^ lane2) + ww2, (T.y ^ lane2) + ww2}, dn[2] = {(T.z ^ lane2) + ww2, (T.w ^ lane2) + ww2};
#pragma unroll
                                for (int d = 0; d < kDiffs; d++) {
                                    const unsigned p1 = lds_u16((up[d >> 1] >> (16 * (d & 1))) & 0xFFFFu);
                                    const unsigned p2 = lds_u16((dn[d >> 1] >> (16 * (d & 1))) & 0xFFFFu);
                                    const unsigned pm = p1 > p2 ? p1 : p2;
                                    // (a diff with no neighbour gives 0; without a branch around it the four loads of
                                    // the table are in flight together)
                                    const float val = __fmul_rn(__uint2float_rn((unsigned)bd.weight[d] * p0 * pm), __ldg(b.lut + p0 + pm));
                                    cval = fmaxf(cval, val);
                                }
                                if (J.plane) J.plane[(size_t)(y0 + r) * w + x0 + lane + 32 * half] = cval;
                            }
                            __syncwarp();  // the counts are read before the next half overwrites them
                            if (cval > 0.0f) {
                                my_sum += (double)cval;
                                my_cnt++;
                                // the first radix digit of the top-k selection, counted by runs of equal digits down
                                // the column (c-values lie in [0.5, 2^15))
                                const unsigned dg = (__float_as_uint(cval) >> 21) - kCvDigit0;
                                if (dg != run[half] >> 16) {
                                    count_run(half);
                                    run[half] = dg << 16;
                                }
                                run[half]++;
                            }
                        }
                        if (inside && (sv || (b0 == 0 && !segments))) lrow[32 * half] = cval;
                    }
                }
                if ((rowbits >> (i + 1)) == 0) break;
                __syncwarp();
                slide(r);
                __syncwarp();
            }
            if (hi == R) break;
            b0 = hi - kDiffs;
            __syncthreads();  // every warp is done with the counts and the table
        }
    }

    // block totals
#pragma unroll
    for (int half = 0; half < 2; half++) count_run(half);
    unsigned long long fx = __double2ull_rn(my_sum * 16777216.0);
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        fx += __shfl_down_sync(kFull, fx, o);
        my_cnt += __shfl_down_sync(kFull, my_cnt, o);
    }
    if (lane == 0) {
        sh.red_sum[warp] = fx;
        sh.red_cnt[warp] = my_cnt;
    }
    __syncthreads();
    if (tid < kCvDigits && sh.hist1[tid]) atomicAdd(&SL.hist[kCvDigit0 + tid], sh.hist1[tid]);
    if (tid == 0) {
        unsigned long long s = 0;
        unsigned n = 0;
        for (int k = 0; k < kWarps; k++) {
            s += sh.red_sum[k];
            n += sh.red_cnt[k];
        }
        if (n) {
            atomicAdd(&SL.sum_fx, s);
            atomicAdd(&SL.count, (unsigned long long)n);
        }
        if (b.tile_mass) b.tile_mass[gt] = s;
    }
}

// kMaxN: the most k-steps of a job of the launch (3 covers pads up to 32, w + h up to 6092; 5 every pad). Above pad 32 a block's
// buffers take 87 KB and more, so two share an SM whatever its registers. Launch to finished score, the block-wide form / this
// one: 4096x2160 10-bit dense (pad 33) 815 / 455 us, 5120x2880 (43) 1437 / 724, 7680x4318 (64) 3730 / 1732.
template <int kMaxN>
__global__ void __launch_bounds__(kCvThreads, kMaxN == 3 ? 3 : 2) cvalues_kernel(const __grid_constant__ CvBatch b)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CvShared sh;
    wait_for_previous();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (b.need_span < 0) {  // the codes whose c-value is needed, when they are no single range
        for (int word = warp; word < 32; word += kWarps) {
            const int code = word * 32 + lane;
            const unsigned m = __ballot_sync(kFull, code < b.band.band_size && needs_cvalue(code, b.band));
            if (lane == 0) sh.needbits[word] = m;
        }
        __syncthreads();
    }
    auto tile_body = [&](int gt, unsigned known) {
        const CvJob &J = b.job[find_job(b.njobs, gt, [&](int k) { return b.job[k].first_tile; })];
        if (b.run && !b.run[J.run_index]) return;
        const int n = cv_ksteps(J.pad);
        if (n == 2) tile_cvalues<2>(b, J, gt, known, smem, sh);
        else if (kMaxN == 3 || n == 3) tile_cvalues<3>(b, J, gt, known, smem, sh);
        else if (kMaxN > 3 && n == 4) tile_cvalues<4>(b, J, gt, known, smem, sh);
        else if (kMaxN > 3) tile_cvalues<5>(b, J, gt, known, smem, sh);
    };
    // tiles are numbered by job, a picture's scales in order; they are taken from the last one on, because the small
    // scales' few tiles hold the most ranks (several passes): taken last, they were a tail in which most SMs idled
    // (a quarter of the launch on one 4K picture)
    if (!b.tiles) {
        tile_body(b.total_tiles - 1 - (int)blockIdx.x, kNoRange);
        return;
    }
    const unsigned count = *b.tile_count;
    for (;;) {
        if (tid == 0) sh.next_tile = atomicAdd(b.tile_next, 1u);
        __syncthreads();
        const unsigned i = sh.next_tile;
        if (i >= count) break;
        tile_body((int)b.tiles[count - 1 - i], b.tile_range ? b.tile_range[count - 1 - i] : kNoRange);
        __syncthreads();
    }
}

// The list of the tiles that can hold a needed code, each with a range of its codes: a warp per tile, from the strips of
// scales 0 and 1 or the words of the others. (From the words of all scales it took 70 us for 16 uneven pairs, which have
// 210 MB of them, now about 18; the strips add 19 us to the 269 of the kernel that makes the words.)
__global__ void __launch_bounds__(kCvThreads) cv_list_kernel(const __grid_constant__ CvBatch b, unsigned *tiles, unsigned *ranges)
{
    __shared__ unsigned found[kWarps];
    wait_for_previous();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = blockIdx.x * kWarps, gt = first + warp;
    unsigned range = kNoRange;  // (no band code is 0xFFFF)
    if (gt < b.total_tiles) {
        const CvJob &J = b.job[find_job(b.njobs, gt, [&](int k) { return b.job[k].first_tile; })];
        const int tile = gt - J.first_tile, th = J.tile_rows ? J.tile_rows : kCvTY;
        const int x0 = (tile % J.tiles_x) * kCvTX, y0 = (tile / J.tiles_x) * th, rows = min(th, J.h - y0);
        unsigned lo = 0xFFFFu, hi = 0;
        if (J.strips) {
            // 8 rows x 64 columns each (scale 0) or 4 x 32 (scale 1): at most 32, a lane each
            const int sc = J.scale, col = (x0 >> (6 - sc)) + (lane & sc), r = (lane >> sc) * (8 >> sc), row = y0 + r;
            const int bx = (J.w + (64 >> sc) - 1) >> (6 - sc);
            if (r < rows && col < bx) {
                const unsigned v = __ldg(J.strips + 8 * ((row >> (6 - sc)) * bx + col) + ((row >> (3 - sc)) & 7));
                lo = v & 0xFFFFu;
                hi = v >> 16;
            }
        } else {
            const int align = row_align(J);
            uint32_t lo2 = 0xFFFFFFFFu, hi2 = 0;  // as prep0_kernel's strips
#pragma unroll 8
            for (int i = lane; i < rows * (kCvTX / 8); i += 32) {
                const uint4 q = load8(J, align, y0 + (i >> 3), x0 + 8 * (i & 7));
                const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    lo2 = min2(lo2, v[k] ^ 0x80008000u);
                    hi2 = max2(hi2, v[k]);
                }
            }
            lo = min(lo2 & 0xFFFFu, lo2 >> 16);
            hi = max(hi2 & 0xFFFFu, hi2 >> 16) & 0x7FFFu;
        }
        const int least = max((int)__reduce_min_sync(kFull, lo), b.need_first), greatest = min((int)__reduce_max_sync(kFull, hi), b.need_last);
        if (least <= greatest) range = (unsigned)(least - b.band.band_base) | (unsigned)(greatest - b.band.band_base) << 16;
        else if (b.tile_mass && lane == 0) b.tile_mass[gt] = 0;
    }
    if (lane == 0) found[warp] = range;
    __syncthreads();
    if (warp == 0) {
        const unsigned r = lane < kWarps ? found[lane] : kNoRange, set = __ballot_sync(kFull, r != kNoRange);
        unsigned at = 0;
        if (lane == 0 && set) at = atomicAdd(b.busy, (unsigned)__popc(set));
        at = __shfl_sync(kFull, at, 0) + __popc(set & ((1u << lane) - 1u));
        if (r != kNoRange) {
            tiles[at] = (unsigned)(first + lane);
            ranges[at] = r;
        }
    }
}

template <int kMaxN>
cudaError_t launch_cvalues_n(CvBatch &b, cudaStream_t s)
{
    const size_t smem = cvalues_smem_bytes(b.max_pad);
    // the most a launch of this form takes, not this launch's size: the attribute is the kernel's, and another thread's
    // smaller picture may set it between here and the launch
    static_assert(cv_ksteps(32) == 3 && cv_ksteps(kMaxPad) == 5, "the pads of the two forms");
    cudaError_t e = cudaFuncSetAttribute(cvalues_kernel<kMaxN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)cvalues_smem_bytes(kMaxN == 3 ? 32 : kMaxPad));
    if (e != cudaSuccess) return e;
    LaunchTimer t("cambi_cvalues", s);
    if (!b.tiles && b.busy) {
        unsigned *tiles = b.busy + 2, *ranges = tiles + b.total_tiles;
        e = launch_kernel(b.chained, cv_list_kernel, dim3((b.total_tiles + kWarps - 1) / kWarps), kCvThreads, 0, s, b, tiles, ranges);
        if (e != cudaSuccess) return e;
        b.tiles = tiles;
        b.tile_range = ranges;
        b.tile_count = b.busy;
        b.tile_next = b.busy + 1;
        b.chained = 1;
    }
    const int grid = b.tiles && b.total_tiles > kCvListBlocks ? kCvListBlocks : b.total_tiles;
    return launch_kernel(b.chained, cvalues_kernel<kMaxN>, dim3(grid), kCvThreads, smem, s, b);
}
}  // namespace

size_t cvalues_smem_bytes(int max_pad)
{
    size_t most = 0;  // the layout is not monotonous in the pad (its k-steps are not)
    for (int p = 0; p <= max_pad; p++) most = most > (size_t)cv_layout(p).total ? most : (size_t)cv_layout(p).total;
    return most;
}

cudaError_t launch_cvalues(const CvBatch &batch, cudaStream_t s)
{
    if (batch.total_tiles <= 0) return cudaSuccess;
    CvBatch b = batch;
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
    b.need_first = lo < 0 ? 1 : lo + b.band.band_base;
    b.need_last = lo < 0 ? 0 : hi + b.band.band_base;
    int n = 2;
    for (int j = 0; j < b.njobs; j++) n = n > cv_ksteps(b.job[j].pad) ? n : cv_ksteps(b.job[j].pad);
    if (n > 5) return cudaErrorInvalidValue;  // a pad over kMaxPad: no kernel form reaches that far
    return n <= 3 ? launch_cvalues_n<3>(b, s) : launch_cvalues_n<5>(b, s);
}

const void *kernel_entry_cvalues() { return (const void *)cvalues_kernel<3>; }

}  // namespace es
