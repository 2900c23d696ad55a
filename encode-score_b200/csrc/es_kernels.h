// Job descriptors and launchers shared by the host code (C++) and the kernels (CUDA).
//
// Kernels take their work as tables of jobs passed by value in the kernel parameters (up to 32 KB since CUDA 12.1),
// so that one launch covers any mix of pictures and scales: the single-picture Cambi path and the batched frame step
// use the same kernels. Each launcher returns the cudaError_t of the launch.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace es {

// Every launcher below ends with after_launch(): it counts the launch (es_launch_count) and returns its error.
void count_launch();
// Adds n (which may be negative) to the launch count: a graph replay counts its kernel nodes, a capture takes back
// the launches its recording counted.
void count_launches(long long n);
// The launch that es_fail_launch asked to fail (once).
bool launch_fails();
inline cudaError_t after_launch()
{
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return launch_fails() ? cudaErrorUnknown : e;
}

// Brackets a launcher's kernel launch with CUDA events on its stream while kernel timing is switched on
// (es_kernel_timing); a no-op otherwise.
struct LaunchTimer {
    int slot = -1;
    cudaStream_t stream;
    LaunchTimer(const char *name, cudaStream_t s);
    ~LaunchTimer();
    LaunchTimer(const LaunchTimer &) = delete;
};
// True while es_kernel_timing(2) is in force: CAMBI instances then queue all their work on the caller's stream and frame
// steps theirs on one stream, so that nothing runs beside a timed kernel and its events bracket that kernel alone.
bool serial_streams();
// True while es_kernel_timing is on (its events need plain launches, so graphs are not used then).
bool kernel_timing_on();

constexpr int kScales = 5;
constexpr int kDiffs = 4;
constexpr uint16_t kNone = 0xFFFF;
constexpr uint16_t kMaskBit = 0x8000;  // a scale's plane holds value | mask << 15
constexpr int kMaxBand = 1024;         // codes of a 10-bit pipeline
constexpr int kMaxPad = 64;            // window 129
constexpr int kMaxPictures = 64;       // pictures in one batched launch
constexpr int kMaxJobs = kMaxPictures * 5;  // pictures x scales in one c-value launch
constexpr int kWin = 16;               // detail window side (src/kernels.cu:331)

#ifdef __CUDACC__
// A launch that is made ready while the kernel before it on the stream runs, and begins when that kernel's last block leaves
// (programmatic dependent launch): `kernel` calls wait_for_previous() before it reads or writes memory, and what comes
// before the launch on the stream is a kernel. Launch to finished score through Python, in the build that brought it: CAMBI
// of one 640x360 picture 77 -> 68 us, of 1920x1080 121 -> 112; a step of a 1920x1080 pair, whose kernels are launched one
// by one, 160 -> 152 us.
// chained = false: a plain launch.
template <typename... P, typename... A>
cudaError_t launch_kernel(bool chained, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, const A &...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = chained ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
    const cudaError_t f = after_launch();
    return e != cudaSuccess ? e : f;
}
// Until the kernels this one was launched to follow are complete and their writes visible (at once in a plain launch).
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Once every block of this kernel has said so or left, the next kernel's blocks may take free places and wait there: 1 us
// more for CAMBI of one picture. Only where a chain has the GPU to itself: beside another chain, the waiting blocks hold
// places that it could use (a step of a 1920 x 800 pair 161 -> 171 us).
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::); }

// The job whose range of blocks or tiles holds t: the last job j with first(j) <= t, by binary search over a job
// table whose first blocks do not decrease (a job without blocks shares its first with the next).
template <typename First>
__device__ __forceinline__ int find_job(int njobs, int t, First first)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (t >= first(mid)) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
#endif

// CAMBI's band parameters (src/kernels.cu:65-69 CambiParams without the per-scale size).
struct Band {
    int band_base, band_size, vlt;
    int tvi[kDiffs];
    int weight[kDiffs];
};

// ---- counters of the c-values -------------------------------------------------------------------------------------
// Per picture-scale counters in device memory. The c-values are exact multiples of 2^-24 (they are at least 0.5), so
// their sum is kept exactly as an integer in those units; the order of additions does not matter.
// The c-value kernel also counts the positive values by the top 11 bits of their floats (the first radix digit of the
// top-k selection): at least 0.5 and, for windows of up to 129 and weights of up to 4, below 2^15 (4 x 129^2 / 4 = 16641 at
// most), so those digits lie in kCvDigit0 .. kCvDigit0 + 60; larger ones, of other weights, are counted one by one.
constexpr unsigned kCvDigit0 = 0x3F000000u >> 21, kCvDigits = 64;
struct CvSlot {
    unsigned long long sum_fx, count;  // positive c-values: sum in 2^-24 units, number
    unsigned long long list_n;         // values in `list`
    unsigned long long n, k;           // pixels of the scale, top-k count
    unsigned long long above_fx, above_n;
    unsigned long long remaining1, remaining2;  // radix select state after each round
    unsigned prefix1, prefix2;
    float *list;                       // c-values, zeros among them (capacity n): every positive one is there once
    unsigned pad_[2];
    alignas(16) unsigned hist[2048];   // counts of the first radix digit
    // counts of the second and the last digit: clear between launches (the score kernel clears what a selection used)
    alignas(16) unsigned hist1[2048];
    alignas(16) unsigned hist2[1024];
};

// ---- scales 0 and 1: preprocessing, zero-derivative mask and mode filter of one plane, then its first decimation --
struct Prep0Job {
    const uint16_t *img;  // input plane, `pitch` pixels per row
    int pitch, w, h, depth, mask_index;
    uint16_t *word;       // out: w x h, mode-filtered value | mask << 15
    int tiles_x, first_tile;  // set by the launcher
    // optional (the tile proposal): the feature map of the words, ceil(h / 4) x ceil(w / 4) (mean, mask share) pairs
    // as the proposal's feature kernel makes it, and per 64 x 64 tile whether a pixel needs a c-value (0 or 1)
    float2 *feat;
    unsigned *need;
    // optional: scale 1 (w1 x h1 = the halved size, rounded up) made in the same pass; nullptr: scale 0 only
    uint16_t *word1;
    int w1, h1;
    // optional, with word1: strips[8 t + g], t a 64 x 64 tile of scale 0: the least and (<< 16) the greatest masked value of
    // rows 8 g .. 8 g + 7 of the tile, a least above the greatest where there is none. After all tiles, the same for 4 rows
    // of each tile's 32 x 32 words of scale 1.
    unsigned *strips;
};
// Words of a w x h picture's strips, both scales.
inline size_t prep0_strips(int w, int h) { return (size_t)((w + 63) / 64) * ((h + 63) / 64) * 16; }
constexpr int kPrep0MaxJobs = kMaxPictures;
struct Prep0Batch {
    Prep0Job job[kPrep0MaxJobs];
    int njobs, total_tiles;  // total_tiles: set by the launcher
    Band band;               // the codes that need c-values, for the need flags
    int need_lo, need_span;  // set by the launcher: the needed values are need_lo .. need_lo + need_span when they
                             // form one range (need_span >= 0), else need_span = -1 and the band's bits decide
    // optional: clears the counters of slots [0, nslots) and sets each slot's n and k
    CvSlot *slots;
    int nslots;
    const unsigned long long *slot_n, *slot_k;
    unsigned *clear;  // optional, with slots: two words set to 0
    int chained;      // what comes before on the stream is the kernel that makes the planes (launch_kernel)
};
cudaError_t launch_prep0(Prep0Batch &b, cudaStream_t s);

// ---- scales 2..4: decimation and mode filter ------------------------------------------------------------------------
struct DecJob {
    const uint16_t *src;  // scale 1's words, rows of sw
    int sw;
    uint16_t *dst[3];     // the words of scales 2, 3 and 4
    int w[3], h[3];       // their sizes
    int first_block;      // set by the launcher
};
constexpr int kDecMaxJobs = kMaxPictures;
struct DecBatch {
    DecJob job[kDecMaxJobs];
    int njobs;
    int chained;  // what comes before on the stream is the kernel of scales 0 and 1
    int early;    // let the next kernel start early (let_next_start)
};
cudaError_t launch_decimate_mode(DecBatch &b, cudaStream_t s);

// ---- c-values --------------------------------------------------------------------------------------------------------
struct CvJob {
    const uint16_t *word;
    int w, h, pad;
    int tiles_x, first_tile;
    int slot;       // index into the CvSlot array
    float *plane;   // optional: every computed c-value at its pixel
    int run_index;  // the entry of CvBatch::run that gates this job (with a run table)
    int tile_rows;  // rows of this job's tiles: 64 (0 means 64), 32 or 16; tiles are numbered row by row
    int scale;      // with strips: 0 or 1
    const unsigned *strips;  // optional, scales 0 and 1, for the busy tiles' list: this scale's part of Prep0Job::strips
};
struct CvBatch {
    CvJob job[kMaxJobs];
    int njobs, total_tiles, max_pad;
    Band band;
    const float *lut;  // lut[i] = 1/i as float, i < (2 max_pad + 1)^2 + 1
    CvSlot *slots;
    // Optional tile list: the launch then has a fixed grid whose blocks take tiles[*tile_next++] (global tile ids, job
    // by job as first_tile numbers them) while the counter is below *tile_count; *tile_next must be 0 at launch.
    const unsigned *tiles;
    const unsigned *tile_count;
    unsigned *tile_next;
    const unsigned *tile_range;  // optional, by list entry: a range of band codes, least | greatest << 16, that holds the tile's
                                 // needed ones
    // Optional, without a list: 2 + 2 total_tiles words, the first two 0 at launch (Prep0Batch::clear). A kernel of its own
    // then first lists the tiles that can hold needed codes.
    unsigned *busy;
    int chained;  // what comes before on the stream is the kernel of scales 2 to 4
    // Optional: per global tile, the exact sum of its positive c-values in 2^-24 units (0 for a tile with none).
    unsigned long long *tile_mass;
    // Optional: run[job.run_index] == 0 skips the job's tiles.
    const int *run;
    int need_lo, need_span;      // set by the launcher: as Prep0Batch's
    int need_first, need_last;   // set by the launcher: the least and greatest needed value
};
// A launch of at least this many tiles lists its busy tiles first (CvBatch::busy). Most tiles of most pictures need no
// c-value, but a block of their own costs 2 to 4 us of a place on an SM to find that out. Without and with the list, in the
// build that brought it: 16 uneven pairs (26.6 thousand tiles) 706 and 588 us of c-values, a step of a 3840 x 2160 pair (5.5
// thousand) 388 and 375; below, the launch more costs what it saves: a step of a 1920 x 1080 pair (2.3 thousand) 170 and 173.
constexpr int kCvBusyTiles = 4096;
// Blocks of a tile-list launch.
constexpr int kCvListBlocks = 148 * 3;
constexpr int kCvTX = 64, kCvTY = 64, kCvThreads = 256, kCvBins = 32;
size_t cvalues_smem_bytes(int max_pad);
// 64 x 64 c-value tiles of a w x h scale.
inline int cv_tiles(int w, int h) { return ((w + kCvTX - 1) / kCvTX) * ((h + kCvTY - 1) / kCvTY); }
// The tile rows of a w x h scale when nothing else asks for a height; tiles0: the launch's 64 x 64 tiles of scale 0, all
// pictures. Short tiles cost more in all (the window margins are staged and counted again for fewer rows) but a block is
// done sooner, which decides where the tiles do not fill the chip's 444 places or hold many ranks (several passes),
// as the small scales' do. Measured, c-values of one picture, 64 rows everywhere / by this rule: 640x360 8-bit 55 / 24
// us, 1920x1080 8-bit 96 / 57 us, 3840x2160 10-bit 190 / 108 us; 32 rows for scale 1 of a dense 4K picture instead of 64:
// 260 against 247 us, 64 rows for scale 0 of the 1080p one instead of 32: 69 against 57 us. The line at 592 tiles was drawn
// from these three; just above it 64 rows are too many: a 1920x800 pair (780 tiles) takes 36 us, with 32 rows at scale 0 29
// us, with the autotuned rows 28.
inline int cv_default_tile_rows(int w, int h, int tiles0)
{
    const int tiles = cv_tiles(w, h);
    if (tiles0 >= 592) return tiles >= 148 ? 64 : tiles >= 74 ? 32 : 16;
    return tiles >= 148 ? 32 : 16;
}
cudaError_t launch_cvalues(const CvBatch &b, cudaStream_t s);

// ---- top-k pooling and score -------------------------------------------------------------------------------------
// The exact k-th largest c-value, and the sum and count of the values above it, of every slot whose positive count
// exceeds k, after the c-value launches (which leave the first digit's counts in each slot): radix rounds of 11, 11 and
// 10 bits, the second and third over the slots' lists, the last one also summing what lies above the selected value. The
// score kernel makes the last pick.
// Follows the c-value kernel on the stream (launch_kernel). early: let_next_start.
cudaError_t launch_topk(CvSlot *slots, int nslots, cudaStream_t s, bool early);
struct ScoreJob {
    int first_slot;  // kScales consecutive slots
    int window;
    double *score;   // out: the score, then the pooled value of each scale
    double *host;    // the same in page-locked host memory, or null
};
constexpr int kScoreMaxJobs = kMaxPictures;
struct ScoreBatch {
    ScoreJob job[kScoreMaxJobs];
    int njobs;
    CvSlot *slots;
};
// Follows the last top-k round on the stream.
cudaError_t launch_score(const ScoreBatch &b, cudaStream_t s);

// ---- frame unpacking ---------------------------------------------------------------------------------------------
struct FrameViewDev {
    const void *y, *u, *v;
    int ypitch, cpitch, semi, bytes, shift, depth;
};
struct UnpackJob {
    FrameViewDev f;
    int x0, y0;
    uint16_t *y16, *u16, *v16;  // w x h, w/2 x h/2
    int w, h, pd;               // common picture area and pipeline depth of this picture's source
    int first_block;            // in blocks of unpack_blocks(w, h)
};
constexpr int kUnpackMaxJobs = kMaxPictures;
// Blocks of 256 threads for one picture of w x h: a thread takes 4 consecutive 2 x 2 groups of a chroma row.
inline int unpack_blocks(int w, int h) { return (int)(((size_t)((w / 2 + 3) / 4) * (h / 2) + 255) / 256); }
struct UnpackView {
    FrameViewDev f;
    int x0, y0;
};
struct UnpackBatch {
    UnpackJob job[kUnpackMaxJobs];
    int njobs, total_blocks;
    // optional: job j's frame view and crop are views[j] in device memory instead of job[j].f, x0, y0 (so a captured
    // graph can take new input addresses each step)
    const UnpackView *views;
};
cudaError_t launch_unpack(const UnpackBatch &b, cudaStream_t s);

// ---- the VMAF picture feed (src/kernels.cu:537-545) -------------------------------------------------------------
struct PictureJob {
    const uint16_t *src;  // w x h values, rows of w
    void *dst;            // rows of `pitch` bytes, `bytes` (1 or 2) per sample
    int w, h, pitch, bytes;
    int first_block;      // set by the launcher
};
constexpr int kPictureMaxJobs = kMaxPictures;
struct PictureBatch {
    PictureJob job[kPictureMaxJobs];
    int njobs;
};
cudaError_t launch_to_pictures(PictureBatch &b, cudaStream_t s);

// ---- detail window statistics ------------------------------------------------------------------------------------
constexpr int kMaxEncodes = 16;
struct WindowJob {
    const uint16_t *yr;                 // source luma (pipeline depth)
    const uint16_t *yd[kMaxEncodes];    // encode luma
    float *stats;                       // [nenc][windows][8]
    int nenc, w, h, up;
    int first_block;                    // set by the launcher
};
// Per-source work of a frame step for up to kMaxSources sources in one launch.
constexpr int kMaxSources = 32;
struct WindowBatch {
    WindowJob job[kMaxSources];
    int njobs;
};
// Follows the squared errors on the stream (launch_kernel).
cudaError_t launch_window_stats(WindowBatch &b, cudaStream_t s);

// ---- lasting texture ------------------------------------------------------------------------------------------------
// Running sums of the source's luma over the even and odd frame offsets of the centre frame c = f - 6:
//   E(c) = sum y(c + k), k = +-2, +-4, +-6;   O(c) = sum y(c + k), k = +-1, +-3, +-5
// with E(c) = O(c-1) - y(c) + y(c+6) and O(c) = E(c-1) - y(c-7) + y(c-1); missing frames count as 0.
struct PersistJob {
    const uint16_t *e_old, *o_old;  // 10-bit scale, w x h
    uint16_t *e_new, *o_new;
    const uint16_t *y_m13, *y_m7, *y_c, *y_f;  // frames f-13, f-7, f-6 (= centre), f; nullptr = zero
    const uint16_t *yd[kMaxEncodes];           // encodes' luma at the centre frame
    float *out;                                // [nenc][windows][5]
    int nenc, w, h, up;
    int stats;  // 0: only advance the running sums
    int first_block;  // set by the launcher
};
struct PersistBatch {
    PersistJob job[kMaxSources];
    int njobs;
};
// Follows the window figures on the stream (launch_kernel).
cudaError_t launch_persist(PersistBatch &b, cudaStream_t s);

// ---- PSNR squared errors and color sums --------------------------------------------------------------------------
struct PairSumsJob {
    const uint16_t *ry, *ru, *rv;  // source planes (pipeline depth)
    const uint16_t *dy[kMaxEncodes], *du[kMaxEncodes], *dv[kMaxEncodes];
    unsigned long long *sse;       // [nenc][3]
    unsigned long long *color;     // [nenc + 1][3]: sum U, sum V, strength in 2^-30 units; source last
    int nenc, w, h, up;
    int first_block;  // set by the launcher
};
struct PairSumsBatch {
    PairSumsJob job[kMaxSources];
    int njobs;
};
cudaError_t launch_pair_sums(PairSumsBatch &b, cudaStream_t s);

// ---- per-frame reduction of the window figures (src/main.cpp:606-641) -------------------------------------------
struct FrameFigures {
    double all_r[3], all_d[3], st_r[3], st_d[3];
    double sh_all_x[2], sh_st_x[2];
    double own, mine;
    unsigned n_structure, n_lasting;
    float threshold;
    unsigned pad_;
};
// The last kernel writes the step's figures to page-locked host memory and leaves the sums and counts it copied clear
// for the step after the next.
struct CollectJob {
    const float *stats;            // [nenc][windows][8]
    const float *persist;          // [nenc][windows][5], centre frame (nullptr: no lasting texture this frame)
    const uint8_t *centre_mask;    // structure mask of the centre frame
    uint8_t *mask;                 // out: structure mask of this frame
    FrameFigures *host_fig;        // out (host): [nenc]
    uint16_t *host_bins;           // out (host): [nenc] of 6 arrays of up to `windows` bins (amount 0-2, matching 0-1,
                                   // lasting), only those that count, from the start of each array in no fixed order
    unsigned *bin_n;               // scratch: [nenc][2], bins in each of the first five arrays (the structure windows)
                                   // and in the lasting array
    unsigned *host_bin_n;          // out (host): the same
    unsigned long long *sums;      // PairSumsJob's sse [nenc][3], then color [nenc + 1][3]
    unsigned long long *host_sums; // out (host): the same
    float *threshold;              // scratch: the frame's structure threshold
    double *partials;              // scratch: [nenc][collect_blocks(windows)][kCollectSums]
    int nenc, windows;
    int first_enc;  // set by the launcher: this job's encodes are grid rows first_enc .. first_enc + nenc - 1
};
struct CollectBatch {
    CollectJob job[kMaxSources];
    int njobs;
};
constexpr int kCollectSums = 20;  // 18 double sums and 2 counts per block
int collect_blocks(int windows);
// The structure threshold and mask (needs the window figures only), then the windows' bins and sums (needs the lasting
// figures too).
cudaError_t launch_collect_threshold(CollectBatch &b, cudaStream_t s);
cudaError_t launch_collect_sums(CollectBatch &b, cudaStream_t s);

// ---- temporal alignment (src/kernels.cu:502-520, src/main.cpp:336-353) -------------------------------------------
constexpr int kThumbW = 64, kThumbH = 36, kThumbPixels = kThumbW * kThumbH;
constexpr int kThumbFrames = 64;  // frames of one thumbnail launch
struct ThumbBatch {
    FrameViewDev f[kThumbFrames];
    int n, x0, y0, w, h;  // frames; the crop of every frame
    float *out;           // [frame][kThumbH][kThumbW]
};
cudaError_t launch_thumbnails(const ThumbBatch &b, cudaStream_t s);
cudaError_t launch_offset_totals(const float *ref, int n_ref, const float *probe, int n_probe, double *totals, cudaStream_t s);
// Totals of a search of up to offset_totals_slot_lags() lags: slot 0 .. offset_totals_slots() - 1 of a fixed device array
// of the CUDA context current on the calling thread.
int offset_totals_slots();
int offset_totals_slot_lags();
cudaError_t offset_totals_slot(int slot, double **ptr);

// ---- learned tile proposal -------------------------------------------------------------------------------------
// A 4-layer network of valid 3 x 3 convolutions (2 -> 16 -> 16 -> 16 -> 1, ReLU after the first three) on 4 x 4
// block features of scale 0 predicts log1p(mean positive c-value) of each 64 x 64 scale-0 tile. Parameters are one
// float array: per layer the weights [co][ci][3][3], then the biases.
constexpr int kNetParams = 5089;
__host__ __device__ constexpr int net_w(int l) { return l == 0 ? 0 : l == 1 ? 304 : l == 2 ? 2624 : 4944; }   // weights of layer l
__host__ __device__ constexpr int net_b(int l) { return l == 0 ? 288 : l == 1 ? 2608 : l == 2 ? 4928 : 5088; }  // its biases
constexpr int kFeatTile = 24;  // feature pixels per side around one tile (16 + 2 x 4 halo)
// mma B fragments: layers 1 and 2 (16 -> 16) [layer][tap][n tile][register][lane], then layer 3 (16 -> 1, its one
// output channel in column 0 of an 8-wide n tile) [tap][register][lane], then layer 0 (2 -> 16, k = 4 tap + 2 part +
// input channel, 36 of 3 k-steps of 16 used) [k-step][n tile][register][lane]
constexpr int kNetFrags12 = 2 * 9 * 2 * 2 * 32;
constexpr int kNetFrags3 = kNetFrags12 + 9 * 2 * 32;
constexpr int kNetFrags = kNetFrags3 + 3 * 2 * 2 * 32;

struct PredJob {
    const uint16_t *word;  // scale-0 words of a picture
    int w, h, tiles_x, tiles_y, first_tile;
    float2 *feat;          // its feature map: ceil(h / 4) x ceil(w / 4) (mean, mask share) pairs
    int first_block;       // set by the features launcher
};
struct PredBatch {
    PredJob job[kMaxPictures];
    int njobs, total_tiles;
    Band band;
    const float *params;    // bfloat16-rounded parameters (as floats)
    const uint32_t *frags;  // B fragments of layers 1, 2 and 3
    unsigned *need;         // per scale-0 tile: non-zero when a pixel of it needs a c-value, then a tile counter
                            // (total_tiles + 1 words, zeroed by the launcher unless features_ready)
    int features_ready;     // the feature maps and need flags were made with scale 0 (prep0): only predict
    float *pred;            // per scale-0 tile: the prediction, -inf where no pixel needs a c-value
};
// Both kernels of a prediction: the feature maps (and need flags) of every picture, then the network per tile.
cudaError_t launch_predict(PredBatch &b, cudaStream_t s);
inline size_t feature_map_size(int w, int h) { return (size_t)((w + 3) / 4) * ((h + 3) / 4); }

// Features of n crops: crop i covers scale-0 pixels from (xy[2 i], xy[2 i + 1]) on, fw x fh feature pixels of 4 x 4.
cudaError_t launch_net_features(const uint16_t *word, int w, int h, const int *xy, int n, int fw, int fh, float *out,
                                cudaStream_t s);
// Training on crops (NCHW float, h even): forward of layer l (input n x ci x h x w, output n x co x (h - 2) x (w - 2),
// ReLU for l < 3); backward of layer l (its weights' and biases' gradients in net_grad_blocks parts of kNetParams floats
// and, for l > 0, the gradient of its input times the ReLU mask of that input into gin); the tile loss of the last layer (n x 1 x 16a x 16b against
// n x a x b labels: per-tile squared differences into loss_parts, the gradient of the last layer's output into gz);
// and the gradients from every layer's parts, with Adam's step on them when lr > 0 (master weights, their
// bfloat16-rounded copy, moments).
constexpr int kNetGradBlocks = 148 * 2;                 // parts at most
constexpr int kNetGradRows = 8, kNetGradCols = 36;      // output pixels of a block's tile
// Parts of a layer with an n x h x w input.
inline int net_grad_blocks(int n, int h, int w)
{
    const size_t tiles = (size_t)n * ((h - 2 + kNetGradRows - 1) / kNetGradRows) * ((w - 2 + kNetGradCols - 1) / kNetGradCols);
    return tiles < (size_t)kNetGradBlocks ? (int)tiles : kNetGradBlocks;
}
cudaError_t launch_net_forward(int layer, const float *in, int n, int h, int w, const float *params, float *out,
                               cudaStream_t s);
cudaError_t launch_net_backward(int layer, const float *gout, const float *in, int n, int h, int w, const float *params,
                                float *gin, float *parts, cudaStream_t s);
cudaError_t launch_net_loss(const float *z, const float *labels, int n, int ta, int tb, float *gz, float *loss_parts,
                            cudaStream_t s);
cudaError_t launch_net_grads(const float *parts, int n, int h, int w, float *params, float *rounded, float *grads, float *m, float *v,
                             float lr, float b1, float b2, float eps, int t, cudaStream_t s);
// The mma B fragments of layers 1 and 2 (kNetFrags words) from the bfloat16-rounded parameters.
cudaError_t launch_net_pack(const float *rounded, uint32_t *frags, cudaStream_t s);

// The proposal of one frame step over the c-value job table: which tiles of scales 0 and 1 run now (proposed or
// audited) and which wait for the fallback; scales 2-4 always run.
constexpr uint8_t kTileSkip = 0, kTileRun = 1, kTileAudit = 2, kTileEmpty = 3;
struct ProposeJob {
    int first_tile, tiles_x, tiles_y, scale, picture;
    int pred_first, pred_tiles_x, pred_tiles_y;  // the picture's scale-0 tile predictions
};
struct ProposeBatch {
    ProposeJob job[kMaxJobs];
    int njobs, total_tiles;
    const float *pred;
    float threshold;
    const float *pic_threshold;           // per picture (budget mode), else null: threshold for all
    unsigned audit_permille[2];           // per scale 0, 1
    const unsigned long long *frame;      // device: the step's frame number (seeds the audit sample)
    unsigned *list_a, *count_a;           // tiles to run now
    unsigned *list_b, *count_b;           // tiles of the fallback
    uint8_t *kind;                        // per global tile
    unsigned *n_audit, *n_skip;           // per job (zeroed before the launch, with the counts)
};
cudaError_t launch_propose(const ProposeBatch &b, cudaStream_t s);
// Budget mode: per picture, the skip threshold T >= `threshold` of the predictions such that the predicted score
// contribution of the scale-0 tiles below T, sum of scale * expm1(pred) * pixels, stays within `budget`.
constexpr int kBudgetBins = 1024;
constexpr float kBudgetBinsPerUnit = 128.0f;  // bins cover predictions 0 .. 8
struct BudgetJob {
    int pred_first, tiles_x, tiles_y, w, h, picture;
    double scale;  // score per unit of scale-0 c-value mass: 16 / (k0 window^2)
};
struct BudgetBatch {
    BudgetJob job[kMaxPictures];
    int njobs;
    const float *pred;
    float threshold;
    double budget;
    float *pic_threshold;  // out, by picture
};
cudaError_t launch_budget(const BudgetBatch &b, cudaStream_t s);
struct AuditJob {
    int job[2];         // the picture's scale-0 and scale-1 jobs in the propose table
    int first_tile[2];  // their global tile ranges
    int tiles[2];
    double k[2];        // their top-k counts
    int window;
};
struct ProposalStats {
    float estimate;     // estimated change of the score from the skipped tiles
    int fallback;       // 1: the skipped tiles ran too
    unsigned run[2], audited[2], skipped[2];
};
struct AuditBatch {
    AuditJob job[kMaxPictures];
    int njobs;
    const unsigned long long *tile_mass;
    const uint8_t *kind;
    const unsigned *n_audit, *n_skip;
    double tolerance;
    int *run;                 // out: per picture, 1 when the fallback runs
    ProposalStats *stats;     // out: per picture
};
cudaError_t launch_audit(const AuditBatch &b, cudaStream_t s);

}  // namespace es
