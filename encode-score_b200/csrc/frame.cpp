// es_frame: the per-frame measures of one source against its encodes, the queue / collect pair of src/main.cpp:518-643
// behind a C ABI: a batch (es_batch) of one source. Frame f's GPU work runs after what is queued on the caller's stream,
// which then waits for it, as one launch per stage for all its pictures; collect(f) waits for the figures in page-locked
// memory and adds them to the caller's accumulators while the GPU works on frame f + 1. Like the reference, whatever a
// frame's figures are read from comes in two, used by f % 2.
//
// It had one CAMBI instance per picture and parity, each with its own chain of launches: 31 launches and 242 us a frame of
// one 1080p encode, as a batch 13 launches and 192 us (152 since, with faster kernels). The steps are launched, not replayed
// from graphs: replays took 183 us then, but capturing a frame's graph takes another 170 us in each of the first 14 ring
// phases.
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "es_internal.h"

using namespace es;

struct es_frame {
    int nenc = 0;
    es_batch *batch = nullptr;
    std::vector<es_frame_view> views;
    std::vector<int> crops;
    ~es_frame() { es_batch_destroy(batch); }
};

namespace {

// A failed call of the batch beneath fails this one alike; its message names the call that was made.
void pass(int status)
{
    if (status == ES_OK) return;
    std::string what = es_last_error();
    const std::string theirs = "es_batch_", ours = "es_frame_";
    for (size_t at = 0; (at = what.find(theirs, at)) != std::string::npos; at += ours.size()) what.replace(at, theirs.size(), ours);
    throw Error(status, what);
}

// the n bins the collect kernel wrote (only those that count)
void add_bins(es_histogram &hist, const uint16_t *bins, unsigned n)
{
    for (unsigned i = 0; i < n; i++) hist.bins[bins[i]]++;
    hist.n += n;
}

}  // namespace

// src/main.cpp:584-641 for one encode of a collected frame step.
es_frame_result es::collect_encode(const EncodeFigures &in, es_accum *frame_acc, es_accum *centre_acc)
{
    const size_t cn = in.n / 4;
    auto color_of = [](const unsigned long long *c, int i) { return i < 2 ? (double)c[i] : (double)c[2] * (1.0 / 1073741824.0); };
    const FrameFigures &fg = *in.fig;
    es_frame_result res{};
    res.cambi = in.banding;
    res.cambi_source = in.source_banding;
    res.psnr[0] = es_psnr(in.sse[0], in.n, in.pd);
    res.psnr[1] = es_psnr(in.sse[1], cn, in.pd);
    res.psnr[2] = es_psnr(in.sse[2], cn, in.pd);
    for (int i = 0; i < 3; i++) {
        res.color_source[i] = color_of(in.source_color, i) / (double)cn;
        res.color_encode[i] = color_of(in.encode_color, i) / (double)cn;
    }
    res.texture = in.texture;
    res.structure_windows = in.windows > 0 ? fg.n_structure : 0;
    res.lasting_windows = in.texture && in.windows > 0 ? fg.n_lasting : 0;
    if (frame_acc) {
        es_accum &acc = *frame_acc;
        acc.frames++;
        acc.cambi += in.banding;
        acc.cambi_source += in.source_banding;
        for (int i = 0; i < 3; i++) {
            acc.psnr[i] += res.psnr[i];
            acc.color_r[i] += color_of(in.source_color, i) / (double)cn;
            acc.color_d[i] += color_of(in.encode_color, i) / (double)cn;
        }
        if (in.windows > 0) {
            for (int k = 0; k < 3; k++) {
                acc.all_r[k] += fg.all_r[k];
                acc.all_d[k] += fg.all_d[k];
                acc.st_r[k] += fg.st_r[k];
                acc.st_d[k] += fg.st_d[k];
            }
            for (int k = 0; k < 2; k++) {
                acc.sh_all_r[k] += fg.all_r[k];
                acc.sh_all_x[k] += fg.sh_all_x[k];
                acc.sh_st_r[k] += fg.st_r[k];
                acc.sh_st_x[k] += fg.sh_st_x[k];
            }
            for (int k = 0; k < 3; k++) add_bins(acc.amount[k], in.bins + (size_t)k * in.windows, in.bin_n[0]);
            for (int k = 0; k < 2; k++) add_bins(acc.matching[k], in.bins + (size_t)(3 + k) * in.windows, in.bin_n[0]);
        }
    }
    if (in.texture && in.windows > 0 && centre_acc) {
        es_accum &cacc = *centre_acc;
        cacc.own += fg.own;
        cacc.mine += fg.mine;
        add_bins(cacc.lasting, in.bins + (size_t)5 * in.windows, in.bin_n[1]);
    }
    return res;
}

extern "C" {

int es_frame_create(const es_module *m, int w, int h, int pd, int n_encodes, es_frame **out)
{
    return guarded([&] {
        require(m != nullptr && out != nullptr, "es_frame_create: NULL argument");
        require(w >= 16 && h >= 16 && w % 2 == 0 && h % 2 == 0, "es_frame_create: the picture must be even and at least 16 x 16");
        require(pd == 8 || pd == 10, "es_frame_create: pipeline depth must be 8 or 10");
        require(n_encodes >= 1 && n_encodes <= kMaxEncodes, "es_frame_create: 1 to 16 encodes");
        auto fr = std::make_unique<es_frame>();
        fr->nenc = n_encodes;
        fr->views.resize(1 + n_encodes);
        fr->crops.resize(2 * (1 + n_encodes));
        const es_batch_source source{w, h, pd, n_encodes, {0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}};
        const es_batch_options direct{0};
        pass(es_batch_create(m, 1, &source, &direct, &fr->batch));
        *out = fr.release();
    });
}

int es_frame_queue(es_frame *fr, long f, const es_frame_view *source, int sx, int sy, int source_cambi,
                   const es_frame_view *encodes, const int *ex, const int *ey, void *stream)
{
    return guarded([&] {
        require(fr != nullptr && source != nullptr && encodes != nullptr, "es_frame_queue: NULL argument");
        fr->views[0] = *source;
        fr->crops[0] = sx;
        fr->crops[1] = sy;
        for (int e = 0; e < fr->nenc; e++) {
            fr->views[1 + e] = encodes[e];
            fr->crops[2 + 2 * e] = ex ? ex[e] : 0;
            fr->crops[3 + 2 * e] = ey ? ey[e] : 0;
        }
        pass(es_batch_queue(fr->batch, f, fr->views.data(), fr->crops.data(), &source_cambi, stream));
    });
}

int es_frame_collect(es_frame *fr, long f, const double *cached_source_cambi, es_accum *const *frame_acc,
                     es_accum *const *centre_acc, es_frame_result *out)
{
    return guarded([&] {
        require(fr != nullptr, "es_frame_collect: NULL frame");
        pass(es_batch_collect(fr->batch, f, cached_source_cambi, frame_acc, centre_acc, out));
    });
}

int es_frame_read_windows(es_frame *fr, int encode, float *stats, float *persist)
{
    return guarded([&] {
        require(fr != nullptr, "es_frame_read_windows: NULL frame");
        pass(es_batch_read_windows(fr->batch, 0, encode, stats, persist));
    });
}

int es_frame_luma(const es_frame *fr, int p, long f, uint64_t *address)
{
    return guarded([&] {
        require(fr != nullptr && address != nullptr, "es_frame_luma: NULL argument");
        pass(es_batch_luma(fr->batch, p, f, address));
    });
}

int es_to_pictures(const es_picture_copy *copies, int n, void *stream)
{
    return guarded([&] {
        require(copies != nullptr && n >= 1 && n <= kPictureMaxJobs, "es_to_pictures: 1 to 64 copies");
        PictureBatch pb{};
        for (int i = 0; i < n; i++) {
            const es_picture_copy &c = copies[i];
            require(c.src != 0 && c.dst != 0, "es_to_pictures: NULL plane or picture");
            require(c.w > 0 && c.h > 0, "es_to_pictures: empty plane");
            require(c.bytes == 1 || c.bytes == 2, "es_to_pictures: samples must be 1 or 2 bytes");
            require(c.pitch >= c.w * c.bytes, "es_to_pictures: pitch is smaller than a row");
            pb.job[pb.njobs++] = PictureJob{(const uint16_t *)c.src, (void *)c.dst, c.w, c.h, c.pitch, c.bytes, 0};
        }
        cuda_check(launch_to_pictures(pb, (cudaStream_t)stream), "copying pictures");
    });
}

void es_frame_destroy(es_frame *fr) { delete fr; }

}  // extern "C"
