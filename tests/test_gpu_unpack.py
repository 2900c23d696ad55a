"""Frame unpacking at the alignments where its loads and stores change form: every sample layout, crops that start off a
multiple of 8 pixels, widths that are multiples of 8, 4 and 2 only, and pitches that keep rows 16-, 4- or 2-byte aligned.
The luma planes are compared whole, the chroma through its exact squared errors and color sums."""

import numpy as np
import pytest

import es_b200
import oracle

pytestmark = pytest.mark.gpu


def planes(rng, fmt, w, h, x0, y0, extra):
    """(stored planes, view arguments, (y, u, v) of the crop as plain samples) of a frame of random samples."""
    size = 1 if fmt in ("planar8", "nv12") else 2
    depth = 8 if size == 1 else 10
    shift = 6 if fmt == "p010" else 0
    fw, fh = x0 + w + 2 * extra, y0 + h
    dt = np.uint8 if size == 1 else np.uint16
    y = (rng.integers(0, 1 << depth, (fh, fw)) << shift).astype(dt)
    u, v = ((rng.integers(0, 1 << depth, (fh // 2, fw // 2)) << shift).astype(dt) for _ in range(2))
    crop = (y[y0:y0 + h, x0:x0 + w] >> shift, u[y0 // 2:(y0 + h) // 2, x0 // 2:(x0 + w) // 2] >> shift,
            v[y0 // 2:(y0 + h) // 2, x0 // 2:(x0 + w) // 2] >> shift)
    semi = fmt in ("nv12", "p010")
    stored = [y, np.stack((u, v), axis=2).reshape(fh // 2, -1)] if semi else [y, u, v]
    return stored, (semi, size, shift, depth), crop


@pytest.mark.parametrize("fmt", ["planar8", "planar16", "nv12", "p010"])
@pytest.mark.parametrize("w,x0,extra", [(64, 0, 0), (64, 8, 4), (68, 2, 1), (66, 4, 0), (16, 6, 3), (130, 0, 7)])
@pytest.mark.parametrize("pd", [8, 10])
def test_unpacked_planes(cuda, module, fmt, w, x0, extra, pd):
    h, y0 = 34, 2
    rng = np.random.default_rng(w + x0 + 7 * extra + pd)
    if pd == 8 and fmt in ("planar16", "p010"):
        pytest.skip("a 10-bit frame needs the 10-bit pipeline")
    keep, views, crops = [], [], []
    for _ in range(2):
        stored, (semi, size, shift, depth), crop = planes(rng, fmt, w, h, x0, y0, extra)
        t = [cuda.from_numpy(a.view(np.uint8 if size == 1 else np.int16)).cuda() for a in stored]
        keep.append(t)
        views.append(es_b200.FrameView(t[0].data_ptr(), t[1].data_ptr(), t[-1].data_ptr(), t[0].stride(0) * size, t[1].stride(0) * size, int(semi),
                                       size, shift, depth))
        crops.append([p.astype(np.uint16) << (pd - depth) for p in crop])
    fr = es_b200.Frame(module, w, h, pd, 1)
    fr.queue(0, views[0], views[1:], cuda.cuda.current_stream().cuda_stream, sx=x0, sy=y0, ex=[x0], ey=[y0])
    res = fr.collect(0, None, None)[0]
    for p in range(2):
        back = cuda.zeros((h, w), dtype=cuda.int16, device="cuda")
        es_b200.to_pictures([(fr.luma(p, 0), back.data_ptr(), w, h, 2 * w, 2)])
        got = back.cpu().numpy().view(np.uint16)
        assert np.array_equal(got, crops[p][0]), p
    fr.close()
    for k in range(3):
        sse = oracle.plane_sse(crops[0][k], crops[1][k])
        assert res.psnr[k] == oracle.psnr(sse, crops[0][k].size, pd), k
    for got, crop in ((res.color_source, crops[0]), (res.color_encode, crops[1])):
        u, v = (c.astype(np.float64) * (1 << (10 - pd)) for c in crop[1:])
        assert got[0] == u.sum() / u.size and got[1] == v.sum() / v.size
        assert abs(got[2] - np.hypot(u - 512, v - 512).mean()) < 1e-6
