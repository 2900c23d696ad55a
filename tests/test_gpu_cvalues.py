"""The c-value kernel at the sizes where its tiles, windows and ranks change form, bit for bit against the CPU oracle:
every number of k-steps a window reaches (pads 0 to 64, from staged regions that start at and off a multiple of 8),
rows that allow 16-, 4- and 2-byte loads, pictures one pixel past a tile, tiles whose codes need several passes or
several segments, and the top-k selection over lists that hold zeros."""

import numpy as np
import pytest

import es_b200
import oracle
from gpu_util import from_dev, to_dev, zeros_dev
from test_gpu_cambi import banded, oracle_params, plateaus

pytestmark = pytest.mark.gpu


def check(torch, module, img, pad, topk=None):
    h, w = img.shape
    p = es_b200.derive_params(w, h)
    p.pad, p.window = pad, 2 * pad + 1
    if topk is not None:
        p.topk = topk
    cam = es_b200.Cambi(module, w, h, 10, p)
    planes = [zeros_dev(torch, (sh, sw), np.float32) for sw, sh in oracle.scale_sizes(w, h)]
    cam.set_cvalue_planes([t.data_ptr() for t in planes])
    d = to_dev(torch, img)
    cam.launch(d.data_ptr(), w, torch.cuda.current_stream().cuda_stream)
    score = cam.finish()
    want = oracle.cambi(img, 10, oracle_params(p), keep=True)
    for s in range(oracle.SCALES):
        assert np.array_equal(from_dev(planes[s], np.float32).view(np.uint32), want.cvalues[s].view(np.uint32)), f"scale {s} c-values"
    pooled, sums, counts = cam.scale_stats()
    cam.close()
    assert sums == want.sums_fx and counts == want.counts and pooled == want.pooled and score == want.score
    return counts


@pytest.mark.parametrize("pad", [0, 1, 8, 15, 16, 17, 32, 33, 47, 48, 49, 64])
def test_windows_of_every_k_step_count(cuda, module, pad):
    counts = check(cuda, module, banded(200, 136, 20 + pad, step=2), pad)
    assert pad == 0 or counts[0] > 0


@pytest.mark.parametrize("w,h", [(128, 64), (129, 65), (130, 66), (136, 80), (65, 129), (1, 40), (40, 1)])
def test_widths_and_heights_around_a_tile(cuda, module, w, h):
    if min(w, h) < 2:
        with pytest.raises(es_b200.EsError):
            es_b200.Cambi(module, w, h, 10)
        return
    check(cuda, module, banded(w, h, 3 * w + h, step=1), 9)


@pytest.mark.parametrize("lo,hi,step", [(60, 330, 1), (53, 563, 1), (500, 600, 1), (60, 560, 4), (60, 560, 5)])
def test_code_ranges_of_several_passes_and_segments(cuda, module, lo, hi, step):
    """Steep gradients: a 64 x 64 tile spans up to the whole band, with neighbours 1 or 4 codes apart, or none (5)."""
    yy, xx = np.mgrid[0:72, 0:128]
    img = (np.round((lo + (hi - lo) * ((xx // 2) * 2 + 0.4 * ((yy // 8) * 8)) / 155) / step) * step).astype(np.uint16)
    counts = check(cuda, module, img, 32)
    assert (step == 5) or counts[0] > 0


@pytest.mark.parametrize("topk", [0.02, 0.3])
def test_top_k_over_lists_with_zeros(cuda, module, topk):
    """More than k positive values among rows that also hold zeros, from tiles of one and of several segments."""
    img = np.concatenate([plateaus(256, 128, size=8), banded(256, 96, 5, step=2)])
    counts = check(cuda, module, img, 32, topk)
    assert counts[0] > int(topk * 256 * 224)
