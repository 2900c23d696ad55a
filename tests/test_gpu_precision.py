"""Texture window energies on larger windows (es_windows_*) against the FP64 oracle (oracle/precision.py): the integer
summed-area tables give every figure exactly (bit-equal doubles); compensated FP32 stays within 1e-5 relative; plain
FP32 is reported by its error, which the compensation must not exceed. Windows of 16, 32 and 64 pixels, 10- and 8-bit."""

import numpy as np
import pytest

import es_b200
import es_synth
import precision
from gpu_util import from_dev, to_dev, zeros_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,depth", [(224, 160, 10), (200, 130, 8)])
def test_window_energies_in_three_arithmetics(cuda, module, w, h, depth):
    step = es_synth.c4_step(0, w=w, h=h) if depth == 10 else es_synth.c1_step(0, w=w, h=h)
    yr, yd = step.source.y, step.encodes[0].y
    up = 10 - depth
    win = es_b200.Windows(w, h)
    r, d = to_dev(cuda, yr), to_dev(cuda, yd)
    win.compute(r.data_ptr(), d.data_ptr(), up)
    for window in (16, 32, 64):
        want = precision.window_figures(yr, yd, up, window)
        n = want.shape[0]
        outs = []
        for mode in range(3):
            o = zeros_dev(cuda, (max(n, 1), 8), np.float64)
            win.figures(window, mode, o.data_ptr())
            outs.append(from_dev(o, np.float64)[:n])
        assert np.array_equal(outs[0], want), window
        scale = np.maximum(np.abs(want), 1e-3 * np.abs(want).max(axis=0, keepdims=True))
        rel_c = np.abs(outs[1] - want) / scale
        rel_p = np.abs(outs[2] - want) / scale
        assert rel_c.max() <= 1e-5, (window, rel_c.max())
        assert rel_c.max() <= rel_p.max() + 1e-12
    win.close()


@pytest.mark.parametrize("w,h", [(16, 16), (65, 33), (130, 63), (64, 96), (191, 32), (16, 16400)])
def test_sizes_around_the_table_bands_and_chunks(cuda, module, w, h):
    """The tables are scanned in bands of 32 rows and chunks of 64 columns, blocks of 16 x 16 read 25 entries a side, and
    pictures of more than 16384 rows take another path: the exact form equals the oracle's, the compensated form stays
    within 1e-5 of it."""
    rng = np.random.default_rng(w + h)
    yy, xx = np.mgrid[0:h, 0:w]
    yr = np.clip(700 + 200 * np.sin(xx / 9 + yy / 23) + rng.normal(0, 20, (h, w)), 0, 1023).astype(np.uint16)
    yd = np.clip(yr + rng.normal(0, 8, (h, w)), 0, 1023).astype(np.uint16)
    win = es_b200.Windows(w, h)
    r, d = to_dev(cuda, yr), to_dev(cuda, yd)
    win.compute(r.data_ptr(), d.data_ptr(), 0)
    for window in (16, 32):
        n = (w // window) * (h // window)
        if not n:
            continue
        want = precision.window_figures(yr, yd, 0, window)
        outs = []
        for mode in range(2):
            o = zeros_dev(cuda, (n, 8), np.float64)
            win.figures(window, mode, o.data_ptr())
            outs.append(from_dev(o, np.float64))
        assert np.array_equal(outs[0], want), window
        scale = np.maximum(np.abs(want), 1e-3 * np.abs(want).max(axis=0, keepdims=True))
        assert (np.abs(outs[1] - want) / scale).max() <= 1e-5
    win.close()


@pytest.mark.parametrize("w,h,depth", [(16, 16, 10), (65, 33, 10), (130, 63, 8), (208, 144, 10), (191, 32, 8), (16, 16400, 10), (50, 16385, 10)])
def test_fp32_figures_bit_for_bit(cuda, module, w, h, depth):
    """The roundings of the FP32 forms are what the study is about: the compensated and the plain figures equal a
    restatement that adds, multiplies and divides in FP32 in the same order, with whole and partial bands and chunks of the
    tables and on both sides of the 16384 rows where their kernels change."""
    rng = np.random.default_rng(w + h)
    yy, xx = np.mgrid[0:h, 0:w]
    top = 1023 if depth == 10 else 255
    yr = np.clip(top * (0.65 + 0.2 * np.sin(xx / 9 + yy / 23)) + rng.normal(0, top / 50, (h, w)), 0, top).astype(np.uint16)
    yd = np.clip(yr + rng.normal(0, top / 100, (h, w)), 0, top).astype(np.uint16)
    up = 10 - depth
    win = es_b200.Windows(w, h)
    r, d = to_dev(cuda, yr), to_dev(cuda, yd)
    win.compute(r.data_ptr(), d.data_ptr(), up)
    for window in (16, 32, 48):
        n = (w // window) * (h // window)
        if not n:
            continue
        for mode in (1, 2):
            o = zeros_dev(cuda, (n, 8), np.float64)
            win.figures(window, mode, o.data_ptr())
            assert np.array_equal(from_dev(o, np.float64), precision.fp32_window_figures(yr, yd, up, window, mode)), (window, mode)
    win.close()
