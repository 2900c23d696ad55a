"""The window-energy oracle of the precision study (oracle/precision.py) on the CPU, pinned on 16 x 16 windows to the
C oracle of the reference's window figures (es_oracle.c, exact integer numerators rounded once to float)."""

import numpy as np

import es_synth
import oracle
import precision


def test_16_pixel_windows_equal_the_c_oracle():
    step = es_synth.c4_step(0, w=208, h=144)
    yr, yd = step.source.y, step.encodes[0].y
    _, want = oracle.window_stats(yr, yd, 0)
    got = precision.window_figures(yr, yd, 0, 16).astype(np.float32)
    assert np.array_equal(got[:, :6], want[:, :6])
    # oriented: same exact sums, the square root's operand grouped differently: within one float step
    assert np.allclose(got[:, 6:], want[:, 6:], rtol=2 ** -23, atol=0)


def test_larger_windows_sum_the_16_pixel_numerators():
    step = es_synth.c4_step(1, w=256, h=192)
    yr, yd = step.source.y, step.encodes[0].y
    f16 = precision.window_figures(yr, yd, 0, 16)
    f64 = precision.window_figures(yr, yd, 0, 64)
    # the first six figures are sums: a 64-pixel window is the sum of its 16 blocks (exact in int64, one rounding)
    b = f16[:, :6].reshape(12, 16, 6)
    blocks = b.reshape(3, 4, 4, 4, 6).transpose(0, 2, 1, 3, 4).reshape(3 * 4, 16, 6).sum(axis=1)
    assert np.allclose(f64[:, :6], blocks, rtol=1e-12)


def test_fp32_forms_reduce_to_the_exact_ones_where_nothing_rounds():
    """On a small picture of values that are multiples of 81 every term is a whole number and every sum below 2^24, so the
    restated FP32 forms have to give the exact figures (the oriented ones up to their last rounding)."""
    rng = np.random.default_rng(3)
    yr, yd = (81 * rng.integers(0, 3, (33, 49)) for _ in range(2))
    want = precision.window_figures(yr, yd, 0, 16)
    for mode in (1, 2):
        got = precision.fp32_window_figures(yr, yd, 0, 16, mode)
        assert np.allclose(got, want, rtol=2 ** -21, atol=0), mode


def test_quotients_by_9_and_81_from_a_reciprocal_are_correctly_rounded():
    """q = x r with r = 1 / b rounded, then q + r (x - b q) in fused multiply-adds, as the window kernels divide: equal to
    FP32 division for every significand of x (the exponent changes nothing away from underflow). The remainder fits 53
    bits and its product with r, added to q, 64, so both fused steps are rounded once here too."""
    x = np.arange(1 << 23, 1 << 24, dtype=np.int64).astype(np.float32)
    for b in (np.float32(9), np.float32(81)):
        r = np.float32(1) / b
        q = x * r
        rem = (x.astype(np.float64) - np.float64(b) * q.astype(np.float64)).astype(np.float32)
        got = (rem.astype(np.longdouble) * np.longdouble(r) + q.astype(np.longdouble)).astype(np.float32)
        assert np.array_equal(got, x / b)
