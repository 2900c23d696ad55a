"""TEST INFRASTRUCTURE, not product code: the FP64 oracle of the texture window energies on windows of 16 k pixels.

Definitions of src/kernels.cu:346-428 and reference/encode_score/compare.py:77-108 (fine = y - box3, mid = box3 - box9,
box-3 gradients by central differences, 0 on the border columns / rows; edge pixels repeated for the boxes), evaluated
exactly in int64 numerators (fine and gradients x 9, mid x 81) and rounded once per figure to float64, in the
operation order of the CUDA exact mode. Only tests and the precision report import this module.
"""

from __future__ import annotations

import numpy as np


def _box(y: np.ndarray, r: int) -> np.ndarray:
    p = np.pad(y.astype(np.int64), r, mode="edge")
    c = np.cumsum(np.cumsum(p, axis=0), axis=1)
    c = np.pad(c, ((1, 0), (1, 0)))
    n = 2 * r + 1
    h, w = y.shape
    return c[n:n + h, n:n + w] - c[0:h, n:n + w] - c[n:n + h, 0:w] + c[0:h, 0:w]


def terms(y: np.ndarray, up: int):
    """Exact numerators (fine x 9, mid x 81, gx x 9, gy x 9) of every pixel of y (values << up)."""
    v = y.astype(np.int64) << up
    s3, s9 = _box(v, 1), _box(v, 4)
    f = 9 * v - s3
    m = 9 * s3 - s9
    gx = np.zeros_like(v)
    gy = np.zeros_like(v)
    gx[:, 1:-1] = s3[:, 2:] - s3[:, :-2]
    gy[1:-1, :] = s3[2:, :] - s3[:-2, :]
    return f, m, gx, gy


def window_figures(yr: np.ndarray, yd: np.ndarray, up: int, window: int) -> np.ndarray:
    """(windows, 8) float64: [src fine^2, src mid^2, enc fine^2, enc mid^2, fine x, mid x, src oriented, enc oriented],
    windows row by row, only whole windows of the 16 x 16 block grid."""
    fr, mr, gxr, gyr = terms(yr, up)
    fd, md, gxd, gyd = terms(yd, up)
    h, w = yr.shape
    k = window // 16
    bw, bh = w // 16, h // 16
    ww, wh = bw // k, bh // k
    H, W = wh * window, ww * window
    q = [fr * fr, mr * mr, fd * fd, md * md, fr * fd, mr * md, gxr * gxr, gyr * gyr, gxr * gyr, gxd * gxd, gyd * gyd, gxd * gyd]
    s = [a[:H, :W].reshape(wh, window, ww, window).sum(axis=(1, 3)).reshape(-1) for a in q]
    out = np.zeros((ww * wh, 8), np.float64)
    out[:, 0] = s[0].astype(np.float64) / 81.0
    out[:, 1] = s[1].astype(np.float64) / 6561.0
    out[:, 2] = s[2].astype(np.float64) / 81.0
    out[:, 3] = s[3].astype(np.float64) / 6561.0
    out[:, 4] = s[4].astype(np.float64) / 81.0
    out[:, 5] = s[5].astype(np.float64) / 6561.0
    dr, xr = (s[6] - s[7]).astype(np.float64), s[8].astype(np.float64)
    dd, xd = (s[9] - s[10]).astype(np.float64), s[11].astype(np.float64)
    out[:, 6] = np.sqrt(dr * dr + 4.0 * xr * xr) / 81.0
    out[:, 7] = np.sqrt(dd * dd + 4.0 * xd * xd) / 81.0
    return out


# ---- the FP32 forms, rounding by rounding ------------------------------------------------------------------------------
F = np.float32


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


class _Comp:
    """Neumaier's accumulator, element by element."""

    def __init__(self, shape):
        self.s, self.c = np.zeros(shape, F), np.zeros(shape, F)

    def add(self, x):
        self.s, e = _two_sum(self.s, x)
        self.c = self.c + e

    def value(self):
        return self.s + self.c


def fp32_tables(v: np.ndarray):
    """(hi, lo, plain): the summed-area tables of integer values v in compensated and plain FP32, each entry the row chain
    of column chains of additions, in order."""
    h, w = v.shape
    cols = [np.zeros((h, w), F) for _ in range(3)]
    hi, lo, p = np.zeros(w, F), np.zeros(w, F), np.zeros(w, F)
    for r in range(h):
        x = v[r].astype(F)
        hi, e = _two_sum(hi, x)
        lo = lo + e
        p = p + x
        for c, a in zip(cols, (hi, lo, p)):
            c[r] = a
    hi, lo, p = np.zeros(h, F), np.zeros(h, F), np.zeros(h, F)
    for x in range(w):
        hi, e = _two_sum(hi, cols[0][:, x])
        lo = (lo + e) + cols[1][:, x]
        p = p + cols[2][:, x]
        for c, a in zip(cols, (hi, lo, p)):
            c[:, x] = a
    return cols


def _fp32_box(v: np.ndarray, tables, r: int):
    """(compensated, plain) box sums of side 2 r + 1: inside the picture the table's four corners in their order, near an
    edge the sum of the clamped pixels, which FP32 adds exactly."""
    h, w = v.shape
    c = _box(v, r).astype(F)
    p = c.copy()
    if h > 2 * r and w > 2 * r:
        hi, lo, pl = (np.pad(t, ((1, 0), (1, 0))) for t in tables)  # entries left of and above the picture are 0
        n = 2 * r + 1

        def corner(t, down, right):
            return t[n if down else 0:, n if right else 0:][:h - 2 * r, :w - 2 * r]

        ch, cl, cp = corner(hi, 1, 1), corner(lo, 1, 1), corner(pl, 1, 1)
        for down, right, sign in ((1, 0, F(-1)), (0, 1, F(-1)), (0, 0, F(1))):
            ch, e = _two_sum(ch, sign * corner(hi, down, right))
            cl = (cl + e) + sign * corner(lo, down, right)
            cp = cp + sign * corner(pl, down, right)
        c[r:h - r, r:w - r] = ch + cl
        p[r:h - r, r:w - r] = cp
    return c, p


def fp32_window_figures(yr: np.ndarray, yd: np.ndarray, up: int, window: int, mode: int) -> np.ndarray:
    """The figures of window_figures in the compensated (mode 1) or plain (mode 2) FP32 form, every addition, product and
    division rounded where the CUDA kernels round it and summed in their order."""
    terms32 = []
    for y in (yr, yd):
        v = y.astype(np.int64) << up
        tables = fp32_tables(v)
        (c3, p3), (c9, p9) = _fp32_box(v, tables, 1), _fp32_box(v, tables, 4)
        x = v.astype(F)
        if mode == 1:
            s, f, m = c3, (F(9) * x - c3) / F(9), (F(9) * c3 - c9) / F(81)
        else:
            s = p3 / F(9)
            f, m = x - s, s - p9 / F(81)
        gx, gy = np.zeros_like(s), np.zeros_like(s)
        gx[:, 1:-1] = s[:, 2:] - s[:, :-2]
        gy[1:-1] = s[2:] - s[:-2]
        terms32.append((f, m, gx, gy))
    (fr, mr, xr, yr_), (fd, md, xd, yd_) = terms32
    q = [fr * fr, mr * mr, fd * fd, md * md, fr * fd, mr * md]
    for gx, gy in ((xr, yr_), (xd, yd_)):
        if mode == 1:
            q += [((gx - gy) * (gx + gy)) / F(81), np.zeros_like(gx), (gx * gy) / F(81)]
        else:
            q += [gx * gx, gy * gy, gx * gy]
    h, w = yr.shape
    bh, bw = h // 16, w // 16
    # a 16 x 16 block: 8 warps of two rows, each a butterfly over its 32 lanes, then the warps in order
    q = np.stack([a[:16 * bh, :16 * bw].reshape(bh, 8, 2, bw, 16).transpose(0, 3, 1, 2, 4).reshape(bh, bw, 8, 32) for a in q])
    s, e = q, np.zeros_like(q)
    while s.shape[-1] > 1:
        n = s.shape[-1] // 2
        if mode == 1:
            t, err = _two_sum(s[..., :n], s[..., n:])
            s, e = t, (e[..., :n] + e[..., n:]) + err
        else:
            s = s[..., :n] + s[..., n:]
    warps = (s + e)[..., 0] if mode == 1 else s[..., 0]

    def total(parts):  # of arrays, in order
        if mode == 1:
            acc = _Comp(parts[0].shape)
            for x in parts:
                acc.add(x)
            return acc.value()
        acc = np.zeros(parts[0].shape, F)
        for x in parts:
            acc = acc + x
        return acc

    blocks = total([warps[..., k] for k in range(8)])
    k = window // 16
    wh, ww = bh // k, bw // k
    t = total([blocks[:, by:wh * k:k, bx:ww * k:k] for by in range(k) for bx in range(k)]).reshape(12, -1)
    out = np.zeros((ww * wh, 8), np.float64)
    for g in range(6):
        out[:, g] = t[g]
    for g, o in ((6, 6), (7, 9)):
        d = t[o] if mode == 1 else t[o] - t[o + 1]
        out[:, g] = np.sqrt(d * d + F(4) * (t[o + 2] * t[o + 2]))
    return out
