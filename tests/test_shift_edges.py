"""Edges of the shift-reuse implicit GEMM (shift_conv.cuh) that its plan has to
get right for any filter, stride and padding it accepts.

CPU: the pixel quads a producer group owns reach every pixel of every tile, over
random problems.  GPU: against FP64, with the tolerances of test_shift_conv.
"""
import ctypes
import random

import numpy as np
import pytest

import test_shift_conv as base

# stride 2, no padding, an even filter height and odd H: image rows that no
# output reads, several images a tile
UNREAD_ROWS = [
    (12, 32, 7, 7, 48, 2, 2, 2, 0, 0),
    (12, 32, 9, 9, 48, 2, 2, 2, 0, 0),
    (12, 32, 7, 7, 48, 4, 4, 2, 0, 0),
    (5, 32, 15, 15, 48, 2, 2, 2, 0, 0),
]


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", UNREAD_ROWS)
def test_quads_with_unread_image_rows(wino, shape, cg):
    base.test_plan_quads_cover_every_row_once(wino, shape, cg)


@pytest.mark.gpu
@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", UNREAD_ROWS)
def test_conv_with_unread_image_rows(wino, cuda, shape, cg):
    base.test_shift_conv(wino, cuda, shape, cg)


def _random_problem(rng):
    """n, c, h, w, k, r, s, u, v, p, q of a problem the kernel's rules may take."""
    r, s = rng.randint(1, 8), rng.randint(1, 8)
    h, w = int(2 ** rng.uniform(0, 7)), int(2 ** rng.uniform(0, 8.3))
    p, q = rng.randint(0, min(4, r + 1)), rng.randint(0, min(4, s + 1))
    return (rng.randint(1, 40), rng.choice([16, 24, 48, 256]), h, w, rng.choice([16, 64, 144, 512]), r, s,
            rng.choice([1, 2]), rng.choice([1, 2]), p, q)


def _quads_needed(kp, g, pt):
    """Quads from a tile's first to the last that holds a pixel of its rows."""
    n, h, w, r, s, u, v, p, q = (getattr(kp, f) for f in ("n", "h", "w", "r", "s", "u", "v", "p", "q"))
    gx_, gy_ = g["GX"], g["GY"]
    line = pt * 128 // gx_
    n0, gy0 = line // gy_, line % gy_
    lo = (gy0 * u - p) * w + (min(max(pt * 128 - line * gx_ - q, 0), w) if u == v == 1 else 0)
    first = n0 * g["qpi"] + (min(max(lo, 0), h * w) >> 2)
    need = 0
    for a in range(g["nu"]):
        for b in range(g["nv"]):
            pos = pt * 128 + np.arange(128 + (r - 1 - a) // u * gx_ + (s - 1 - b) // v)
            im, rem = pos // (gx_ * gy_), pos % (gx_ * gy_)
            y, x = rem // gx_ * u + a - p, rem % gx_ * v + b - q
            quad = (im * g["qpi"] + (y * w + x) // 4)[(im < n) & (y >= 0) & (y < h) & (x >= 0) & (x < w)] - first
            if quad.size:
                assert quad.min() >= 0
                need = max(need, int(quad.max()) + 1)
    return need


@pytest.mark.parametrize("seed", range(4))
def test_quads_of_random_problems(wino, seed):
    L, rng, taken = wino.lib(), random.Random(seed), 0
    while taken < 150:
        kp = base._Param()
        for f, x in zip(("n", "c", "h", "w", "k", "r", "s", "u", "v", "p", "q"), _random_problem(rng)):
            setattr(kp, f, x)
        if kp.h + 2 * kp.p < kp.r or kp.w + 2 * kp.q < kp.s:
            continue
        kp.Oh, kp.Ow = (kp.h - kp.r + 2 * kp.p) // kp.u + 1, (kp.w - kp.s + 2 * kp.q) // kp.v + 1
        if L.wino_shift_cg(ctypes.byref(kp)) == 0:
            continue
        taken += 1
        for cg in (1, 2):
            g = base._plan(L, kp, cg)
            tiles = -(-(((kp.n - 1) * g["GY"] + kp.Oh - 1) * g["GX"] + kp.Ow) // 128)
            for pt in {0, 1, tiles - 1} | {rng.randrange(tiles) for _ in range(12)}:
                if pt < tiles:
                    assert _quads_needed(kp, g, pt) <= g["qmax"], [getattr(kp, f) for f, _ in kp._fields_[6:]]
