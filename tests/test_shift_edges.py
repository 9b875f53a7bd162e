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


@pytest.mark.parametrize("head", [0, 2, 4, 6])
@pytest.mark.parametrize("n,c,hw,ch", [(1, 16, 25, 4), (2, 9, 49, 4), (1, 9, 15, 8), (3, 16, 12, 4), (1, 3, 3, 8), (2, 24, 1, 4)])
def test_unaligned_words_stay_inside_the_input(wino, n, c, hw, ch, head):
    """Items of unaligned quads load the 8-byte words around their pixels except
    where item_at_edge says that one may reach outside the input; few do."""
    total, plane, edges, items = 2 * n * c * hw, 2 * hw, 0, 0
    for img in range(n):
        for c0 in range(0, c, ch):
            for i0 in range(0, hw, 4):
                o = (img * c + c0) * plane + 2 * i0
                items += 1
                if wino.lib().wino_shift_item_at_edge(o, head, total, plane, ch):
                    edges += 1
                    continue
                for e in range(min(ch, c - c0)):
                    at = head + o + e * plane
                    first = at & ~7
                    last = first + (16 if (at >> 1 & 3) + min(4, hw - i0) > 4 else 8)
                    assert first >= head and last <= head + total
    assert edges <= 3 * ch + 4 or edges < items // 4
    # products past 32 bits saturate
    assert wino.lib().wino_shift_item_at_edge(0, 0, 2 ** 32 - 2, 2 ** 31 - 2, 4)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", [(3, 9, 5, 5, 24, 3, 3, 1, 1, 1), (2, 16, 12, 10, 32, 3, 3, 1, 1, 1),
                                   (2, 18, 7, 9, 24, 1, 1, 1, 0, 0), (2, 17, 15, 15, 24, 3, 3, 2, 1, 1),
                                   (1, 19, 1, 1, 16, 3, 3, 1, 1, 1), (3, 24, 2, 1, 16, 2, 1, 1, 0, 0)])
def test_first_and_last_pixels_of_an_unaligned_input(wino, cuda, shape, shift):
    """`shift` elements off an 8-byte word, with NaN on both sides."""
    import torch
    n, c, h, w, k, r, s, stride, p, q = shape
    gen = torch.Generator(device=cuda).manual_seed(sum(shape) + shift)
    room = torch.full((n * c * h * w + 16,), float("nan"), device=cuda, dtype=torch.float16)
    x = room[4 + shift:][:n * c * h * w].view(n, c, h, w)
    x.copy_(torch.randn(x.shape, device=cuda, generator=gen))
    wt = (torch.randn((k, c, r, s), device=cuda, generator=gen) / (c * r * s) ** 0.5).half()
    for cg in (1, 2):
        base._check(base._conv(wino, x, wt, stride, p, q, cg), x, wt, stride, p, q)


@pytest.mark.gpu
@pytest.mark.parametrize("n,c,h,w,k", [(8, 128, 28, 28, 128), (16, 128, 15, 15, 144)])
def test_unaligned_input_through_the_entry_points(wino, cuda, n, c, h, w, k):
    """x one element into its allocation: drop-in, fused conv, epilogue, batch."""
    import torch
    xa, wt, bias, res = base._fused_case(cuda, (n, c, h, w, k), 11)
    x = torch.full((xa.numel() + 16,), float("nan"), device=cuda, dtype=torch.float16)[1:][:xa.numel()].view(xa.shape)
    x.copy_(xa)
    ref = torch.nn.functional.conv2d(xa.double(), wt.double(), padding=1)
    u = wino.filter_transform(wt)
    ws = torch.empty(wino.fused_conv_workspace_bytes(n, c, h, w, k), dtype=torch.uint8, device=cuda)
    y = torch.empty_like(res)
    b = wino.Batch()
    b.add(x, u, k, y, workspace=ws)
    b.run()
    fused = wino.conv2d_fused(x, u, k)
    epi = wino.conv2d_fused_epilogue(x, u, k, bias=bias, residual=res, relu=True)
    base._check(wino.dropin_conv2d(x, wt), xa, wt, 1, 1, 1)
    assert torch.equal(y, fused)
    b.close()
    assert float((fused.double() - ref).norm() / ref.norm()) <= base.FUSED_REL
    ref = torch.relu(ref + bias.double().view(1, -1, 1, 1) + res.double())
    assert float((epi.double() - ref).norm() / ref.norm()) <= base.FUSED_REL
    assert wino.error_read_clear() == 0
