"""The shift-reuse implicit GEMM (shift_conv.cuh), the drop-in's kernel for
problems of 64 MFLOP and more.

CPU: the plan's position grid, operand rows and weight operand against their
definitions (every tap of every output reads the right input element or a
zero; the pixel quads cover every operand row once).  GPU: both schedules (one
CTA and a pair of CTAs a unit) against FP64.  The kernel accumulates in fp32
and rounds y once: the rounding alone is a relative error of 2^-11 / sqrt(3) =
2.8e-4 at worst in the 2-norm, and 2^-11 = 4.9e-4 of the largest output.
"""
import ctypes

import numpy as np
import pytest

REL_L2 = 3e-4
MAX_NORM = 5.5e-4

# n, c, h, w, k, r, s, stride, p, q
SHAPES = [
    (1, 16, 5, 5, 16, 3, 3, 1, 1, 1),        # one tile, one K-step a tap
    (2, 32, 12, 10, 32, 3, 3, 1, 1, 1),      # even rows: paired stores
    (3, 48, 9, 7, 144, 3, 3, 1, 1, 1),       # odd H * W (unaligned quads), K past 128
    (4, 24, 30, 2, 24, 3, 3, 1, 1, 1),       # rows narrower than a quad, ragged C and K
    (33, 24, 2, 2, 24, 3, 3, 1, 1, 1),       # many images a tile
    (9, 40, 3, 3, 24, 3, 3, 1, 1, 1),
    (1, 16, 1, 1, 16, 3, 3, 1, 1, 1),        # one pixel
    (2, 16, 60, 224, 32, 3, 3, 1, 1, 1),     # long rows: three items a producer
    (2, 64, 33, 57, 272, 3, 3, 1, 1, 1),     # two weight blocks, the last short
    (2, 256, 28, 28, 256, 3, 3, 1, 1, 1),    # the ring of stages wraps
    (16, 64, 56, 56, 64, 3, 3, 1, 1, 1),     # several units a CTA: both accumulators
    (3, 64, 14, 14, 320, 3, 3, 2, 1, 1),     # stride 2: four planes
    (2, 64, 112, 112, 64, 3, 3, 2, 1, 1),
    (3, 32, 7, 7, 48, 1, 3, 1, 0, 1),        # 1x3
    (2, 48, 10, 12, 24, 5, 5, 1, 2, 2),      # 25 taps
    (24, 32, 56, 56, 256, 5, 5, 1, 2, 2),    # a ring of two stages, two a unit
    (2, 32, 9, 11, 48, 2, 2, 1, 0, 0),       # two 16-channel blocks a stage
    (3, 96, 10, 14, 40, 1, 1, 1, 0, 0),      # 1x1: the grid has no padding
    (3, 72, 7, 9, 40, 1, 1, 1, 0, 0),
    (2, 64, 15, 15, 64, 3, 3, 2, 1, 1),      # stride 2, unaligned quads
    (1, 32, 14, 126, 32, 3, 3, 2, 1, 1),     # stride 2, long rows
]


class _Param(ctypes.Structure):
    _fields_ = [(f, ctypes.c_void_p) for f in ("pin", "pweight", "pout", "pinws", "filt", "mid")] + [
        (f, ctypes.c_short) for f in ("n", "c", "h", "w", "k", "r", "s", "u", "v", "p", "q", "Oh", "Ow")]


def _param(shape):
    n, c, h, w, k, r, s, st, p, q = shape
    kp = _Param()
    for f, x in zip(("n", "c", "h", "w", "k", "r", "s", "u", "v", "p", "q"), (n, c, h, w, k, r, s, st, st, p, q)):
        setattr(kp, f, x)
    kp.Oh, kp.Ow = (h - r + 2 * p) // st + 1, (w - s + 2 * q) // st + 1
    return kp


PLAN = ("GX", "GY", "rows", "cps", "nst", "nstage", "stageA", "stageB", "NB", "units", "nu", "nv", "qmax", "qpi")


def _plan(L, kp, cg):
    out = (ctypes.c_int * len(PLAN))()
    L.wino_shift_plan(ctypes.byref(kp), cg, out)
    return dict(zip(PLAN, out))


def _planes(g, r, s, st):
    """(a, b) -> (first operand row, rows) in the stage."""
    out, base = {}, 0
    for a in range(g["nu"]):
        for b in range(g["nv"]):
            rows = 128 + (r - 1 - a) // st * g["GX"] + (s - 1 - b) // st
            out[a, b] = (base, rows)
            base += rows
    assert base == g["rows"]
    return out


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_plan_reads_every_tap(wino, shape, cg):
    n, c, h, w, k, r, s, st, p, q = shape
    L = wino.lib()
    kp = _param(shape)
    assert L.wino_shift_cg(ctypes.byref(kp)) in (1, 2)
    g = _plan(L, kp, cg)
    oh, ow, per = kp.Oh, kp.Ow, g["GX"] * g["GY"]
    assert 2 <= g["nstage"] <= 8 and g["nstage"] * (g["stageA"] + g["stageB"]) <= 225 * 1024
    assert 2 * g["cps"] * g["rows"] * 16 + 16 <= g["stageA"]
    planes = _planes(g, r, s, st)
    x = np.random.default_rng(0).integers(1, 1 << 30, (n, h, w))
    tiles = -(-(((n - 1) * g["GY"] + oh - 1) * g["GX"] + ow) // (128 * cg))
    oy, ox = np.meshgrid(np.arange(oh), np.arange(ow), indexing="ij")
    for (a, b), (base, rows) in planes.items():
        pos = np.arange(tiles * 128 * cg + rows)
        im, rem = pos // per, pos % per
        y, xx = rem // g["GX"] * st + a - p, rem % g["GX"] * st + b - q
        ok = (im < n) & (y >= 0) & (y < h) & (xx >= 0) & (xx < w)
        plane = np.where(ok, x[np.clip(im, 0, n - 1), np.clip(y, 0, h - 1), np.clip(xx, 0, w - 1)], 0)
        for i in range(n):
            at = (i * g["GY"] + oy) * g["GX"] + ox
            for rr in range(a, r, st):
                for ss in range(b, s, st):
                    shift = rr // st * g["GX"] + ss // st
                    assert shift + 128 <= rows
                    yy, cc = oy * st + rr - p, ox * st + ss - q
                    ref = np.where((yy >= 0) & (yy < h) & (cc >= 0) & (cc < w),
                                   x[i][np.clip(yy, 0, h - 1), np.clip(cc, 0, w - 1)], 0)
                    assert np.array_equal(plane[at + shift], ref), (a, b, rr, ss)


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_plan_quads_cover_every_row_once(wino, shape, cg):
    """The producers' pixel quads, as produce() numbers them from a tile's
    first position, reach every operand row that holds a pixel exactly once."""
    n, c, h, w, k, r, s, st, p, q = shape
    g = _plan(wino.lib(), _param(shape), cg)
    planes = _planes(g, r, s, st)
    gx_, gy_, hw = g["GX"], g["GY"], h * w
    kp = _param(shape)
    tiles = -(-(((n - 1) * gy_ + kp.Oh - 1) * gx_ + kp.Ow) // 128)
    for pt in sorted({0, 1, tiles // 2, tiles - 1} & set(range(tiles))):
        line = pt * 128 // gx_
        gx0, n0, gy0 = pt * 128 - line * gx_, line // gy_, line % gy_
        lo = (gy0 * st - p) * w + (min(max(gx0 - q, 0), w) if st == 1 else 0)
        q0 = min(max(lo, 0), hw) >> 2
        got = {}
        for iq in range(g["qmax"]):
            dn, qq = divmod(q0 + iq, g["qpi"])
            for i in range(4 * qq, min(4 * qq + 4, hw)):
                y, x = divmod(i, w)
                a, b = (y + p) % st, (x + q) % st
                gy, gx = (y + p) // st, (x + q) // st
                if n0 + dn >= n or (a, b) not in planes or gx >= gx_ or gy >= gy_:
                    continue
                row = (dn * gy_ + gy - gy0) * gx_ + gx - gx0
                if 0 <= row < planes[a, b][1]:
                    at = planes[a, b][0] + row
                    assert at not in got
                    got[at] = (n0 + dn, y, x)
        for (a, b), (base, rows) in planes.items():
            for row in range(rows):
                t = gx0 + row
                l2 = gy0 + t // gx_
                im, y, x = n0 + l2 // gy_, l2 % gy_ * st + a - p, t % gx_ * st + b - q
                inside = im < n and 0 <= y < h and 0 <= x < w
                assert got.get(base + row) == ((im, y, x) if inside else None)


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_weight_operand_is_a_bijection(wino, shape, cg):
    n, c, h, w, k, r, s, st, p, q = shape
    L = wino.lib()
    kp = _param(shape)
    g = _plan(L, kp, cg)
    L.wino_shift_weight_bytes.restype = ctypes.c_size_t
    total = L.wino_shift_weight_bytes(ctypes.byref(kp), cg)
    nks, k16, nb = (c + 15) // 16 * r * s, (k + 15) // 16 * 16, g["NB"]
    rows = lambda k0: (min(nb, k16 - k0) + 31) // 32 * 32 if cg == 2 else min(nb, k16 - k0)
    last = (k16 - 1) // nb * nb
    assert total == (last + rows(last)) * nks * 32
    at = set()
    for k0 in range(0, k16, nb):
        half = rows(k0) // cg
        assert half % 8 == 0 and rows(k0) % (32 if cg == 2 else 16) == 0
        assert g["cps"] * r * s * half * 32 <= g["stageB"]
        for row in range(rows(k0)):
            rank, rr = divmod(row, half)
            for ks in range(nks):
                for hh in range(2):
                    at.add(((k0 + rank * half) * nks + ks * half) * 32 + (rr >> 3) * 256 + hh * 128 + (rr & 7) * 16)
    assert len(at) * 16 == total and max(at) == total - 16


def _conv(wino, x, w, stride, p, q, cg):
    import torch
    n, c, h, wd = x.shape
    k, _, r, s = w.shape
    oh, ow = (h - r + 2 * p) // stride + 1, (wd - s + 2 * q) // stride + 1
    wop = torch.empty((k + 64) * ((c + 15) // 16) * r * s * 32, dtype=torch.uint8, device=x.device)
    y = torch.full((n, k, oh, ow), float("nan"), dtype=torch.float16, device=x.device)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = wino.lib().wino_conv2d_shift(ptr(x), ptr(w), ptr(wop), ptr(y), n, c, h, wd, k, r, s, stride, stride, p, q, cg,
                                      wino._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert wino.error_read_clear() == 0
    return y


def _check(y, x, w, stride, p, q):
    import torch
    ref = torch.nn.functional.conv2d(x.double(), w.double(), stride=stride, padding=(p, q))
    d = y.double() - ref
    assert float(d.norm() / ref.norm()) <= REL_L2
    assert float(d.abs().max() / ref.abs().max()) <= MAX_NORM


@pytest.mark.gpu
@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_shift_conv(wino, cuda, shape, cg):
    import torch
    n, c, h, w, k, r, s, stride, p, q = shape
    gen = torch.Generator(device=cuda).manual_seed(sum(shape))
    x = torch.randn((n, c, h, w), device=cuda, generator=gen).half()
    wt = (torch.randn((k, c, r, s), device=cuda, generator=gen) / (c * r * s) ** 0.5).half()
    _check(_conv(wino, x, wt, stride, p, q, cg), x, wt, stride, p, q)


# few channels: the filter's columns become channels
FOLDED = [
    (2, 3, 32, 32, 64, 7, 7, 2, 3, 3),       # RGB stem
    (3, 3, 37, 45, 40, 7, 7, 2, 3, 3),       # odd height and width, ragged K
    (2, 3, 64, 60, 96, 7, 7, 2, 3, 3),       # several units
    (1, 3, 9, 8, 16, 7, 7, 2, 3, 3),         # image smaller than the filter's reach
    (3, 5, 20, 17, 24, 3, 3, 1, 1, 1),       # 15 of 16 virtual channels, stride 1
    (2, 8, 15, 15, 32, 3, 3, 2, 1, 1),       # 24 virtual channels
    (2, 4, 12, 18, 16, 2, 5, 1, 0, 2),       # 2x5 filter
    (2, 2, 21, 19, 32, 3, 3, 1, 1, 1),       # one K-step
]


@pytest.mark.gpu
@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("shape", FOLDED)
def test_folded_conv(wino, cuda, shape, cg):
    test_shift_conv(wino, cuda, shape, cg)


@pytest.mark.gpu
def test_dropin_stem(wino, cuda):
    """A stem's operand does not fit transform_filter and goes to
    transform_pin; without one the direct kernel runs."""
    import torch
    gen = torch.Generator(device=cuda).manual_seed(5)
    x = torch.randn((4, 3, 112, 112), device=cuda, generator=gen).half()
    wt = (torch.randn((64, 3, 7, 7), device=cuda, generator=gen) / 12).half()
    for pin in (True, False):
        y = wino.dropin_conv2d(x, wt, transform_pin=pin, stride=2, pad=3)
        torch.cuda.synchronize()
        assert wino.error_read_clear() == 0
        _check(y, x, wt, 2, 3, 3)


@pytest.mark.gpu
def test_shift_conv_unaligned_input(wino, cuda):
    """An input 2 bytes off its allocation takes the unaligned quads."""
    import torch
    gen = torch.Generator(device=cuda).manual_seed(1)
    x = torch.randn(2 * 32 * 12 * 12 + 1, device=cuda, generator=gen).half()[1:].view(2, 32, 12, 12)
    wt = (torch.randn((48, 32, 3, 3), device=cuda, generator=gen) / 17).half()
    _check(_conv(wino, x, wt, 1, 1, 1, 1), x, wt, 1, 1, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,pin", [((64, 256, 14, 14, 256), True),    # hosted by the two-stage route's kernels
                                       ((64, 256, 14, 14, 256), False),   # no transform_pin: its own kernel
                                       ((96, 128, 28, 28, 256), True),    # CTA pairs
                                       ((8, 512, 7, 7, 512), True)])
def test_dropin_takes_the_shift_route(wino, cuda, shape, pin):
    import torch
    n, c, h, w, k = shape
    gen = torch.Generator(device=cuda).manual_seed(2)
    x = torch.randn((n, c, h, w), device=cuda, generator=gen).relu_().half()
    wt = (torch.randn((k, c, 3, 3), device=cuda, generator=gen) * (2 / (9 * c)) ** 0.5).half()
    ws = wino.DropinWorkspaces(n, c, h, w, k, cuda, transform_pin=pin)
    pr = wino.make_problem(x, wt, x, ws.transform_pin, ws.transform_filter, ws.mid_result)
    assert wino.lib().wino_dropin_route(ctypes.byref(pr)) == 5
    y = wino.dropin_conv2d(x, wt, ws=ws)
    torch.cuda.synchronize()
    assert wino.error_read_clear() == 0
    _check(y, x, wt, 1, 1, 1)


def _fused_case(cuda, shape, seed):
    import torch
    n, c, h, w, k = shape
    gen = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn((n, c, h, w), device=cuda, generator=gen).relu_().half()
    wt = (torch.randn((k, c, 3, 3), device=cuda, generator=gen) * (2 / (9 * c)) ** 0.5).half()
    bias = torch.randn(k, device=cuda, generator=gen) * 0.5
    res = (torch.randn((n, k, h, w), device=cuda, generator=gen) * 0.5).half()
    return x, wt, bias, res


# At least 512 MFLOP: one CTA a unit, pairs, odd rows (2-byte stores), a K
# block of 16 beside a full one.
FUSED = [(8, 128, 28, 28, 128), (48, 128, 28, 28, 256), (16, 128, 15, 15, 144), (40, 64, 30, 22, 272)]
# short units one producer group takes, between layers of many stages
RING = [(8, c, h, h, c) for c, h in ((64, 56), (128, 28), (256, 14), (512, 7)) for _ in range(2)]
# The filter from the fp16 U is off by 2.2e-4 in the 2-norm, y's rounding by at
# most 2.8e-4, twice with a residual.
FUSED_REL = 5e-4


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "bias_relu", "residual", "all_in_place"])
@pytest.mark.parametrize("shape", FUSED)
def test_fused_conv_on_a_u_cache(wino, cuda, shape, mode):
    import torch
    x, wt, bias, res = _fused_case(cuda, shape, 3)
    k = shape[4]
    p = wino.fused_conv_workspace_bytes(*shape)
    ws = torch.empty(p, dtype=torch.uint8, device=cuda)
    u = wino.filter_transform(wt)
    ref = torch.nn.functional.conv2d(x.double(), wt.double(), padding=1)
    if mode == "plain":
        y = wino.conv2d_fused(x, u, k, workspace=ws)
    elif mode == "bias_relu":
        y = wino.conv2d_fused_epilogue(x, u, k, bias=bias, relu=True, workspace=ws)
        ref = torch.relu(ref + bias.double().view(1, -1, 1, 1))
    elif mode == "residual":
        y = wino.conv2d_fused_epilogue(x, u, k, residual=res, workspace=ws)
        ref = ref + res.double()
    else:
        ref = torch.relu(ref + bias.double().view(1, -1, 1, 1) + res.double())
        y = wino.conv2d_fused_epilogue(x, u, k, bias=bias, residual=res, relu=True, workspace=ws, out=res)
    torch.cuda.synchronize()
    assert wino.error_read_clear() == 0
    assert float((y.double() - ref).norm() / ref.norm()) <= FUSED_REL


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [FUSED + [(2, 32, 14, 14, 32)], RING])
def test_batch_mixes_kernels(wino, cuda, shapes):
    """Layers of at least 512 MFLOP run in one launch of the shift kernel, the
    others in the fused kernel's; both equal the single-layer calls, from
    capture too and after the U cache was rewritten in place."""
    import torch
    cases = [_fused_case(cuda, s, 4 + i) for i, s in enumerate(shapes)]
    b, outs = wino.Batch(), []
    for x, wt, _, res in cases:
        u = wino.filter_transform(wt)
        n, c, h, w = x.shape
        ws = torch.empty(wino.fused_conv_workspace_bytes(n, c, h, w, wt.shape[0]), dtype=torch.uint8, device=cuda)
        y = torch.full_like(res, float("nan"))
        b.add(x, u, wt.shape[0], y, workspace=ws)
        outs.append((x, u, wt, y))
    torch.cuda.synchronize()
    b.run()
    b.capture()
    for round_ in range(2):
        torch.cuda.synchronize()
        for x, u, wt, y in outs:
            assert torch.equal(y, wino.conv2d_fused(x, u, wt.shape[0]))
            y.fill_(float("nan"))
            if round_ == 0:
                u.copy_(wino.filter_transform(wt * 0.5))
        b.launch()
    torch.cuda.synchronize()
    for x, u, wt, y in outs:
        assert torch.equal(y, wino.conv2d_fused(x, u, wt.shape[0]))
    b.close()
    assert wino.error_read_clear() == 0
