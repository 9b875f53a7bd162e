"""The drop-in's slots on both sides of the shift route's threshold, launched as a
harness launches them: four plain cudaLaunchKernel calls.

A problem that the two-stage route fits but the shift route takes has the conv in
slot 2; slots 3 and 4 hold the two-stage kernels, which find no M and return.
Below the threshold they are that route, and equal its entry point bit for bit.
"""
import ctypes

import pytest

import test_shift_conv as base

pytestmark = pytest.mark.gpu


class _Dim3(ctypes.Structure):
    _fields_ = [("x", ctypes.c_uint), ("y", ctypes.c_uint), ("z", ctypes.c_uint)]


def _info(wino, x, wt, y, ws):
    pr = wino.make_problem(x, wt, y, ws.transform_pin, ws.transform_filter, ws.mid_result)
    param = (ctypes.c_char * wino.get_param_size(pr))()
    rc, ki = wino.get_kernel_info(pr, param)
    assert rc == 0
    return ki, param, wino.lib().wino_dropin_route(ctypes.byref(pr))


def _harness(wino, ki, param):
    rt = ctypes.CDLL("libcudart.so.12")     # the instance the library is linked to
    rt.cudaLaunchKernel.argtypes = [ctypes.c_void_p, _Dim3, _Dim3, ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t,
                                    ctypes.c_void_p]
    args = (ctypes.c_void_p * 1)(ctypes.addressof(param))
    for i in (1, 2, 3, 4):
        s = ki.slot(i)
        assert rt.cudaLaunchKernel(s["kernel"], _Dim3(*s["grid"]), _Dim3(*s["block"]), args, s["lds"], wino._stream()) == 0


# 604 MFLOP, one CTA a unit; 3.7 GFLOP, pairs; 65 MFLOP, just past the threshold
@pytest.mark.parametrize("shape", [(8, 64, 32, 32, 64), (64, 256, 14, 14, 256), (2, 64, 22, 20, 64)])
def test_shift_route_runs_in_slot_2(wino, cuda, shape):
    import torch
    n, c, h, w, k = shape
    x, wt, _, _ = base._fused_case(cuda, shape, 21)
    ws = wino.DropinWorkspaces(n, c, h, w, k, cuda)
    ws.mid_result.fill_(float("nan"))
    y = torch.full((n, k, h, w), float("nan"), dtype=torch.float16, device=cuda)
    ki, param, route = _info(wino, x, wt, y, ws)
    L = wino.lib()
    assert route == wino.ROUTE_SHIFT
    assert ki.slot(2)["lds"] == L.wino_shift_smem_bytes() and ki.slot(2)["block"][0] == L.wino_shift_threads()
    assert ki.slot(3)["kernel"] == L.wino_twostage_gemm_kernel_ptr_for(c) and ki.slot(3)["lds"] == 0
    assert ki.slot(4)["kernel"] == L.wino_twostage_output_kernel_ptr()
    _harness(wino, ki, param)
    torch.cuda.synchronize()
    base._check(y, x, wt, 1, 1, 1)
    assert torch.equal(y, wino.dropin_conv2d(x, wt, ws=ws))
    assert bool(ws.mid_result.isnan().all())
    assert wino.error_read_clear() == 0


# 57 to 59 MFLOP: the two-stage route itself
@pytest.mark.parametrize("shape", [(2, 64, 20, 20, 64), (1, 128, 16, 16, 96), (2, 256, 8, 8, 96)])
def test_two_stage_route_below_the_threshold(wino, cuda, shape):
    import torch
    n, c, h, w, k = shape
    x, wt, _, _ = base._fused_case(cuda, shape, 22)
    ws = wino.DropinWorkspaces(n, c, h, w, k, cuda)
    y = torch.full((n, k, h, w), float("nan"), dtype=torch.float16, device=cuda)
    ki, param, route = _info(wino, x, wt, y, ws)
    assert route == 3 and ki.slot(3)["lds"] > 48 * 1024
    assert ki.slot(3)["kernel"] == wino.lib().wino_twostage_gemm_kernel_ptr_for(c)
    _harness(wino, ki, param)
    two = wino.conv2d_twostage(x, wino.filter_transform_unfused(wt), k)
    torch.cuda.synchronize()
    assert torch.equal(y, two) and torch.equal(y, wino.dropin_conv2d(x, wt, ws=ws))
    ref = torch.nn.functional.conv2d(x.double(), wt.double(), padding=1)
    assert float((y.double() - ref).norm() / ref.norm()) <= 2e-3
    assert wino.error_read_clear() == 0


@pytest.mark.parametrize("r,s,stride,shift", [(1, 1, 2, False), (1, 2, 2, False), (2, 1, 2, False), (3, 1, 2, True),
                                              (1, 2, 1, True), (2, 1, 1, True)])
def test_strided_filters_of_two_taps_gather(wino, cuda, r, s, stride, shift):
    """They read few of the pixels: the implicit GEMM that gathers them serves
    strided filters of up to two taps, the shift kernel the others."""
    import torch
    gen = torch.Generator(device=cuda).manual_seed(r + 8 * s)
    x = torch.randn((10, 32, 61, 58), device=cuda, generator=gen).half()
    wt = (torch.randn((128, 32, r, s), device=cuda, generator=gen) / (32 * r * s) ** 0.5).half()
    ws = wino.DropinWorkspaces(10, 32, 61, 58, 128, cuda)
    oh, ow = (61 - r) // stride + 1, (58 - s) // stride + 1
    y = torch.empty((10, 128, oh, ow), dtype=torch.float16, device=cuda)
    pr = wino.make_problem(x, wt, y, ws.transform_pin, ws.transform_filter, ws.mid_result, r=r, s=s, u=stride, v=stride,
                           p=0, q=0)
    rc, ki = wino.get_kernel_info(pr, (ctypes.c_char * wino.get_param_size(pr))())
    assert rc == 0
    assert (ki.slot(3)["lds"] == wino.lib().wino_shift_smem_bytes()) is shift
    y = wino.dropin_conv2d(x, wt, ws=ws, stride=stride, pad=0)
    torch.cuda.synchronize()
    base._check(y, x, wt, stride, 0, 0)
    assert wino.error_read_clear() == 0
