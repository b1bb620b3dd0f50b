"""The persistent tcgen05 convolution (weights resident in shared memory, or
streamed): each of its tiles (32, 64 and 128 outputs; 1024, 512 and 256
positions), K loops of one to sixteen stages, images smaller than a tile and than a strip's reach,
several tiles a CTA, outputs that start on 16 but not on 32 bytes, every set of
epilogue operands -- against a float64 reference on the same bf16 operands.
The sums are exact to K 2^-24 of their magnitude, the stored pre-activation to
one bf16 rounding (2^-8) more, the activation to tanh.approx's 2^-11 more."""
import ctypes
import math

import pytest
import torch
import torch.nn.functional as F

from symphas_b200 import _capi as C

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def conv64(x, w):
    n, h, wd, ci = x.shape
    out = 0
    for t in range(9):
        xs = torch.roll(x.double(), (1 - t // 3, 1 - t % 3), (1, 2))
        out = out + xs.reshape(-1, ci) @ w.double()[:, t // 3, t % 3].t()
    return out.view(n, h, wd, -1)


@pytest.mark.parametrize("n,h,w,ci,co", [
    (1, 1, 1, 32, 32), (1, 2, 3, 32, 64), (3, 33, 17, 64, 32), (2, 70, 300, 32, 32),
    (1, 40, 400, 128, 32), (5, 67, 67, 64, 64), (2, 20, 130, 128, 64), (2, 31, 64, 64, 128),
    (1, 9, 11, 32, 256), (40, 100, 101, 32, 32), (1, 16, 16, 256, 32), (2, 128, 128, 32, 64),
    # weights streamed: one and several tiles a CTA, K blocks of 16 channels, two
    # output blocks, a strip wider than its tile
    (1, 5, 7, 128, 128), (2, 130, 130, 144, 128), (1, 33, 17, 256, 256), (1, 6, 640, 128, 128)])
@pytest.mark.parametrize("ops", ["bias,res,z,a", "a", "z"])
def test_flow_convolution(n, h, w, ci, co, ops):
    torch.manual_seed(h * w + ci)
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16()
    wt = (torch.randn(co, 3, 3, ci, device="cuda") / (3 * ci ** 0.5)).bfloat16()
    b = 0.1 * torch.randn(co, device="cuda") if "bias" in ops else None
    res = torch.randn(n, h, w, co, device="cuda").bfloat16() if "res" in ops else None
    scratch = torch.empty(9 * ci * co, device="cuda", dtype=torch.bfloat16)
    off = 8 if n == 3 else 0  # elements: 16 bytes

    def out(on):
        if not on:
            return None
        buf = torch.full((n * h * w * co + off,), float("nan"), device="cuda", dtype=torch.bfloat16)
        return buf[off:].view(n, h, w, co)

    z, a = out("z" in ops), out("a" in ops.split(","))
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert C.lib().sp_conv3x3_fwd_strip(ptr(x), ptr(wt), ptr(scratch), ptr(b), ptr(res), ptr(z),
                                        ptr(a), n, h, w, ci, co, s) == C.SP_OK
    flag = ctypes.c_int(-1)
    assert C.lib().sp_conv_tc_status(ctypes.byref(flag)) == C.SP_OK and flag.value == 0
    zr = conv64(x, wt) + (0 if b is None else b.double()) + (0 if res is None else res.double())
    for got, want in ((z, zr), (a, F.gelu(zr, approximate="tanh"))):
        if got is not None:
            assert torch.allclose(got.double(), want, rtol=2.0 ** -7, atol=2e-3)


@pytest.mark.parametrize("ci,co", [(32, 32), (32, 64), (128, 128)])
@pytest.mark.parametrize("off_w,off_res", [(1, 0), (0, 2), (8, 2), (3, 6)])
@pytest.mark.parametrize("up", [False, True])
def test_weights_and_residual_off_16_bytes(ci, co, off_w, off_res, up):
    """w on any element and res on any pair of channels (offsets in elements of
    bf16): such calls keep the strip kernel, whose accesses are that narrow."""
    torch.manual_seed(ci + co)
    n, h, w = 2, 12, 18
    x = torch.randn(n, h // 2 if up else h, w // 2 if up else w, ci, device="cuda").bfloat16()
    xr = x.repeat_interleave(2, 1).repeat_interleave(2, 2) if up else x

    def at(shape, off, scale):
        buf = (scale * torch.randn(math.prod(shape) + off, device="cuda")).bfloat16()
        return buf[off:].view(shape)

    wt = at((co, 3, 3, ci), off_w, 1 / (3 * ci ** 0.5))
    res = at((n, h, w, co), off_res, 1.0)
    assert (wt.data_ptr() % 16 or res.data_ptr() % 16) and res.data_ptr() % 4 == 0
    scratch = torch.empty(9 * ci * co, device="cuda", dtype=torch.bfloat16)
    z = torch.full((n, h, w, co), float("nan"), device="cuda", dtype=torch.bfloat16)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    fwd = C.lib().sp_conv3x3_fwd_strip_up2 if up else C.lib().sp_conv3x3_fwd_strip
    assert fwd(ptr(x), ptr(wt), ptr(scratch), None, ptr(res), ptr(z), None, n, h, w, ci, co,
               s) == C.SP_OK
    flag = ctypes.c_int(-1)
    assert C.lib().sp_conv_tc_status(ctypes.byref(flag)) == C.SP_OK and flag.value == 0
    assert torch.allclose(z.double(), conv64(xr, wt) + res.double(), rtol=2.0 ** -7, atol=2e-3)
