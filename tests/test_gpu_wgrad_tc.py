"""The tcgen05 weight gradient against a float64 reference on the same bf16
operands, at the edges of its tiles: images smaller than a block, widths that
are not a multiple of an MMA's 16 pixels or of a column block (128), a last
row block that is not full, every channel tile (32, 64, 128 outputs; 32, 64,
128 inputs), circular wrap on every side, and accumulation into dw.

Products of bf16 values are exact in fp32; a sum of K of them in fp32 is off
by at most about K 2^-24 of the sum of magnitudes and by sqrt(K) 2^-24 of it
in the mean: 1e-4 of the largest gradient is well above that for the sizes
here (K <= 17000) and far below one wrong or missing pixel."""
import ctypes
import pathlib
import subprocess
import sys

import pytest
import torch
import torch.nn.functional as F

from symphas_b200 import _capi as C

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def reference(x, dy, co, ci):
    """dw [co][3][3][ci] by one matrix product per tap, in float64."""
    out = torch.zeros(co, 3, 3, ci, device="cuda", dtype=torch.float64)
    d = dy.double().reshape(-1, co)
    for t in range(9):
        xs = torch.roll(x.double(), (1 - t // 3, 1 - t % 3), (1, 2)).reshape(-1, ci)
        out[:, t // 3, t % 3] = d.t() @ xs
    return out


@pytest.mark.parametrize("n,h,w,ci,co", [
    (1, 1, 1, 32, 32), (1, 2, 3, 64, 64), (2, 5, 7, 32, 32), (1, 9, 130, 32, 32),
    (3, 33, 17, 32, 64), (1, 8, 8, 64, 64), (2, 16, 24, 96, 64), (1, 20, 36, 64, 128),
    (1, 7, 63, 128, 128), (2, 32, 32, 128, 256), (1, 3, 260, 256, 32), (1, 40, 16, 128, 32),
    (2, 9, 11, 256, 128), (1, 64, 256, 32, 32), (4, 64, 64, 64, 32)])
def test_weight_gradient(n, h, w, ci, co):
    torch.manual_seed(n + h + w + ci + co)
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16()
    dy = torch.randn(n, h, w, co, device="cuda").bfloat16()
    base = torch.randn(co, 3, 3, ci, device="cuda")
    dw = base.clone()
    flag = ctypes.c_int(-1)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert C.lib().sp_conv3x3_wgrad(ptr(x), ptr(dy), ptr(dw), n, h, w, ci, co, s) == C.SP_OK
    assert C.lib().sp_conv_tc_status(ctypes.byref(flag)) == C.SP_OK and flag.value == 0
    want = reference(x, dy, co, ci)
    err = (dw.double() - base.double() - want).abs().max() / want.abs().max()
    assert float(err) < 1e-4, float(err)


def test_weight_gradient_unaligned_output():
    """dw that does not start on 16 bytes: the sums are added one by one."""
    torch.manual_seed(0)
    n, h, w, ci, co = 1, 12, 20, 32, 64
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16()
    dy = torch.randn(n, h, w, co, device="cuda").bfloat16()
    buf = torch.zeros(co * 9 * ci + 1, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert C.lib().sp_conv3x3_wgrad(ptr(x), ptr(dy), ctypes.c_void_p(buf.data_ptr() + 4), n, h, w,
                                    ci, co, s) == C.SP_OK
    torch.cuda.synchronize()
    want = reference(x, dy, co, ci)
    got = buf[1:].view(co, 3, 3, ci).double()
    assert float((got - want).abs().max() / want.abs().max()) < 1e-4


CAPTURED_FIRST_CALL = """
import ctypes, torch
from symphas_b200 import _capi as C
p = lambda t: ctypes.c_void_p(t.data_ptr())
torch.manual_seed(0)
x = torch.randn(1, 12, 20, 32, device="cuda").bfloat16()
dy = torch.randn(1, 12, 20, 64, device="cuda").bfloat16()
dw = torch.zeros(64, 3, 3, 32, device="cuda")
C.lib()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert C.lib().sp_conv3x3_wgrad(p(x), p(dy), p(dw), 1, 12, 20, 32, 64, s) == C.SP_OK
g.replay()
torch.cuda.synchronize()
d = dy.double().reshape(-1, 64)
for t in range(9):
    xs = torch.roll(x.double(), (1 - t // 3, 1 - t % 3), (1, 2)).reshape(-1, 32)
    want = d.t() @ xs
    err = (dw[:, t // 3, t % 3].double() - want).abs().max() / want.abs().max()
    assert float(err) < 1e-4, (t, float(err))
"""


def test_first_call_of_a_process_under_capture():
    """Nothing is allocated on the way: a process whose first convolution call
    is a weight gradient in a stream capture replays it."""
    r = subprocess.run([sys.executable, "-c", CAPTURED_FIRST_CALL], capture_output=True, text=True,
                       timeout=300, cwd=str(pathlib.Path(__file__).resolve().parent.parent))
    assert r.returncode == 0, r.stderr[-2000:]
