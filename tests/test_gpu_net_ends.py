"""The jump network's first and last convolutions as kernels of their own, the
element-wise backward with the bias gradient, and a layer's autograd function,
against float64 references on the same bf16 operands: image edges (circular
wrap, extents 1 and 2, column blocks of 64 and 62, row blocks of 32), every
channel count of the dispatch.  Outputs stored in bf16 are within one rounding
(2^-8 of the value) plus tanh.approx's 2^-11; fp32 sums of K bf16 products
within K 2^-24 of the sum of magnitudes."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from symphas_b200 import _capi as C
from symphas_b200 import surrogate as S

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def conv64(x, w, b=None):
    n, h, wd, ci = x.shape
    out = 0
    for t in range(9):
        xs = torch.roll(x.double(), (1 - t // 3, 1 - t % 3), (1, 2))
        out = out + xs.reshape(-1, ci) @ w.double()[:, t // 3, t % 3].t()
    return (out if b is None else out + b.double()).view(n, h, wd, -1)


SIZES = [(1, 1, 1), (2, 2, 3), (1, 33, 64), (2, 32, 65), (1, 31, 62), (1, 64, 63), (1, 5, 256)]


@pytest.mark.parametrize("n,h,w", SIZES)
@pytest.mark.parametrize("co", [32, 96])
def test_first_layer(n, h, w, co):
    torch.manual_seed(h + w)
    psi = torch.randn(n, h, w, device="cuda")
    wt = (torch.randn(co, 3, 3, 32, device="cuda") / 3).bfloat16()
    b = 0.1 * torch.randn(co, device="cuda")
    a = torch.full((n, h, w, co), float("nan"), device="cuda", dtype=torch.bfloat16)
    assert C.lib().sp_conv3x3_in1(ptr(psi), ptr(wt), ptr(b), ptr(a), n, h, w, 32, co,
                                  stream()) == C.SP_OK
    want = F.gelu(conv64(psi.bfloat16()[..., None], wt[..., :1], b), approximate="tanh")
    assert torch.allclose(a.double(), want, rtol=2.0 ** -7, atol=2e-3)
    assert C.lib().sp_conv3x3_in1(ptr(psi), ptr(wt), ptr(b), ptr(a), n, h, w, 32, 48,
                                  stream()) == C.SP_EINVAL


@pytest.mark.parametrize("n,h,w", SIZES)
@pytest.mark.parametrize("ci", [32, 64])
def test_last_layer(n, h, w, ci):
    torch.manual_seed(h + w)
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16()
    wt = torch.randn(32, 3, 3, ci, device="cuda").bfloat16()
    b = torch.randn(32, device="cuda")
    out = torch.full((n, h, w), float("nan"), device="cuda")
    assert C.lib().sp_conv3x3_out1(ptr(x), ptr(wt), ptr(b), ptr(out), n, h, w, ci,
                                   stream()) == C.SP_OK
    want = conv64(x, wt[:1], b[:1])[..., 0]
    mag = conv64(x.abs(), wt[:1].abs())[..., 0]
    assert ((out.double() - want).abs() <= 9 * ci * 2.0 ** -24 * (mag + 1)).all()
    assert C.lib().sp_conv3x3_out1(ptr(x), ptr(wt), ptr(b), ptr(out), n, h, w, 16,
                                   stream()) == C.SP_EINVAL


@pytest.mark.parametrize("npix,c", [(1, 8), (7, 24), (1000, 32), (33, 256), (5, 2048), (9, 2056), (70000, 64)])
def test_gelu_backward_and_bias_gradient(npix, c):
    torch.manual_seed(c)
    z = (3 * torch.randn(npix, c, device="cuda")).bfloat16()
    z[0, :4] = torch.tensor([0.0, -30.0, 30.0, 1e4])
    da = torch.randn(npix, c, device="cuda").bfloat16()
    dz = torch.full_like(z, float("nan"))
    db = torch.ones(c, device="cuda")
    assert C.lib().sp_gelu_bwd_bf16(ptr(z), ptr(da), ptr(dz), ptr(db), npix, c, stream()) == C.SP_OK
    zr = z.double().requires_grad_()
    F.gelu(zr, approximate="tanh").backward(da.double())
    # the derivative in fp32 to ~2e-6 absolute, then one bf16 rounding
    tol = 2.0 ** -8 * zr.grad.abs() + 2e-6 * da.double().abs() + 1e-30
    assert ((dz.double() - zr.grad).abs() <= tol).all()
    bound = npix * 2.0 ** -24 * (dz.double().abs().sum(0) + 1) + 1e-6
    assert ((db.double() - 1 - dz.double().sum(0)).abs() <= bound).all()
    db2 = torch.zeros(c, device="cuda")
    assert C.lib().sp_gelu_bwd_bf16(None, ptr(da), None, ptr(db2), npix, c, stream()) == C.SP_OK
    bound = npix * 2.0 ** -24 * (da.double().abs().sum(0) + 1) + 1e-6
    assert ((db2.double() - da.double().sum(0)).abs() <= bound).all()
    assert C.lib().sp_gelu_bwd_bf16(ptr(z), ptr(da), None, ptr(db), npix, c,
                                    stream()) == C.SP_EINVAL


@pytest.mark.parametrize("skip", [False, True])
def test_layer_autograd(skip):
    """conv_gelu under autograd, with an upstream gradient that does not start
    on a 16-byte boundary."""
    torch.manual_seed(5)
    n, h, w, ci, co = 2, 12, 20, 32, 64
    layer = S.ConvLayer(ci, co, torch.Generator().manual_seed(1))
    layer.b.normal_()
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16().requires_grad_()
    res = torch.randn(n, h, w, co, device="cuda").bfloat16().requires_grad_() if skip else None
    buf = torch.randn(n * h * w * co + 1, device="cuda").bfloat16()
    dy = buf[1:].view(n, h, w, co)
    y = S.conv_gelu(x, layer, res)
    y.backward(dy)
    xr, wr = x.detach().double().requires_grad_(), layer.wb.double().requires_grad_()
    br = layer.b.double().requires_grad_()
    zr = conv64(xr, wr, br)
    rr = res.detach().double().requires_grad_() if skip else None
    yr = F.gelu(zr if rr is None else zr + rr, approximate="tanh")
    yr.backward(dy.double())

    def rel(a, b):
        return float((a.double() - b).norm() / b.norm())

    assert rel(y, yr) < 4e-3 and rel(x.grad, xr.grad) < 8e-3
    assert rel(layer.gw, wr.grad) < 4e-3 and rel(layer.gb, br.grad) < 8e-3
    if skip:
        assert rel(res.grad, rr.grad) < 4e-3


def strided(t, how):
    """The values of t in a tensor that is not dense (or not on 16 bytes)."""
    if how == "permuted":
        return t.permute(0, 3, 1, 2).contiguous().permute(0, 2, 3, 1)
    if how == "expanded":
        return t[:1, :1, :1].expand(t.shape)
    buf = torch.zeros(t.numel() + 1, device="cuda", dtype=t.dtype)
    buf[1:].copy_(t.reshape(-1))
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("how", ["permuted", "expanded", "off"])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("entry", ["conv", "conv_gelu", "conv_gelu_up"])
def test_layers_take_any_strides(entry, grad, how):
    """Inputs and skips that are views: as the same values in dense tensors."""
    torch.manual_seed(6)
    n, h, w, ci, co = 2, 6, 10, 32, 64
    up = 2 if entry == "conv_gelu_up" else 1
    layer = S.ConvLayer(ci, co, torch.Generator().manual_seed(1))
    x = strided(torch.randn(n, h, w, ci, device="cuda").bfloat16(), how)
    res = strided(torch.randn(n, up * h, up * w, co, device="cuda").bfloat16(), how)
    dy = torch.randn(n, up * h, up * w, co, device="cuda").bfloat16()
    outs = []
    for a, r in ((x, res), (x.clone(memory_format=torch.contiguous_format),
                            res.clone(memory_format=torch.contiguous_format))):
        layer.zero_grad()
        with torch.set_grad_enabled(grad):
            a, r = a.detach().requires_grad_(grad), r.detach().requires_grad_(grad)
            y = getattr(S, entry)(a, layer, r)
            if grad:
                y.backward(dy)
                outs.append((y.detach(), a.grad, r.grad, layer.gb.clone()))
                wg = layer.gw.clone()
            else:
                outs.append((y.detach(),))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    if grad:  # (the weight gradient's sums have no fixed order)
        first = outs[0]
        layer.zero_grad()
        a = x.detach().requires_grad_()
        getattr(S, entry)(a, layer, res.detach()).backward(dy)
        assert float((layer.gw - wg).norm() / wg.norm()) < 1e-5 and len(first) == 4


@pytest.mark.parametrize("ch,nb", [((32, 64), 3), ((32, 64, 128), 2), ((32, 64, 128, 256), 3)])
def test_network_down_to_one_pixel(ch, nb):
    """A field whose deepest level is one pixel: training reads the up-sampled
    pixel as inference does."""
    torch.manual_seed(8)
    net = S.JumpNet(ch, seed=2)
    side = 2 ** (len(ch) - 1)
    psi = torch.rand(nb, side, side, device="cuda") - 0.5
    with torch.no_grad():
        want = net(psi)
    got = net(psi)
    got.square().sum().backward()
    # bf16 activations through two paths that round at the ends differently, and
    # the mean of a few values taken off
    assert torch.isfinite(got).all()
    assert float((got.detach() - want).abs().max()) < 0.1 * float(want.abs().max()) + 1e-3
    assert all(torch.isfinite(l.gw).all() and torch.isfinite(l.gb).all() for l in net.layers())


@pytest.mark.parametrize("kernel", ["strip", "tc", "mma"])
@pytest.mark.parametrize("co", [32, 128])
def test_training_activation_is_rounded_once(kernel, co, monkeypatch):
    """conv_gelu under autograd through a layer that copies its input (the centre
    tap the identity, so that the pre-activation is every bf16 value in turn): the
    activation is within half a unit in the last place of bf16 (2^-8 of the
    value at most) and the 2^-20 that its fp32 arithmetic may add, also where 1 +
    tanh cancels (down to fp32's smallest normal values, 12 / 2^126)."""
    monkeypatch.setattr(S, "KERNEL", kernel)
    v = torch.arange(0, 65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    v = v[(v.double().abs() <= 12) & (v.double().abs() >= 2.0 ** -20)].cuda()
    v = torch.cat([v, v[: -v.numel() % (64 * co)]])
    x = v.view(1, -1, 64, co).contiguous().requires_grad_()
    layer = S.ConvLayer(co, co, torch.Generator().manual_seed(0))
    layer.wb.zero_()
    layer.wb[:, 1, 1, :] = torch.eye(co, device="cuda").bfloat16()
    a = S.conv_gelu(x, layer).detach().double()
    z = x.detach().double()
    want = z / (1 + torch.exp(-2 * 0.7978845608028654 * (z + 0.044715 * z ** 3)))
    assert ((a - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs() + 12 * 2.0 ** -126).all()


@pytest.mark.parametrize("npix,c", [(1, 8), (7, 24), (1000, 32), (33, 256), (9, 2056), (300000, 64)])
@pytest.mark.parametrize("with_z", [False, True])
def test_ordered_bias_gradient(npix, c, with_z):
    """The same bits in every run, and the sums of dz as stored."""
    torch.manual_seed(c)
    z = (3 * torch.randn(npix, c, device="cuda")).bfloat16() if with_z else None
    da = torch.randn(npix, c, device="cuda").bfloat16()
    dz = torch.empty_like(da) if with_z else None
    need = ctypes.c_longlong()
    assert C.lib().sp_gelu_bwd_scratch(npix, c, ctypes.byref(need)) == C.SP_OK
    got = []
    for _ in range(8):
        db = torch.ones(c, device="cuda")
        ws = torch.full((need.value + 1,), float("nan"), device="cuda")
        assert C.lib().sp_gelu_bwd_ordered_bf16(ptr(z), ptr(da), ptr(dz), ptr(db), ptr(ws), npix, c,
                                                stream()) == C.SP_OK
        assert torch.isnan(ws[-1])
        got.append(db)
    assert all(torch.equal(got[0], g) for g in got)
    v = (dz if with_z else da).double()
    bound = npix * 2.0 ** -24 * (v.abs().sum(0) + 1) + 1e-6
    assert ((got[0].double() - 1 - v.sum(0)).abs() <= bound).all()
    assert C.lib().sp_gelu_bwd_ordered_bf16(ptr(z), ptr(da), ptr(dz), ptr(got[0]), None, npix, c,
                                            stream()) == C.SP_EINVAL


def test_layer_bias_gradient_repeats_itself():
    torch.manual_seed(9)
    n, h, w, ci, co = 8, 96, 96, 32, 64
    layer = S.ConvLayer(ci, co, torch.Generator().manual_seed(1))
    x = torch.randn(n, h, w, ci, device="cuda").bfloat16()
    dy = torch.randn(n, h, w, co, device="cuda").bfloat16()
    got = []
    for _ in range(6):
        layer.zero_grad()
        S.conv_gelu(x, layer).backward(dy)
        got.append(layer.gb.clone())
    assert all(torch.equal(got[0], g) for g in got)
