"""Batched device copies (sp_upload_batch_device / sp_download_batch_device):
one field of every instance to or from one dense device array.  They must
move the same values as the per-instance copies, and an upload must leave
the halos as the per-instance upload does (the steps after it give the same
bits), for periodic and Dirichlet sides, 2D and 3D, FP32 and FP64."""
import ctypes

import numpy as np
import pytest
import torch

import symphas_b200 as sp
from symphas_b200 import _capi as C

pytestmark = pytest.mark.gpu


def make(dim, n, dtype, batch, dirichlet=False):
    P, D = sp.BoundaryType.PERIODIC, sp.BoundaryType.DEFAULT
    bc = [D, D] + [P] * 4 if dirichlet else [P] * 6
    st = sp.Stencil2d2h(5, 6, 13) if dim == 2 else sp.Stencil3d2h(7, 10, 25)
    return sp.model_MB_t(dim, sp.SolverFT(st, form="fused"),
                         sp.ProblemParameters((n,) * dim, h=1.0, boundary=bc, boundary_value=0.3),
                         dtype=dtype, batch=batch)


@pytest.mark.parametrize("dim,n", [(2, 40), (3, 20)])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("dirichlet", [False, True])
def test_batch_copies_match_per_instance_copies(dim, n, dtype, dirichlet):
    torch.cuda.set_device(0)
    batch = 5
    tdt = torch.float32 if dtype == "f32" else torch.float64
    g = torch.Generator(device="cuda").manual_seed(3)
    x = (0.2 * torch.rand((batch,) + (n,) * dim, device="cuda", generator=g, dtype=tdt) - 0.1)
    a = make(dim, n, dtype, batch, dirichlet)
    b = make(dim, n, dtype, batch, dirichlet)
    esz = x.element_size()
    sites = n ** dim
    a.batch_from_device(0, x.data_ptr(), x.numel() * esz)
    for i in range(batch):
        b.field_from_device(0, x[i].data_ptr(), sites * esz, inst=i)
    torch.cuda.synchronize()
    for i in range(batch):
        assert np.array_equal(a.get_field(0, inst=i), x[i].cpu().numpy())
    a.step(0.002, 7)
    b.step(0.002, 7)
    out = torch.empty_like(x)
    a.batch_to_device(0, out.data_ptr(), out.numel() * esz)
    a.synchronize()
    for i in range(batch):
        got = b.get_field(0, inst=i)
        assert np.array_equal(a.get_field(0, inst=i), got), i
        assert np.array_equal(out[i].cpu().numpy(), got), i
    a.close()
    b.close()


def test_batch_copy_rejects_wrong_sizes():
    torch.cuda.set_device(0)
    m = make(2, 16, "f32", 3)
    x = torch.zeros(2, 16, 16, device="cuda")
    with pytest.raises(C.SymPhasError):
        m.batch_from_device(0, x.data_ptr(), x.numel() * 4)
    with pytest.raises(C.SymPhasError):
        m.batch_to_device(1, x.data_ptr(), 3 * 256 * 4)
    m.close()


def managed(nbytes):
    """(address, free): memory that a copy engine takes and no kernel is sent to."""
    rt = ctypes.CDLL("libcudart.so.12")
    p = ctypes.c_void_p()
    assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(nbytes), 1) == 0
    return p.value, lambda: rt.cudaFree(p)


@pytest.mark.parametrize("dims,batch", [((33, 21), 3), ((8, 700), 2), ((61, 9, 7), 2), ((36, 5, 4), 3),
                                        ((128, 640), 64)])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("off", [0, 1])
def test_copies_of_ragged_rows_and_unaligned_arrays(dims, batch, dtype, off):
    """Rows that are no whole 16-byte units, dense arrays that start on a value
    but not on 16 bytes, one and four rows a thread, one instance and all."""
    torch.cuda.set_device(0)
    tdt = torch.float32 if dtype == "f32" else torch.float64
    sites = int(np.prod(dims))
    x = torch.rand(batch * sites + off, device="cuda", dtype=tdt)[off:]
    esz = x.element_size()
    assert off == 0 or x.data_ptr() % 16 != 0
    dim = len(dims)
    st = sp.Stencil2d2h(5, 6, 13) if dim == 2 else sp.Stencil3d2h(7, 10, 25)
    m = sp.model_MA_t(dim, sp.SolverFT(st, form="fused"), sp.ProblemParameters(dims), dtype=dtype,
                      batch=batch)
    m.batch_from_device(0, x.data_ptr(), x.numel() * esz)
    out = torch.full((batch * sites + off + 1,), -7.0, device="cuda", dtype=tdt)
    m.batch_to_device(0, out.data_ptr() + off * esz, batch * sites * esz)
    one = torch.full((sites + off + 1,), -7.0, device="cuda", dtype=tdt)
    last = batch - 1
    m.field_to_device(0, one.data_ptr() + off * esz, sites * esz, inst=last)
    y = torch.rand(sites + off, device="cuda", dtype=tdt)[off:]
    torch.cuda.synchronize()  # (the model works on a stream of its own)
    m.field_from_device(0, y.data_ptr(), sites * esz, inst=0)
    m.synchronize()
    assert torch.equal(out[off:-1], x) and torch.equal(one[off:-1], x[last * sites:])
    assert out[-1] == -7.0 and one[-1] == -7.0 and (off == 0 or (out[0] == -7.0 and one[0] == -7.0))
    assert np.array_equal(m.get_field(0, inst=0).ravel(), y.cpu().numpy())
    if batch > 1:
        assert np.array_equal(m.get_field(0, inst=last).ravel(), x[last * sites:].cpu().numpy())
    m.close()


@pytest.mark.parametrize("dims", [(40, 24), (33, 10, 6)])
def test_copies_to_and_from_managed_memory(dims):
    """Memory that is not plain device memory takes the copy engine."""
    torch.cuda.set_device(0)
    sites = int(np.prod(dims))
    dim = len(dims)
    st = sp.Stencil2d2h(5, 6, 13) if dim == 2 else sp.Stencil3d2h(7, 10, 25)
    m = sp.model_MA_t(dim, sp.SolverFT(st, form="fused"), sp.ProblemParameters(dims), dtype="f64")
    p, free = managed(8 * sites)
    host = np.ctypeslib.as_array((ctypes.c_double * sites).from_address(p))
    host[:] = np.random.default_rng(1).uniform(size=sites)
    want = host.copy()
    m.field_from_device(0, p, 8 * sites)
    m.synchronize()
    host[:] = 0.0
    m.field_to_device(0, p, 8 * sites)
    m.synchronize()
    assert np.array_equal(host, want) and np.array_equal(m.get_field(0).ravel(), want)
    m.close()
    free()
