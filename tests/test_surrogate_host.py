"""Host-side logic of the learned jump (no GPU): the sizes of the fallback
pool, which redoes only the members the judge rejects on a model of about
their count."""
import pytest
import torch

from symphas_b200 import _capi as C
from symphas_b200 import surrogate as S


@pytest.mark.parametrize("batch", [1, 2, 7, 64, 256, 1000])
def test_fallback_pool_sizes(batch):
    pool = S.FdPool(256, batch, 0.01)
    sizes = pool.sizes
    assert sizes[0] == 1 and sizes[-1] == batch
    assert all(b > a for a, b in zip(sizes, sizes[1:]))
    # every count of rejected members is padded by at most a quarter (and one)
    for a, b in zip(sizes, sizes[1:]):
        assert b <= max(a + 1, int(a * 1.25 + 0.5)) or b == batch
    assert pool.models == {}  # nothing is created before it is needed


@pytest.mark.parametrize("shape", [(2, 1, 1, 8), (3, 1, 4, 8), (3, 4, 1, 8), (2, 3, 5, 8)])
def test_layers_hand_dense_tensors_to_the_kernels(shape):
    """up2 of one pixel is a view with strides of zero, which reshape keeps: what
    the kernels get of it is dense (they read n h w c values from its start)."""
    x = torch.arange(float(torch.Size(shape).numel())).view(shape)
    up = S.up2(x)
    want = x.repeat_interleave(2, 1).repeat_interleave(2, 2)
    got = S._dense(up)
    assert got.is_contiguous() and torch.equal(got, want)
    off = torch.zeros(x.numel() + 1)[1:].view(shape)
    assert S._dense(off).data_ptr() % 16 == 0 and S._dense(None) is None


class FakeLib:
    """A library whose convolutions gave up `n` times since the last look."""

    def __init__(self, n):
        self.n = n

    def sp_conv_tc_status(self, flag):
        flag._obj.value, self.n = int(self.n > 0), 0
        return C.SP_OK


def test_check_waits_raises_once_for_a_kernel_that_gave_up(monkeypatch):
    fake = FakeLib(2)
    monkeypatch.setattr(C, "lib", lambda: fake)
    with pytest.raises(C.SymPhasError) as e:
        S.check_waits()
    assert e.value.code == C.SP_ETIMEOUT
    S.check_waits()
