"""What the front end hands to the kernels, on the CPU."""
import pytest
import torch

import genfft_gb300 as G
from genfft_gb300 import torchfft  # noqa: F401  (binds the dtype tables)


def test_dense_tensors_hold_their_values():
    z = torch.randn(3, 4, dtype=torch.complex64)
    for x in (z, z.conj(), z.t(), z.t().conj(), z.conj().imag, z.real, torch._neg_view(z).conj()):
        d = G._dense(x)
        assert d.is_contiguous() and not d.is_conj() and not d.is_neg() and torch.equal(d, x)
        if x.is_contiguous() and not x.is_conj() and not x.is_neg():
            assert d is x
    assert G._stored(z) is z
    for x in (z.conj(), z.conj().imag):
        with pytest.raises(ValueError):
            G._stored(x)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_reals_start_on_a_pair(dtype):
    x = torch.arange(12, dtype=dtype)
    size = 2 * x.element_size()
    for v in (x[1:9], x[3:], x[1:9].view(2, 4)):
        d = G._dense(v)
        assert v.data_ptr() % size and d.data_ptr() % size == 0 and torch.equal(d, v)
    assert G._dense(x[2:]).data_ptr() == x[2:].data_ptr()
