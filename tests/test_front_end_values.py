"""What the front end hands to the kernels, on the CPU."""
import pytest
import torch

import genfft_gb300 as G


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
