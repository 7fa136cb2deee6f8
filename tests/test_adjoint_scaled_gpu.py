"""The scaled adjoint (the backward pass of norm=) against the plain one times
the factor, over the real transforms' paths."""
import math

import pytest

pytestmark = pytest.mark.gpu

# (n, batch): one point, fused, persistent fused, multi-pass, batches in odd numbers
SHAPES = [(1, 3), (2, 3), (64, 5), (8192, 3), (8192, 4001), (32768, 201), (65536, 3), (1 << 18, 3), (1 << 20, 1),
          (1 << 23, 1)]


@pytest.mark.parametrize("n,batch", SHAPES)
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("half", [True, False])
def test_scaled_adjoint(gfft, n, batch, dtype, inverse, half):
    import torch
    if inverse and not half:
        pytest.skip("the inverse takes the half spectrum")
    real, cplx = (torch.float32, torch.complex64) if dtype == "f32" else (torch.float64, torch.complex128)
    m = n // 2 + 1 if half else n
    plan = gfft.Plan(gfft.KIND_R2C, gfft.F32 if dtype == "f32" else gfft.F64, n, 0, batch,
                     gfft.FLAG_HALF_SPECTRUM if half else 0)
    gen = torch.Generator(device="cuda").manual_seed(n + batch)
    bins, reals = ((batch, m), cplx), ((batch, n), real)
    src, dst = (reals, bins) if inverse else (bins, reals)
    g = torch.randn(*src[0], dtype=src[1], device="cuda", generator=gen)
    out = [torch.empty(*dst[0], dtype=dst[1], device="cuda") for _ in range(2)]
    plan.adjoint(out[0], g, inverse)
    # a power of two is exact; any other factor rounds once
    plan.adjoint(out[1], g, inverse, scale=2.0 ** -7)
    assert torch.equal(out[1], out[0] * 2.0 ** -7)
    f = 1.0 / math.sqrt(3.0)
    plan.adjoint(out[1], g, inverse, scale=f)
    eps = torch.finfo(real).eps
    assert float((out[1] - out[0] * f).abs().max()) <= 2 * eps * float(out[0].abs().max())
