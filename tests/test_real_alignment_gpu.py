"""Real arrays that start between two pairs of elements: the C ABI refuses them
before any launch, the tensor functions transform a copy."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("logn", [1, 4, 13, 16, 18])
def test_plans_refuse(gfft, dtype, logn):
    import torch
    real, cplx = (torch.float32, torch.complex64) if dtype == "f32" else (torch.float64, torch.complex128)
    code, n = (gfft.F32 if dtype == "f32" else gfft.F64), 1 << logn
    x = torch.randn(2 * n + 1, dtype=real, device="cuda")[1:].view(2, n)
    f = torch.randn(2, n // 2 + 1, dtype=cplx, device="cuda")
    p = gfft.Plan(gfft.KIND_R2C, code, n, 0, 2, gfft.FLAG_HALF_SPECTRUM)
    keep, fkeep = x.clone(), f.clone()
    for call in (lambda: p.exec(f, x), lambda: p.exec(x, f, True), lambda: p.adjoint(x, f), lambda: p.adjoint(f, x, True)):
        with pytest.raises(gfft.GFFTError) as e:
            call()
        assert e.value.name == "GFFT_ERR_ALIGN"
    if logn > 1:
        q = gfft.Plan(gfft.KIND_R2C_2D, code, n // 2, 2, 2, gfft.FLAG_HALF_SPECTRUM)
        with pytest.raises(gfft.GFFTError) as e:
            q.exec(torch.empty(2, 2, n // 4 + 1, dtype=cplx, device="cuda"), x)
        assert e.value.name == "GFFT_ERR_ALIGN"
    torch.cuda.synchronize()
    assert torch.equal(x, keep) and torch.equal(torch.view_as_real(f), torch.view_as_real(fkeep))


@pytest.mark.parametrize("n", [1, 2, 64, 1 << 14, 1 << 16])
def test_tensor_functions_take_any_slice(gfft, n):
    import torch
    from genfft_gb300 import autograd as GA
    from genfft_gb300 import torchfft as GT
    x = torch.randn(4 * n + 1, device="cuda")[1:].view(4, n)
    y, bound = torch.fft.rfft(x.double()), 2e-7 * 16
    rel = lambda a, b: float((a.to(b.dtype) - b).norm() / b.norm())
    assert rel(gfft.rfft(x), y) <= bound and rel(GT.rfft(x), y) <= bound and rel(GA.rfft(x), y) <= bound
    assert rel(gfft.rfft2(x, half=True), torch.fft.rfft2(x.double())) <= bound
    assert rel(GT.rfft2(x), torch.fft.rfft2(x.double())) <= bound
    f = y.to(torch.complex64).requires_grad_()
    if n > 1:
        g = torch.randn(4 * n + 1, device="cuda")[1:].view(4, n)
        GT.irfft(f, n=n).backward(g)
        f64 = y.clone().requires_grad_()
        torch.fft.irfft(f64, n=n).backward(g.double())
        assert rel(f.grad, f64.grad) <= bound
