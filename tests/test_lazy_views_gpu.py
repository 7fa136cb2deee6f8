"""Lazily conjugated and negated tensors (x.conj(), x.conj().imag) are
transformed by their values, not by what is stored, forward and backward;
outputs of that kind are refused.  Against torch.fft in FP64, at the fp32
bound 2e-7*log2(n)."""
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.to(b.dtype) - b).norm() / b.norm())


def lazy_real(shape, g):
    """reals that are the negated imaginary parts of a conjugated tensor"""
    import torch
    z = torch.randn(*shape, dtype=torch.complex64, device="cuda", generator=g)
    x = z.conj().imag
    assert x.is_neg()
    return x


NAMES = ["fft", "ifft", "rfft", "irfft", "fft2", "ifft2", "rfft2", "irfft2"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("dims", ["last", "first"])
def test_torchfft_values(gfft, name, dims):
    import torch
    from genfft_gb300 import torchfft as GT
    g = torch.Generator(device="cuda").manual_seed(5)
    shape = (32, 64)
    if name in ("irfft", "irfft2"):
        shape = (32, 33) if dims == "last" else (33, 32)
    x = lazy_real(shape, g) if name.startswith("rfft") else torch.randn(*shape, dtype=torch.complex64, device="cuda",
                                                                       generator=g).conj()
    kw = {"dim": ((-2, -1) if dims == "last" else (1, 0)) if name.endswith("2") else (-1 if dims == "last" else 0)}
    x64 = x.to(torch.float64 if name.startswith("rfft") else torch.complex128).resolve_conj()
    assert rel(getattr(GT, name)(x, **kw), getattr(torch.fft, name)(x64, **kw)) <= 2e-7 * 11


@pytest.mark.parametrize("name", ["fft", "ifft", "rfft", "irfft", "fft2", "ifft2"])
def test_gradient_through_a_conjugation(gfft, name):
    """The gradient that reaches backward() is lazily conjugated itself."""
    import torch
    from genfft_gb300 import torchfft as GT
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(4, 64, dtype=torch.float32 if name == "rfft" else torch.complex64, device="cuda", generator=g)
    if name == "irfft":
        x = x[:, :33].contiguous()
    grads = []
    for mod, dt in ((GT, x.dtype), (torch.fft, torch.float64 if name == "rfft" else torch.complex128)):
        v = x.detach().clone().to(dt).requires_grad_()
        y = getattr(mod, name)(v if name != "irfft" else v.conj())
        w = torch.arange(1, y.numel() + 1, device="cuda", dtype=y.real.dtype).view(y.shape)
        (y if name == "irfft" else y.conj()).mul(w * (1.0 if name == "irfft" else 1 + 2j)).sum().abs().backward()
        grads.append(v.grad)
    assert rel(grads[0], grads[1]) <= 2e-7 * 12


def test_autograd_module(gfft):
    import torch
    from genfft_gb300 import autograd as GA
    z = torch.randn(4, 64, dtype=torch.complex64, device="cuda")
    z64 = z.to(torch.complex128)
    plan = gfft.RaggedPlan([64, 64, 128])
    assert rel(GA.fft(z.conj()), torch.fft.fft(z64.conj())) <= 2e-7 * 6
    assert rel(GA.irfft(z[:, :33].conj(), 64), torch.fft.irfft(z64[:, :33].conj(), n=64, norm="forward")) <= 2e-7 * 6
    p = GA.ragged_fft(z.reshape(-1).conj(), plan)
    assert rel(p[:64], torch.fft.fft(z64[0].conj())) <= 2e-7 * 6
    v = z.clone().requires_grad_()
    (GA.fft(v).conj() * torch.arange(64, device="cuda")).sum().abs().backward()
    v64 = z64.clone().requires_grad_()
    (torch.fft.fft(v64).conj() * torch.arange(64, device="cuda")).sum().abs().backward()
    assert rel(v.grad, v64.grad) <= 2e-7 * 7


def test_module_functions_and_plans(gfft):
    import torch
    z = torch.randn(32, 64, dtype=torch.complex64, device="cuda")
    c, c64 = z.conj(), z.to(torch.complex128).conj()
    assert rel(gfft.fft(c), torch.fft.fft(c64)) <= 2e-7 * 6
    assert rel(gfft.ifft(c), torch.fft.ifft(c64, norm="forward")) <= 2e-7 * 6
    assert rel(gfft.fft2(c), torch.fft.fft2(c64)) <= 2e-7 * 11
    assert rel(gfft.fft_vert(c), torch.fft.fft(c64, dim=0)) <= 2e-7 * 5
    t = torch.randn(2, 256, dtype=torch.complex64, device="cuda")
    assert rel(gfft.fft_tc(t.conj()), torch.fft.fft(t.to(torch.complex128).conj())) <= 4e-6
    p = gfft.Plan(gfft.KIND_C2C, gfft.F32, 64, 0, 32)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    y = p.exec(torch.empty_like(z), c, stream=s)
    h = p.adjoint(torch.empty_like(z), c, scale=0.5, stream=s)
    s.synchronize()
    assert rel(y, torch.fft.fft(c64)) <= 2e-7 * 6
    assert rel(h, 0.5 * torch.fft.ifft(c64, norm="forward")) <= 2e-7 * 6


def test_lazy_outputs_are_refused(gfft):
    import torch
    z = torch.randn(32, 64, dtype=torch.complex64, device="cuda")
    keep = z.clone()
    p = gfft.Plan(gfft.KIND_C2C, gfft.F32, 64, 0, 32)
    x = torch.zeros_like(z)
    for call in (lambda: gfft.fft(x, out=z.conj()), lambda: gfft.fft2(x, out=z.conj()),
                 lambda: gfft.fft_vert(x, out=z.conj()), lambda: p.exec(z.conj(), x),
                 lambda: p.adjoint(z.conj(), x), lambda: gfft.fft_no_scramble(z.conj()),
                 lambda: gfft.fft_vert_no_scramble(z.conj())):
        with pytest.raises(ValueError):
            call()
    assert torch.equal(z, keep)
