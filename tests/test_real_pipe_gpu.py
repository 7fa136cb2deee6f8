"""fp32 R2C and half-spectrum C2R of n = 2^18 .. 2^22 on the pipelined passes
(csrc/real_pipe.cu) against FP64 at the fp32 bound 2e-7*log2(n): odd
batches (every other transform's spectrum starts off a 16-byte boundary),
more tiles than stages on every SM, unaligned bases, the adjoints with their
interior weights, scaling, and guard bands around the outputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bound(n):
    return 2e-7 * int(np.log2(n))


def rel(a, b):
    return float((a.to(b.dtype) - b).norm() / b.norm())


def guarded(count, dtype, shift=0, pad=64):
    import torch
    real = 2 if dtype == torch.complex64 else 1
    buf = torch.full((real * (count + 2 * pad + 2),), float("nan"), device="cuda")
    buf = buf.view(torch.complex64) if real == 2 else buf
    return buf, buf[pad + shift:pad + shift + count]


def untouched(buf, out):
    import torch
    off = (out.data_ptr() - buf.data_ptr()) // buf.element_size()
    flat = torch.view_as_real(buf) if buf.is_complex() else buf
    return bool(torch.isnan(flat[:off]).all() and torch.isnan(flat[off + out.numel():]).all())


@pytest.mark.parametrize("logn,batch", [(18, 1), (18, 37), (19, 2), (19, 23), (20, 1), (20, 9), (21, 3), (22, 1),
                                        (22, 5), (23, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward_inverse_adjoint(gfft, logn, batch, shift):
    import torch
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    g = torch.Generator(device="cuda").manual_seed(logn * 100 + batch)
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    # the input starts 8 bytes off a 16-byte boundary where shift is 1
    x = torch.randn(batch * n + 2, device="cuda", generator=g)[2 * shift:2 * shift + batch * n].view(batch, n)
    exact = torch.fft.rfft(x.double())
    buf, y = guarded(batch * m, torch.complex64, shift)
    p.exec(y, x, scale=0.5)
    for b in {0, batch // 2, batch - 1}:
        assert rel(2 * y.view(batch, m)[b], exact[b]) <= bound(n), b
    assert untouched(buf, y)
    # inverse of any bins; the imaginary parts of F_0 and F_(n/2) do not count
    f = torch.randn(batch * m + 1, dtype=torch.complex64, device="cuda", generator=g)[shift:shift + batch * m]
    f = f.view(batch, m)
    buf, z = guarded(batch * n, torch.float32, 2 * shift)
    p.exec(z, f, True)
    exact = torch.fft.irfft(f.to(torch.complex128), n=n, norm="forward")
    for b in {0, batch // 2, batch - 1}:
        assert rel(z.view(batch, n)[b], exact[b]) <= bound(n), b
    assert untouched(buf, z)
    # adjoint of the forward transform: interior bins halved
    gx = torch.empty(batch, n, device="cuda")
    p.adjoint(gx, f, False)
    h = f.to(torch.complex128).clone()
    h[:, 1:-1] *= 0.5
    assert rel(gx, torch.fft.irfft(h, n=n, norm="forward")) <= bound(n)
    # adjoint of the inverse: interior bins doubled
    gf = torch.empty(batch, m, dtype=torch.complex64, device="cuda")
    p.adjoint(gf, x, True)
    exact = torch.fft.rfft(x.double())
    exact[:, 1:-1] *= 2
    assert rel(gf, exact) <= bound(n)
    assert gfft.device_error() == 0


def test_full_spectrum_and_its_adjoint(gfft):
    import torch
    n, batch = 1 << 20, 3
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(batch, n, device="cuda", generator=g)
    y = gfft.rfft(x, half=False)
    assert rel(y, torch.fft.fft(x.double())) <= bound(n)
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch)
    gy = torch.randn(batch, n, dtype=torch.complex64, device="cuda", generator=g)
    gx = torch.empty(batch, n, device="cuda")
    p.adjoint(gx, gy, False)
    assert rel(gx, torch.fft.ifft(gy.to(torch.complex128), norm="forward").real) <= bound(n)
