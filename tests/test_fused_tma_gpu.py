"""The persistent fused kernels of fp32 complex lengths 2^12 .. 2^14
(csrc/fused_tma.cu) against FP64 at the fp32 bound 2e-7*log2(n) and, where
both hold 32 points a thread, bit for bit against the plain kernels, which
small batches and transforms that start off a 16-byte boundary take:
batches of one, of a group more or less than a wave of the 152 SMs, of
several waves; padded distances; in place; between guard bands; beside the
tensor-core path, the other user of tensor memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bound(n):
    return 2e-7 * int(np.log2(n))


def rel(a, b):
    return float((a.to(b.dtype) - b).norm() / b.norm())


@pytest.mark.parametrize("logn,batch", [(12, 1), (12, 7296), (12, 7297), (12, 9001), (13, 1), (13, 912), (13, 913),
                                        (13, 2001),
                                        (14, 1), (14, 152), (14, 153), (14, 305), (14, 1001)])
def test_against_fp64_and_plain_kernel(gfft, logn, batch):
    import torch
    n, pad = 1 << logn, 64
    g = torch.Generator(device="cuda").manual_seed(logn * 10000 + batch)
    store = torch.randn(batch * n + 1, dtype=torch.complex64, device="cuda", generator=g)
    x, keep = store[:batch * n].view(batch, n), store.clone()
    off = torch.empty_like(store)
    off[1:] = store[:-1]
    p = gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, batch)
    for inv in (False, True):
        buf = torch.full((2 * (batch * n + 2 * pad),), float("nan"), device="cuda").view(torch.complex64)
        y = buf[pad:pad + batch * n].view(batch, n)
        p.exec(y, x, inv, scale=0.5)
        x64 = x.to(torch.complex128)
        exact = 0.5 * (torch.fft.ifft(x64, norm="forward") if inv else torch.fft.fft(x64))
        assert rel(y, exact) <= bound(n)
        assert torch.isnan(torch.view_as_real(buf[:pad])).all()
        assert torch.isnan(torch.view_as_real(buf[pad + batch * n:])).all()
        assert torch.equal(torch.view_as_real(store), torch.view_as_real(keep))
        z = torch.empty_like(x)
        p.exec(z, off[1:].view(batch, n), inv, scale=0.5)  # 8 bytes off: the plain kernel
        assert logn == 12 or torch.equal(z, y)
        assert rel(z, exact) <= bound(n)
    z = x.clone()
    p.exec(z, z)
    y = torch.empty_like(x)
    p.exec(y, x)
    assert torch.equal(z, y)
    assert gfft.device_error() == 0


@pytest.mark.parametrize("logn,batch", [(12, 7500), (13, 1000), (14, 200)])
def test_padded_distances(gfft, logn, batch):
    import torch
    n = 1 << logn
    for idist, odist in ((n + 6, n + 3), (n + 5, n + 2)):  # even (copies) and odd (plain kernel)
        x = torch.randn(batch, idist, dtype=torch.complex64, device="cuda")
        out = torch.zeros(batch, odist, dtype=torch.complex64, device="cuda")
        p = gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, batch, 0, 1, idist, 1, odist)
        p.exec(out, x)
        assert rel(out[:, :n], torch.fft.fft(x[:, :n].to(torch.complex128))) <= bound(n)
        assert (out[:, n:] == 0).all()


@pytest.mark.parametrize("logn,batch", [(13, 3649), (13, 5001), (14, 913), (14, 1501), (15, 153), (15, 401)])
@pytest.mark.parametrize("shift", [0, 1])
def test_real_transforms(gfft, logn, batch, shift):
    """R2C and C2R of 2^13 .. 2^15 reals and their adjoints; the same rows in
    small batches go through the plain kernels."""
    import torch
    n, m, pad = 1 << logn, (1 << (logn - 1)) + 1, 64
    g = torch.Generator(device="cuda").manual_seed(logn * 10000 + batch)
    x = torch.randn(batch, n, device="cuda", generator=g)
    f = torch.randn(batch * m + 1, dtype=torch.complex64, device="cuda", generator=g)[shift:shift + batch * m]
    f = f.view(batch, m)
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    small = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, 50, gfft.FLAG_HALF_SPECTRUM)
    buf = torch.full((2 * (batch * m + 2 * pad + 1),), float("nan"), device="cuda").view(torch.complex64)
    y = buf[pad + shift:pad + shift + batch * m].view(batch, m)
    p.exec(y, x, scale=0.5)
    assert rel(y, 0.5 * torch.fft.rfft(x.double())) <= bound(n)
    assert torch.isnan(torch.view_as_real(buf[:pad + shift])).all()
    assert torch.isnan(torch.view_as_real(buf[pad + shift + batch * m:])).all()
    buf = torch.full((batch * n + 2 * pad,), float("nan"), device="cuda")
    z = buf[pad:pad + batch * n].view(batch, n)
    p.exec(z, f, True, scale=0.5)
    assert rel(z, 0.5 * torch.fft.irfft(f.to(torch.complex128), n=n, norm="forward")) <= bound(n)
    assert torch.isnan(buf[:pad]).all() and torch.isnan(buf[pad + batch * n:]).all()
    gx, gf = torch.empty(batch, n, device="cuda"), torch.empty(batch, m, dtype=torch.complex64, device="cuda")
    p.adjoint(gx, f, False)
    p.adjoint(gf, x, True)
    h = f.to(torch.complex128).clone()
    h[:, 1:-1] *= 0.5
    assert rel(gx, torch.fft.irfft(h, n=n, norm="forward")) <= bound(n)
    h = torch.fft.rfft(x.double())
    h[:, 1:-1] *= 2
    assert rel(gf, h) <= bound(n)
    if logn > 13:  # 32 points a thread in both
        for k in (0, batch - 50):
            rows = slice(k, k + 50)
            a, b = torch.empty(50, m, dtype=torch.complex64, device="cuda"), torch.empty(50, n, device="cuda")
            fr = f[rows].contiguous()
            assert torch.equal(small.exec(a, x[rows], scale=0.5), y[rows])
            assert torch.equal(small.exec(b, fr, True, scale=0.5), z[rows])
            assert torch.equal(small.adjoint(b, fr, False), gx[rows])
            assert torch.equal(small.adjoint(a, x[rows], True), gf[rows])
    assert gfft.device_error() == 0


def test_beside_the_tensor_core_path(gfft):
    """Both kernels take tensor memory; back to back on one stream and on two
    streams at once they give what they give alone."""
    import torch
    x = torch.randn(1000, 1 << 13, dtype=torch.complex64, device="cuda")
    z = torch.randn(2000, 4096, dtype=torch.complex64, device="cuda")
    a, b = gfft.fft(x), gfft.fft_tc(z)
    torch.cuda.synchronize()
    s = [torch.cuda.Stream() for _ in range(2)]
    for two in (False, True):
        outs = []
        for _ in range(5):
            with torch.cuda.stream(s[0]):
                u = gfft.fft(x)
            with torch.cuda.stream(s[1] if two else s[0]):
                outs.append((u, gfft.fft_tc(z)))
        torch.cuda.synchronize()
        for u, v in outs:
            assert torch.equal(u, a) and torch.equal(v, b)
    assert gfft.device_error() == 0
