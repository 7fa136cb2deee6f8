"""The pipelined tile kernels (csrc/tiles_pipe.cuh): the column and row passes
of fp32 C2C n = 2^17 .. 2^24 and the fp32 column FFTs of 2^9 .. 2^12 points,
against FP64 at the fp32 bound 2e-7*log2(n).  Batches and column counts sit
at the edges of tiles and waves (one tile, one more, a last partial tile,
more tiles than stages on every SM), row strides and bases on and off
16-byte boundaries, in place and out of place, between guard bands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bound(n):
    return 2e-7 * int(np.log2(n))


def rel(a, b):
    return float((a.to(b.dtype) - b).norm() / b.norm())


@pytest.mark.parametrize("logn,batch", [(17, 1), (17, 301), (18, 3), (18, 97), (19, 41), (20, 1), (20, 23), (21, 2),
                                        (21, 13), (22, 3), (23, 1), (24, 1)])
def test_c2c_two_passes(gfft, logn, batch):
    import torch
    n = 1 << logn
    g = torch.Generator(device="cuda").manual_seed(logn * 1000 + batch)
    x = torch.randn(batch, n, dtype=torch.complex64, device="cuda", generator=g)
    x64 = x.to(torch.complex128)
    for inv in (False, True):
        y = gfft.fft(x, inv)
        exact = torch.fft.ifft(x64, norm="forward") if inv else torch.fft.fft(x64)
        for b in {0, batch // 2, batch - 1}:
            assert rel(y[b], exact[b]) <= bound(n), (inv, b)
        del exact
    z = x.clone()
    gfft.fft(z, out=z)
    assert torch.equal(z, gfft.fft(x))
    assert gfft.device_error() == 0


# columns around one tile, one wave of short tiles (608) and several waves;
# odd counts put every other row off a 16-byte boundary
@pytest.mark.parametrize("logl,cols", [(9, 1), (9, 15), (9, 17), (9, 4097), (9, 16384), (10, 7), (10, 9), (10, 4999),
                                       (10, 8192), (11, 1), (11, 608), (11, 609), (11, 612), (11, 2049), (11, 4096),
                                       (12, 3), (12, 609), (12, 612), (12, 2049), (12, 2052)])
@pytest.mark.parametrize("shift", [0, 1])
def test_columns(gfft, logl, cols, shift):
    import torch
    n = 1 << logl
    g = torch.Generator(device="cuda").manual_seed(logl * 100000 + cols)
    store = torch.randn(n * cols + 2, dtype=torch.complex64, device="cuda", generator=g)
    x = store[shift:shift + n * cols].view(n, cols)  # base 8 bytes off a 16-byte boundary where shift is 1
    keep = store.clone()
    x64 = x.to(torch.complex128)
    pad = 64
    p = gfft.Plan(gfft.KIND_VERT, gfft.F32, n, cols)
    for inv in (False, True):
        exact = torch.fft.ifft(x64, dim=0, norm="forward") if inv else torch.fft.fft(x64, dim=0)
        buf = torch.full((2 * (n * cols + 2 * pad),), float("nan"), device="cuda").view(torch.complex64)
        y = buf[pad:pad + n * cols].view(n, cols)
        p.exec(y, x, inv)
        assert rel(y, exact) <= bound(n), inv
        assert torch.isnan(torch.view_as_real(buf[:pad])).all()
        assert torch.isnan(torch.view_as_real(buf[pad + n * cols:])).all()
        assert torch.equal(torch.view_as_real(store), torch.view_as_real(keep))
    z = store.clone()[shift:shift + n * cols].view(n, cols)
    p.exec(z, z)
    q = torch.empty(n, cols, dtype=torch.complex64, device="cuda")
    p.exec(q, x)
    assert torch.equal(z, q)
    assert gfft.device_error() == 0


@pytest.mark.parametrize("h,w", [(512, 96), (1024, 64), (2048, 2048), (4096, 1024)])
def test_real_2d_half_and_full(gfft, h, w):
    """Half-width output (odd row stride) and full-width output (Hermitian
    store) of real images hold the same bits in the shared columns."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(h + w)
    x = torch.randn(3, h, w, device="cuda", generator=g)
    if w & (w - 1):
        w = 1 << (w.bit_length() - 1)
        x = x[..., :w].contiguous()
    half = gfft.rfft2(x, half=True)
    full = gfft.rfft2(x)
    exact = torch.fft.rfft2(x.double())
    assert rel(half, exact) <= bound(h * w)
    assert torch.equal(half, full[..., : w // 2 + 1].contiguous())
    k = (-torch.arange(h, device="cuda")) % h
    assert torch.equal(full[..., w // 2 + 1:].contiguous(), half[:, k][..., 1:w // 2].flip(-1).conj().resolve_conj())
    assert gfft.device_error() == 0
