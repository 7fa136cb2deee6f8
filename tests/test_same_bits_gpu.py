"""A transform's bits do not depend on what stands beside it: a batch, its
parts and the host-buffer calls (which go through the device in chunks) give
the same rows, whichever kernels their sizes select."""
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    import torch
    return torch.equal(torch.view_as_real(a) if a.is_complex() else a, torch.view_as_real(b) if b.is_complex() else b)


@pytest.mark.parametrize("logn,batch", [(11, 9001), (12, 9001), (12, 1825), (13, 1501), (14, 305)])
def test_c2c_rows(gfft, logn, batch):
    import torch
    n = 1 << logn
    x = torch.randn(batch, n, dtype=torch.complex64, device="cuda")
    p, one = gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, batch), gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, 3)
    for inv in (False, True):
        y = p.exec(torch.empty_like(x), x, inv)
        for k in (0, batch // 2, batch - 3):
            assert same(one.exec(torch.empty_like(x[:3]), x[k:k + 3], inv), y[k:k + 3])
        odd = torch.empty(batch * n + 1, dtype=torch.complex64, device="cuda")[1:].view(batch, n)
        odd.copy_(x)  # off a 16-byte boundary
        assert same(p.exec(torch.empty_like(x), odd, inv), y)
    hx = x.cpu()
    for pin in (False, True):
        src, dst = (t.pin_memory() if pin else t for t in (hx.clone(), torch.zeros_like(hx)))
        p.exec_host_ptr(dst.data_ptr(), src.data_ptr(), True)
        assert same(dst, y.cpu())


@pytest.mark.parametrize("logn,batch", [(12, 9001), (13, 1217), (13, 5001), (14, 1501), (15, 401)])
def test_real_rows(gfft, logn, batch):
    import torch
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    x = torch.randn(batch, n, device="cuda")
    f = torch.randn(batch, m, dtype=torch.complex64, device="cuda")
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    one = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, 3, gfft.FLAG_HALF_SPECTRUM)
    y, z = torch.empty_like(f), torch.empty_like(x)
    for call, args, out in (("exec", (x, False), y), ("exec", (f, True), z), ("adjoint", (f, False), z),
                            ("adjoint", (x, True), y)):
        getattr(p, call)(out, *args)
        for k in (0, batch - 3):
            part = getattr(one, call)(torch.empty_like(out[:3]), args[0][k:k + 3].clone(), args[1])
            assert same(part, out[k:k + 3]), (call, args[1])
    p.exec(y, x)
    hx, hy = x.cpu(), torch.zeros(batch, m, dtype=torch.complex64)
    p.exec_host_ptr(hy.data_ptr(), hx.data_ptr())
    assert same(hy, y.cpu())


@pytest.mark.parametrize("logl", [9, 10, 11, 12])
def test_columns(gfft, logl):
    """Any columns of any number of columns, whatever the row stride and the
    boundary the rows start on."""
    import torch
    h = 1 << logl
    x = torch.randn(h, 700, dtype=torch.complex64, device="cuda")
    whole = gfft.fft_vert(x)
    for w in (1, 2, 3, 4, 5, 8, 9, 16, 17, 152, 153, 304, 513, 608, 609):
        assert same(gfft.fft_vert(x[:, :w].contiguous()), whole[:, :w].contiguous()), w
        p = gfft.Plan(gfft.KIND_VERT, gfft.F32, h, w, 1, 0, 700, 0, 700)
        y = torch.empty_like(x)
        p.exec(y[:, 1:], x[:, 1:])
        assert same(y[:, 1:1 + w].contiguous(), whole[:, 1:1 + w].contiguous()), w


@pytest.mark.parametrize("logl,w,batch", [(11, 64, 6), (11, 33, 9), (12, 3, 300), (12, 33, 33), (12, 513, 3)])
def test_batches_of_columns(gfft, logl, w, batch):
    import torch
    h = 1 << logl
    x = torch.randn(batch, h, w, dtype=torch.complex64, device="cuda")
    p, one = gfft.Plan(gfft.KIND_VERT, gfft.F32, h, w, batch), gfft.Plan(gfft.KIND_VERT, gfft.F32, h, w, 1)
    y = p.exec(torch.empty_like(x), x)
    for b in range(0, batch, 4):
        assert same(one.exec(torch.empty_like(x[0]), x[b]), y[b]), b
    hx = x.cpu()
    hy = torch.zeros_like(hx)
    p.exec_host_ptr(hy.data_ptr(), hx.data_ptr())
    assert same(hy, y.cpu())


@pytest.mark.parametrize("h,w,batch", [(2048, 64, 12), (4096, 32, 40), (4096, 512, 5)])
def test_batches_of_real_images(gfft, h, w, batch):
    import torch
    x = torch.randn(batch, h, w, device="cuda")
    half, full = gfft.rfft2(x, half=True), gfft.rfft2(x)
    assert same(half, full[..., :w // 2 + 1].contiguous())
    for b in (0, batch - 1):
        assert same(gfft.rfft2(x[b], half=True), half[b]) and same(gfft.rfft2(x[b]), full[b])


@pytest.mark.parametrize("dtype,logn,batch", [("f32", 15, 7), ("f32", 16, 9), ("f32", 17, 5), ("f32", 18, 80), ("f32", 20, 5),
                                              ("f32", 22, 3), ("f32", 24, 2), ("f64", 13, 30), ("f64", 14, 9),
                                              ("f64", 16, 5), ("f64", 20, 2)])
def test_multipass_rows(gfft, dtype, logn, batch):
    import torch
    n, code = 1 << logn, gfft.F32 if dtype == "f32" else gfft.F64
    cplx = torch.complex64 if dtype == "f32" else torch.complex128
    x = torch.randn(batch, n, dtype=cplx, device="cuda")
    p, one = gfft.Plan(gfft.KIND_C2C, code, n, 0, batch), gfft.Plan(gfft.KIND_C2C, code, n, 0, 1)
    for inv in (False, True):
        y = p.exec(torch.empty_like(x), x, inv)
        for k in (0, batch - 1):
            assert same(one.exec(torch.empty_like(x[:1]), x[k:k + 1].clone(), inv), y[k:k + 1])
        if dtype == "f32":
            odd = torch.empty(batch * n + 1, dtype=cplx, device="cuda")[1:].view(batch, n)
            odd.copy_(x)  # off a 16-byte boundary
            assert same(p.exec(torch.empty_like(x), odd, inv), y)


@pytest.mark.parametrize("logn,batch", [(16, 5), (17, 4), (18, 70), (19, 3), (20, 3), (22, 2), (23, 2)])
def test_multipass_real_rows(gfft, logn, batch):
    import torch
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    x = torch.randn(batch, n, device="cuda")
    f = torch.randn(batch, m, dtype=torch.complex64, device="cuda")
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    one = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, 1, gfft.FLAG_HALF_SPECTRUM)
    y, z = torch.empty_like(f), torch.empty_like(x)
    for call, src, inv, out in (("exec", x, False, y), ("exec", f, True, z), ("adjoint", f, False, z),
                                ("adjoint", x, True, y)):
        getattr(p, call)(out, src, inv)
        for k in (0, batch - 1):
            assert same(getattr(one, call)(torch.empty_like(out[:1]), src[k:k + 1].clone(), inv), out[k:k + 1]), (call, inv)
        pad = 2 if src is x else 1
        odd = torch.empty(src.numel() + pad, dtype=src.dtype, device="cuda")[pad:].view(src.shape)
        odd.copy_(src)
        assert same(getattr(p, call)(torch.empty_like(out), odd, inv), out), (call, inv)


@pytest.mark.parametrize("h,w,batch", [(64, 4096, 40), (1024, 512, 9), (2048, 2048, 3), (32, 1 << 16, 3)])
def test_batches_of_images(gfft, h, w, batch):
    import torch
    x = torch.randn(batch, h, w, dtype=torch.complex64, device="cuda")
    y = gfft.fft2(x)
    for b in (0, batch - 1):
        assert same(gfft.fft2(x[b].clone()), y[b])
