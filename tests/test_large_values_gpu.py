"""Values near the type's limits and non-finite ones through the real
transforms' kernels of every length: what does not overflow in the sum that
defines the result does not overflow inside, and a NaN or an infinity stays in
its own transform."""
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [(10, 3), (14, 3), (14, 1000), (15, 400), (16, 2), (18, 2), (20, 2), (22, 1)]


@pytest.mark.parametrize("logn,batch", LENGTHS)
def test_adjoint_of_one_large_bin(gfft, logn, batch):
    """The adjoint of the half-spectrum R2C halves its interior bins: one bin g
    gives values of size |g|.  Two neighbouring outputs are one complex value
    inside, whose parts a twiddle may turn into one another, so |g| sqrt(2) has
    to stay below 3.4e38: g = 2.3e38, of which the sum of two would not.  (Bin
    n/4 pairs with itself, bin 5 with n/2 - 5.)"""
    import torch
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    for k in (0, 5, n // 4, n // 2):
        f = torch.zeros(batch, m, dtype=torch.complex64, device="cuda")
        f[:, k] = 2.3e38
        x = p.adjoint(torch.empty(batch, n, device="cuda"), f, False)
        j = torch.arange(n, device="cuda", dtype=torch.float64)
        exact = 2.3e38 * torch.cos(2 * torch.pi * ((j * k) % n) / n)
        assert float((x.double() - exact).abs().max()) <= 2.3e38 * 2e-7 * logn, k


@pytest.mark.parametrize("logn,batch", LENGTHS)
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_non_finite_values_stay_in_their_transform(gfft, logn, batch, bad):
    import torch
    if batch == 1:
        batch = 3
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, batch, gfft.FLAG_HALF_SPECTRUM)
    x = torch.randn(batch, n, device="cuda")
    f = torch.randn(batch, m, dtype=torch.complex64, device="cuda")
    for call, v, out in (("exec", x, f), ("exec", f, x), ("adjoint", f, x), ("adjoint", x, f)):
        inverse = (call == "exec") == v.is_complex()
        good = getattr(p, call)(torch.empty_like(out), v, inverse)
        w = v.clone()
        w[1, 7] = bad
        y = getattr(p, call)(torch.empty_like(out), w, inverse)
        rest = [i for i in range(batch) if i != 1]
        assert torch.equal(y[rest], good[rest])
        assert not torch.isfinite(torch.view_as_real(y[1]) if y.is_complex() else y[1]).any(dim=-1).all()
    assert gfft.device_error() == 0


@pytest.mark.parametrize("logn,batch", [(13, 1000), (14, 200), (17, 3), (20, 2)])
def test_non_finite_c2c(gfft, logn, batch):
    import torch
    n = 1 << logn
    p = gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, batch)
    x = torch.randn(batch, n, dtype=torch.complex64, device="cuda")
    good = p.exec(torch.empty_like(x), x)
    w = x.clone()
    w[1, 7] = float("nan")
    y = p.exec(torch.empty_like(x), w)
    rest = [i for i in range(batch) if i != 1]
    assert torch.equal(y[rest], good[rest]) and torch.isnan(y[1]).all()
