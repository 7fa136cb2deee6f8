"""The Python front end's short ways: calls outside autograd skip the
autograd.Function (torchfft), functions that make a plan a call keep the
plans that hold no workspace.  Both give the bits of the general way, and
calls the short way is not for still take the general one."""
import threading

import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((5, 64), -1), ((64, 5), 0), ((3, 32, 7), 1), ((2, 4096), -1)]


@pytest.mark.parametrize("name", ["fft", "ifft", "rfft", "irfft"])
@pytest.mark.parametrize("shape,dim", SHAPES)
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_plain_calls_match_autograd_calls(gfft, name, shape, dim, dtype):
    import torch
    from genfft_gb300 import torchfft as GT
    real = torch.float32 if dtype == "f32" else torch.float64
    cplx = torch.complex64 if dtype == "f32" else torch.complex128
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(*shape, dtype=real if name == "rfft" else cplx, device="cuda", generator=g)
    kw = {"n": shape[dim]} if name == "irfft" else {}
    f = getattr(GT, name)
    with torch.no_grad():
        a = f(x, dim=dim, norm="ortho", **kw)
    y = x.clone().requires_grad_()
    b = f(y, dim=dim, norm="ortho", **kw)
    assert b.requires_grad and not a.requires_grad
    assert a.shape == b.shape and torch.equal(a, b.detach())
    with torch.inference_mode():
        assert torch.equal(f(x, dim=dim, norm="ortho", **kw), a)
    b.abs().sum().backward()
    assert y.grad is not None


@pytest.mark.parametrize("dims", [(-2, -1), (0, 1), (2, 0)])
def test_plain_2d_calls_match_autograd_calls(gfft, dims):
    import torch
    from genfft_gb300 import torchfft as GT
    x = torch.randn(16, 32, 64, dtype=torch.complex64, device="cuda")
    for f in (GT.fft2, GT.ifft2):
        a = f(x, dim=dims)
        b = f(x.clone().requires_grad_(), dim=dims)
        assert b.requires_grad and torch.equal(a, b.detach())
        exact = getattr(torch.fft, f.__name__)(x.to(torch.complex128), dim=dims)
        assert float((a - exact).norm() / exact.norm()) <= 2e-7 * 11


def test_transforms_and_dual_tensors_take_the_general_way(gfft):
    import torch
    import torch.autograd.forward_ad as fwd
    from genfft_gb300 import torchfft as GT
    x = torch.randn(4, 64, dtype=torch.complex64, device="cuda")
    with pytest.raises(RuntimeError):  # no vmap rule for the kernels
        torch.func.vmap(GT.fft)(x)
    with fwd.dual_level():
        assert not GT._plain(x)
        d = fwd.make_dual(x, torch.ones_like(x))
        with pytest.raises((RuntimeError, NotImplementedError)):  # no forward-mode rule either
            GT.fft(d)
    assert GT._plain(x)


@pytest.mark.parametrize("name", ["fft", "ifft", "rfft", "irfft", "fft2", "ifft2"])
def test_traced_calls_run_again(gfft, name):
    import torch
    from genfft_gb300 import torchfft as GT
    f = getattr(GT, name)
    x, y = (torch.randn(4, 64, dtype=torch.float32 if name == "rfft" else torch.complex64, device="cuda")
            for _ in range(2))
    if name == "irfft":
        x, y = x[:, :33].contiguous(), y[:, :33].contiguous()
    # (a length read off a traced shape is a tensor, which irfft refuses)
    kw = {"n": 64} if name == "irfft" else {}
    traced = torch.jit.trace(lambda v: f(v, norm="ortho", **kw), x, check_trace=False)
    assert torch.equal(traced(y), f(y, norm="ortho", **kw))


def test_kept_plans_from_two_threads(gfft):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    ims = [torch.randn(3, 64, 128, dtype=torch.complex64, device="cuda", generator=g) for _ in range(2)]
    res = [torch.randn(5, 4096, device="cuda", generator=g) for _ in range(2)]
    want = [(gfft.fft2(ims[i]), gfft.rfft(res[i])) for i in range(2)]
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for _ in range(50):
                    got[i].append((gfft.fft2(ims[i]), gfft.rfft(res[i])))
            s.synchronize()
        except Exception as e:
            errors.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    for i in range(2):
        for a, b in got[i]:
            assert torch.equal(a, want[i][0]) and torch.equal(b, want[i][1])
    # the pool is bounded, and plans with a workspace are not in it
    for k in range(80):
        gfft.rfft(torch.ones(k + 1, 16, device="cuda"))
    gfft.rfft(torch.ones(1, 1 << 20, device="cuda"))
    assert len(gfft._STATELESS) <= gfft._STATELESS_MAX
    assert all(key[3] < (1 << 20) for key in gfft._STATELESS)
