"""Paths that other tests name but their defaults left: the shared persistent
ring (fp32 2^16) from two threads, captures of the three passes, the real
passes and the full-width real 2D transform, and images of columns an odd
distance apart, whose rows no pair of tensor maps describes."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.to(b.dtype) - b).norm() / b.norm())


def test_shared_ring_from_two_threads(gfft):
    import torch
    n, batch, reps = 1 << 16, 24, 12
    g = torch.Generator(device="cuda").manual_seed(16)
    xs = [torch.randn(batch, n, dtype=torch.complex64, device="cuda", generator=g) for _ in range(2)]
    assert gfft.Plan(gfft.KIND_C2C, gfft.F32, n, 0, batch).launches() == 1  # the persistent kernel
    refs = [gfft.fft(x) for x in xs]
    torch.cuda.synchronize()
    outs = [[torch.empty_like(xs[0]) for _ in range(reps)] for _ in range(2)]
    errors = []

    def worker(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for o in outs[i]:
                    gfft.fft(xs[i], out=o)
            s.synchronize()
        except Exception as e:
            errors.append(e)

    th = [threading.Thread(target=worker, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    assert all(torch.equal(o, refs[i]) for i in range(2) for o in outs[i])
    assert gfft.device_error() == 0


@pytest.mark.parametrize("kind,n0,n1,batch,env", [
    ("c2c", 1 << 22, 0, 2, {"GFFT_3PASS": "1"}), ("c2c", 1 << 20, 0, 3, {}), ("c2c", 1 << 12, 0, 2000, {}),
    ("c2c", 1 << 14, 0, 200, {}), ("real", 1 << 20, 0, 2, {}), ("real", 1 << 13, 0, 1300, {}),
    ("r2c_2d", 512, 2048, 1, {}), ("r2c_2d", 64, 4096, 3, {})])
def test_capture_and_replay(gfft, monkeypatch, kind, n0, n1, batch, env):
    import torch
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    if kind == "c2c":
        p = gfft.Plan(gfft.KIND_C2C, gfft.F32, n0, 0, batch)
        assert p.launches() == (3 if env else 1 if n0 <= 1 << 14 else 2)
        x = torch.randn(batch, n0, dtype=torch.complex64, device="cuda")
        y, z = torch.empty_like(x), torch.empty_like(x)
    elif kind == "real":
        p = gfft.Plan(gfft.KIND_R2C, gfft.F32, n0, 0, batch, gfft.FLAG_HALF_SPECTRUM)
        x = torch.randn(batch, n0, device="cuda")
        y, z = torch.empty(batch, n0 // 2 + 1, dtype=torch.complex64, device="cuda"), torch.empty_like(x)
    else:  # full width: columns, then the mirrored half
        p = gfft.Plan(gfft.KIND_R2C_2D, gfft.F32, n0, n1, batch)
        x, z = torch.randn(batch, n1, n0, device="cuda"), None
        y = torch.empty(batch, n1, n0, dtype=torch.complex64, device="cuda")

    def calls():
        p.exec(y, x)
        if z is not None:
            p.exec(z, y, True)

    calls()
    torch.cuda.synchronize()
    ye, ze = y.clone(), None if z is None else z.clone()
    y.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ye) and (z is None or torch.equal(z, ze))
    exact = torch.fft.fft(x.to(torch.complex128)) if kind == "c2c" else \
        torch.fft.rfft(x.double()) if kind == "real" else torch.fft.fft2(x.to(torch.complex128))
    assert rel(y, exact) <= 2e-7 * 22
    assert gfft.device_error() == 0


@pytest.mark.parametrize("logl", [9, 10, 11, 12])
@pytest.mark.parametrize("w,batch", [(33, 2), (257, 3), (64, 3)])
def test_images_of_columns_an_odd_distance_apart(gfft, logl, w, batch):
    import torch
    h = 1 << logl
    d = h * w + 1
    store = torch.randn(batch * d, dtype=torch.complex64, device="cuda")
    out = torch.full((2 * batch * d,), float("nan"), device="cuda").view(torch.complex64)
    assert d % 2 == 1
    p = gfft.Plan(gfft.KIND_VERT, gfft.F32, h, w, batch, 0, w, d, w, d)
    p.exec(out, store)
    for b in range(batch):
        x, y = (t[b * d:b * d + h * w].view(h, w) for t in (store, out))
        assert rel(y, torch.fft.fft(x.to(torch.complex128), dim=0)) <= 2e-7 * logl
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(gfft.fft_vert(x.clone())))
        assert torch.isnan(torch.view_as_real(out[b * d + h * w])).all()
