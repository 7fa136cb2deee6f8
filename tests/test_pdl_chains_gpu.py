"""Calls that follow one another on a stream without a pause, through the same
workspaces and buffers, each on other values: a kernel that starts while the one before it still
runs reads what that one wrote, not what an earlier call had left there.  The
plain kernels (GFFT_NO_TMA) and the TMA ones, against FP64, and call for call
the same bits as with a synchronisation after each."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, torch
sys.path.insert(0, %r)
import genfft_gb300 as G
c64 = torch.complex64
g = torch.Generator(device="cuda").manual_seed(3)
CALLS = 6
rel = lambda a, b: float((a.to(b.dtype) - b).norm() / b.norm())

def check(name, xs, shape, call, exact, bound):
    # the same plan on one input after the other, with and without a pause
    res = {}
    for pause in (True, False):
        outs = [torch.empty_like(shape) for _ in xs]
        torch.cuda.synchronize()
        for o, x in zip(outs, xs):
            call(o, x)
            if pause:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        res[pause] = outs
    for x, a, b in zip(xs, res[True], res[False]):
        e = rel(a, exact(x)), rel(b, exact(x))
        assert max(e) <= bound, (name, e)
        assert torch.equal(a, b), name

def chain(name, plans, xs, bufs, exact, bound):
    # one buffer to the next, plan by plan, without a pause
    outs = []
    for x in xs:
        bufs[0].copy_(x)
        for k, (p, inv) in enumerate(plans):
            p.exec(bufs[k + 1], bufs[k], inv)
        outs.append(bufs[-1].clone())
    torch.cuda.synchronize()
    for x, o in zip(xs, outs):
        assert rel(o, exact(x)) <= bound, (name, rel(o, exact(x)))

for dt in (c64, torch.complex128):
    code, real = (G.F32, torch.float32) if dt == c64 else (G.F64, torch.float64)
    eps = 2e-7 if dt == c64 else 1e-15
    for n, b in ((1 << 15, 2), (1 << 17, 1), (1 << 18, 3), (1 << 20, 1), (1 << 21, 1), (1 << 24, 1)) if dt == c64 else ((1 << 14, 3), (1 << 16, 2), (1 << 21, 1)):
        l = n.bit_length() - 1
        xs = [torch.randn(b, n, dtype=dt, device="cuda", generator=g) for _ in range(CALLS if n < 1 << 22 else 2)]
        p = G.Plan(G.KIND_C2C, code, n, 0, b)
        buf, out = torch.empty_like(xs[0]), torch.empty_like(xs[0])
        check(f"c2c {n}", xs, out, lambda o, i: p.exec(o, i), lambda x: torch.fft.fft(x.to(torch.complex128)), eps * l)
        chain(f"c2c {n} there and back", [(p, False), (p, True)] * 2, xs, [torch.empty_like(buf) for _ in range(5)],
              lambda x: x.to(torch.complex128) * float(n) ** 2, 4 * eps * l)
    for n, b in ((1 << 14, 40), (1 << 16, 2), (1 << 17, 2), (1 << 18, 1), (1 << 19, 2), (1 << 20, 1), (1 << 22, 1), (1 << 23, 1)) if dt == c64 else ((1 << 16, 2), (1 << 18, 1)):
        l, m = n.bit_length() - 1, n // 2 + 1
        xs = [torch.randn(b, n, dtype=real, device="cuda", generator=g) for _ in range(CALLS if n < 1 << 22 else 2)]
        p = G.Plan(G.KIND_R2C, code, n, 0, b, G.FLAG_HALF_SPECTRUM)
        buf, spec, back = torch.empty_like(xs[0]), torch.empty(b, m, dtype=dt, device="cuda"), torch.empty_like(xs[0])
        check(f"r2c {n}", xs, spec, lambda o, i: p.exec(o, i), lambda x: torch.fft.rfft(x.double()), eps * l)
        fs = [torch.fft.rfft(x) for x in xs]
        check(f"c2r {n}", fs, back, lambda o, i: p.exec(o, i, True),
              lambda f: torch.fft.irfft(f.to(torch.complex128), n=n, norm="forward"), eps * l)
        chain(f"r2c c2r {n}", [(p, False), (p, True)], xs, [buf, spec, back], lambda x: x.double() * n, 2 * eps * l)
        outs = []
        for f in fs:  # the adjoint and the inverse in turn, through one workspace
            outs.append((p.adjoint(torch.empty_like(back), f), p.exec(torch.empty_like(back), f, True)))
        torch.cuda.synchronize()
        for f, (a, c) in zip(fs, outs):
            h = f.to(torch.complex128).clone()
            assert rel(c, torch.fft.irfft(h, n=n, norm="forward")) <= eps * l
            h[:, 1:-1] *= 0.5
            assert rel(a, torch.fft.irfft(h, n=n, norm="forward")) <= eps * l, n
for h, w in ((256, 256), (512, 33), (2048, 65), (4096, 100), (4096, 7)):
    xs = [torch.randn(h, w, dtype=c64, device="cuda", generator=g) for _ in range(CALLS)]
    buf, out = torch.empty_like(xs[0]), torch.empty_like(xs[0])
    v = G.Plan(G.KIND_VERT, G.F32, h, w, 1)
    check(f"columns {h}x{w}", xs, out, lambda o, i: v.exec(o, i),
          lambda x: torch.fft.fft(x.to(torch.complex128), dim=0), 2e-7 * 12)
    chain(f"columns {h}x{w} there and back", [(v, False), (v, True)] * 2, xs, [torch.empty_like(buf) for _ in range(5)],
          lambda x: x.to(torch.complex128) * float(h) ** 2, 8e-7 * 12)
for h, w in ((512, 64), (2048, 128), (4096, 64)):
    xs = [torch.randn(h, w, device="cuda", generator=g) for _ in range(CALLS)]
    buf, out = torch.empty_like(xs[0]), torch.empty(h, w // 2 + 1, dtype=c64, device="cuda")
    p = G.Plan(G.KIND_R2C_2D, G.F32, w, h, 1, G.FLAG_HALF_SPECTRUM)
    check(f"real 2D {h}x{w}", xs, out, lambda o, i: p.exec(o, i), lambda x: torch.fft.rfft2(x.double()), 2e-7 * 20)
assert G.device_error() == 0
"""


@pytest.mark.parametrize("env", [{}, {"GFFT_NO_TMA": "1"}, {"GFFT_NO_TMA": "1", "GFFT_PIPE": "0"}, {"GFFT_3PASS": "1"}],
                         ids=["default", "no_tma", "no_tma_no_pipe", "threepass"])
def test_calls_without_a_pause(gfft, env):
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT], env=dict(os.environ, **env), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
