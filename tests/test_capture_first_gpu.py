"""A plan's first exec may be inside a stream capture: what a launch needs on
the device is there when the plan has been created.  Each case runs in a
process of its own, whose first exec of all is the captured one."""
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
kind, n0, n1, batch = sys.argv[1], *map(int, sys.argv[2:5])
c64, real = torch.complex64, kind in ("r2c", "r2c_2d")
shape = (batch, n0) if kind in ("c2c", "r2c") else (batch, n0, n1) if kind == "vert" else (batch, n1, n0)
x = torch.randn(*shape, dtype=torch.float32 if real else c64, device="cuda")
code = {"c2c": G.KIND_C2C, "r2c": G.KIND_R2C, "c2c_2d": G.KIND_C2C_2D, "r2c_2d": G.KIND_R2C_2D, "vert": G.KIND_VERT}
p = G.Plan(code[kind], G.F32, n0, n1, batch, G.FLAG_HALF_SPECTRUM if real else 0)
exact = {"c2c": lambda v: torch.fft.fft(v), "r2c": lambda v: torch.fft.rfft(v), "vert": lambda v: torch.fft.fft(v, dim=1),
         "c2c_2d": lambda v: torch.fft.fft2(v), "r2c_2d": lambda v: torch.fft.rfft2(v)}[kind](x.double() if real else x.to(torch.complex128))
y = torch.empty(exact.shape, dtype=c64, device="cuda")
z = torch.empty_like(x)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    p.exec(y, x)
    if kind == "r2c":
        p.exec(z, y, True)
graph.replay()
torch.cuda.synchronize()
n = n0 * max(n1, 1) if kind.endswith("2d") else n0
bound = 2e-7 * (n.bit_length() - 1)
rel = lambda a, b: float((a.to(b.dtype) - b).norm() / b.norm())
assert rel(y, exact) <= bound, rel(y, exact)
if kind == "r2c":
    assert rel(z, torch.fft.irfft(y.to(torch.complex128), n=n0, norm="forward")) <= bound
assert G.device_error() == 0
"""


@pytest.mark.parametrize("kind,n0,n1,batch", [
    ("c2c", 1 << 12, 0, 2000), ("c2c", 1 << 13, 0, 1000),  # persistent fused kernels
    ("c2c", 1 << 15, 0, 2), ("c2c", 1 << 17, 0, 3), ("c2c", 1 << 21, 0, 1),  # column and row passes
    ("r2c", 1 << 15, 0, 400),        # persistent fused kernels
    ("r2c", 1 << 18, 0, 2),          # real passes
    ("c2c_2d", 512, 1024, 1), ("r2c_2d", 512, 1024, 1), ("vert", 2048, 700, 1)])
def test_first_exec_is_captured(gfft, kind, n0, n1, batch):
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT, kind, str(n0), str(n1), str(batch)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
