"""GFFT_NO_TMA=1 selects kernels that use no TMA copies, with the same bits,
in the persistent fused, pipelined real and ragged paths too; inputs that no
tensor map describes take the same way."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, numpy as np, torch
sys.path.insert(0, %r)
import genfft_gb300 as G
g = torch.Generator(device="cuda").manual_seed(7)
outs = {}
def run():
    for n, b in ((1 << 13, 1000), (1 << 14, 200)):
        x = torch.randn(b, n, dtype=torch.complex64, device="cuda", generator=g)
        outs[f"c2c_{n}"] = G.fft(x)
    for n, b in ((1 << 15, 160), (1 << 18, 3), (1 << 19, 2), (1 << 20, 2), (1 << 21, 1), (1 << 22, 1)):
        m = n // 2 + 1
        p = G.Plan(G.KIND_R2C, G.F32, n, 0, b, G.FLAG_HALF_SPECTRUM)
        x = torch.randn(b, n, device="cuda", generator=g)
        for off in (0, 1):
            f = torch.randn(b * m + 1, dtype=torch.complex64, device="cuda", generator=g)[off:off + b * m].view(b, m)
            outs[f"r2c_{n}_{off}"] = p.exec(torch.empty_like(f), x)
            outs[f"c2r_{n}_{off}"] = p.exec(torch.empty_like(x), f, True)
            outs[f"adj_{n}_{off}"] = p.adjoint(torch.empty_like(x), f, False)
    sizes = [1 << 13] * 1024 + [1 << 16] * 128 + [64] * 10
    r = G.RaggedPlan(sizes)
    x = torch.randn(r.elements, dtype=torch.complex64, device="cuda", generator=g)
    y = r.exec(torch.empty_like(x), x)
    exact = torch.fft.fft(x[:1 << 23].view(1024, -1).to(torch.complex128))
    assert float((y[:1 << 23].view(1024, -1) - exact).norm() / exact.norm()) <= 2e-7 * 13
    torch.cuda.synchronize()
    return r.launches
launches = run()
assert G.device_error() == 0, "device-side timeout"
np.savez(sys.argv[1], launches=launches, **{k: v.cpu().numpy() for k, v in outs.items()})
"""


def test_no_tma_kernels_and_bits(gfft, tmp_path):
    """(the ragged batch takes four launches with TMA, the persistent ragged
    kernel's one without)"""
    import numpy as np
    res = {}
    for mode in ("0", "1"):
        out = str(tmp_path / f"{mode}.npz")
        r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT, out], env=dict(os.environ, GFFT_NO_TMA=mode),
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        res[mode] = np.load(out)
    for k in res["0"].files:
        if k not in ("launches",):
            a, b = res["0"][k], res["1"][k]
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), (k, np.max(np.abs(a - b)))
    assert int(res["0"]["launches"]) == 4 and int(res["1"]["launches"]) == 1


@pytest.mark.parametrize("logn", [18, 21])
def test_bins_too_far_apart_for_a_tensor_map(gfft, logn):
    """A plan of one transform may name any distance between transforms,
    2^40 bytes among them, which a tensor map cannot hold."""
    import torch
    n, m = 1 << logn, (1 << (logn - 1)) + 1
    f = torch.randn(m, dtype=torch.complex64, device="cuda")
    far = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, 1, gfft.FLAG_HALF_SPECTRUM, 1, n, 1, 1 << 37)
    near = gfft.Plan(gfft.KIND_R2C, gfft.F32, n, 0, 1, gfft.FLAG_HALF_SPECTRUM)
    a, b = (p.adjoint(torch.empty(n, device="cuda"), f, False) for p in (far, near))
    assert torch.equal(a, b)
    h = f.to(torch.complex128).clone()
    h[1:-1] *= 0.5
    exact = torch.fft.irfft(h, n=n, norm="forward")
    assert float((a - exact).norm() / exact.norm()) <= 2e-7 * logn
