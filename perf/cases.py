"""The workloads whose speed this library is held to.

listed() names them: single small transforms, ordinary batches and the
largest ones; C2C, real, 2D, column and ragged transforms; forward and
inverse, and the backward passes; fp32 and fp64; odd batch and column counts.
draw() gives others from the same ranges.  prepare() makes a case's inputs
and keeps the plan a program would keep, run() is one pass through the
public entry points, work() the bytes and operations it cannot do without,
exact() its results in 64 bits.
"""
from __future__ import annotations

import math

import torch

import genfft_gb300 as G
from genfft_gb300 import autograd as GA
from genfft_gb300 import torchfft as GT

# real and complex types of a precision
TYPES = {"f32": (torch.float32, torch.complex64), "f64": (torch.float64, torch.complex128)}
CODE = {"f32": G.F32, "f64": G.F64}


def listed():
    return [
        # one signal at a time, as an interactive program or a control loop
        # has it: latency of the call
        {"name": "single_1024", "kind": "c2c", "dtype": "f32", "n": 1024, "batch": 1, "api": "module"},
        # spectra of many short frames, the library's headline batch
        {"name": "frames_4096", "kind": "c2c", "dtype": "f32", "n": 4096, "batch": 16384, "api": "plan"},
        # long frames, an odd number of them
        {"name": "frames_16384", "kind": "c2c", "dtype": "f32", "n": 16384, "batch": 1501, "api": "module"},
        # records longer than a CTA holds (multi-pass), an odd number of them
        {"name": "records_131072", "kind": "c2c", "dtype": "f32", "n": 131072, "batch": 333, "api": "module"},
        # few very long records
        {"name": "records_4194304", "kind": "c2c", "dtype": "f32", "n": 1 << 22, "batch": 32, "api": "plan"},
        # double precision
        {"name": "records_f64_65536", "kind": "c2c", "dtype": "f64", "n": 65536, "batch": 512, "api": "plan"},
        # real signals to the half spectrum and back
        {"name": "real_1048576", "kind": "real", "dtype": "f32", "n": 1 << 20, "batch": 64, "norm": "backward"},
        # a complex image, forward and unscaled inverse
        {"name": "image_4096", "kind": "c2d", "dtype": "f32", "h": 4096, "w": 4096, "batch": 1, "norm": "unscaled"},
        # a real image to the half spectrum and back
        {"name": "real_image_4096", "kind": "r2d", "dtype": "f32", "h": 4096, "w": 4096, "batch": 1,
         "norm": "ortho"},
        # columns of a matrix with an odd number of them (rows not aligned
        # to 16 bytes)
        {"name": "columns_2048", "kind": "vert", "dtype": "f32", "h": 2048, "w": 1001},
        # a spectral-convolution layer in training: half spectrum, filter,
        # back, and the gradients of signal and filter
        {"name": "conv_layer_8192", "kind": "conv", "dtype": "f32", "n": 8192, "batch": 6001},
        # thousands of transforms of uneven size in one call, and the
        # adjoint of all of them
        {"name": "ragged_10000", "kind": "ragged", "dtype": "f32", "count": 10000, "lo": 6, "hi": 18,
         "sizes_seed": 1},
    ]


def _count(rng, most):
    """1 .. most, spread over the logarithm."""
    return max(1, min(most, int(round(2.0 ** rng.uniform(0.0, math.log2(most))))))


def draw(rng):
    kind = rng.choice(["c2c", "c2c", "c2c", "real", "real", "c2d", "r2d", "vert", "conv", "ragged"])
    dtype = "f32" if kind in ("conv", "ragged") or rng.random() < 0.75 else "f64"
    most = 1 << (26 if dtype == "f32" else 24)  # points of a pass
    if kind == "ragged":
        lo = rng.randint(4, 10)
        return {"kind": kind, "dtype": dtype, "count": 100 + _count(rng, 4000), "lo": lo, "hi": rng.randint(lo + 2, 18),
                "sizes_seed": rng.randrange(1 << 20)}
    if kind == "vert":
        h = 1 << rng.randint(5, 13)
        return {"kind": kind, "dtype": dtype, "h": h, "w": 16 + _count(rng, (most >> 1) // h)}
    if kind in ("c2d", "r2d"):
        h, w = 1 << rng.randint(5, 12), 1 << rng.randint(5, 12)
        return {"kind": kind, "dtype": dtype, "h": h, "w": w, "batch": _count(rng, most // (h * w)),
                "norm": rng.choice(["unscaled", "backward", "ortho"] if kind == "c2d" else ["backward", "ortho"])}
    n = 1 << rng.randint(5, 14 if kind == "conv" else 23)
    case = {"kind": kind, "dtype": dtype, "n": n, "batch": _count(rng, most // n)}
    if kind == "c2c":
        case["api"] = rng.choice(["module", "plan"])
    if kind == "real":
        case["norm"] = rng.choice(["backward", "ortho"])
    return case


def _shape(case):
    """(rows..., last) of the case's input."""
    k = case["kind"]
    if k == "vert":
        return (case["h"], case["w"])
    if k in ("c2d", "r2d"):
        return (case["batch"], case["h"], case["w"])
    return (case["batch"], case["n"])


def _sizes(case):
    """Power-of-two sizes, log-uniform between 2^lo and 2^hi."""
    g = torch.Generator().manual_seed(case["sizes_seed"])
    return [1 << int(k) for k in torch.randint(case["lo"], case["hi"] + 1, (case["count"],), generator=g)]


def _inputs(case, seed):
    """Standard-normal signals on the GPU; where a backward pass belongs to
    the case, the filter and the gradient that arrives from the loss too."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    real, cplx = TYPES[case["dtype"]]

    def normal(shape, dtype):
        return torch.randn(*shape, dtype=dtype, device="cuda", generator=gen)

    k = case["kind"]
    if k == "ragged":
        total = sum(_sizes(case))
        return {"x": normal((total,), cplx), "gy": normal((total,), cplx)}
    if k == "conv":
        n = case["n"]
        return {"x": normal(_shape(case), real), "f": normal((n // 2 + 1,), cplx), "gy": normal(_shape(case), real)}
    return {"x": normal(_shape(case), real if k in ("real", "r2d") else cplx)}


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    if case["kind"] == "c2c" and case["api"] == "plan":
        s["plan"] = G.Plan(G.KIND_C2C, CODE[case["dtype"]], case["n"], 0, case["batch"])
        s["y"], s["z"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif case["kind"] == "ragged":
        s["plan"] = G.RaggedPlan(_sizes(case))
        s["x"].requires_grad_()
    elif case["kind"] == "conv":
        s["x"].requires_grad_()
        s["f"].requires_grad_()
    return s


def run(s):
    case, x = s["case"], s["x"]
    kind = case["kind"]
    if kind == "c2c" and case["api"] == "plan":
        s["plan"].exec(s["y"], x)
        s["plan"].exec(s["z"], s["y"], True)
        return s["y"], s["z"]
    if kind == "c2c":
        y = G.fft(x)
        return y, G.ifft(y)
    if kind == "real":
        y = GT.rfft(x, norm=case["norm"])
        return y, GT.irfft(y, n=case["n"], norm=case["norm"])
    if kind == "c2d" and case["norm"] == "unscaled":
        y = G.fft2(x)
        return y, G.fft2(y, True)
    if kind == "c2d":
        y = GT.fft2(x, norm=case["norm"])
        return y, GT.ifft2(y, norm=case["norm"])
    if kind == "r2d":
        y = GT.rfft2(x, norm=case["norm"])
        return y, GT.irfft2(y, s=(case["h"], case["w"]), norm=case["norm"])
    if kind == "vert":
        y = G.fft_vert(x)
        return y, G.fft_vert(y, True)
    if kind == "conv":
        y = GT.irfft(GT.rfft(x) * s["f"], n=case["n"])
        gx, gf = torch.autograd.grad(y, (x, s["f"]), s["gy"])
        return y.detach(), gx, gf
    y = GA.ragged_fft(x, s["plan"])
    (gx,) = torch.autograd.grad(y, x, s["gy"])
    return y.detach(), gx


def work(case):
    """Bytes: every transform's input read once and its output written once
    (a real input as reals, its spectrum as the half spectrum).  Operations:
    5 N log2 N a complex transform of N points, half that a real one."""
    rb = 4 if case["dtype"] == "f32" else 8
    k = case["kind"]
    if k == "ragged":
        sizes = _sizes(case)
        return {"bytes": 2.0 * sum(sizes) * 4 * rb, "flops": 2.0 * sum(5.0 * n * math.log2(n) for n in sizes)}
    shape = _shape(case)
    points = float(math.prod(shape))
    if k == "vert":
        return {"bytes": 2 * points * 4 * rb, "flops": 2 * 5.0 * points * math.log2(case["h"])}
    n = case["h"] * case["w"] if k in ("c2d", "r2d") else case["n"]
    if k in ("c2c", "c2d"):
        return {"bytes": 2 * points * 4 * rb, "flops": 2 * 5.0 * points * math.log2(n)}
    m = shape[-1] // 2 + 1
    one = points * rb + points / shape[-1] * m * 2 * rb
    flops = 2.5 * points * math.log2(n)
    return {"bytes": (4 if k == "conv" else 2) * one, "flops": (4 if k == "conv" else 2) * flops}


def exact(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    x = s["x"].to(torch.float64 if k in ("real", "r2d", "conv") else torch.complex128)
    if k == "c2c":
        y = torch.fft.fft(x)
        return y, torch.fft.ifft(y, norm="forward")
    if k == "real":
        y = torch.fft.rfft(x, norm=case["norm"])
        return y, torch.fft.irfft(y, n=case["n"], norm=case["norm"])
    if k == "c2d":
        unscaled = case["norm"] == "unscaled"
        y = torch.fft.fft2(x, norm="backward" if unscaled else case["norm"])
        return y, torch.fft.ifft2(y, norm="forward" if unscaled else case["norm"])
    if k == "r2d":
        y = torch.fft.rfft2(x, norm=case["norm"])
        return y, torch.fft.irfft2(y, s=(case["h"], case["w"]), norm=case["norm"])
    if k == "vert":
        y = torch.fft.fft(x, dim=0)
        return y, torch.fft.ifft(y, dim=0, norm="forward")
    if k == "conv":
        f, x = s["f"].to(torch.complex128).requires_grad_(), x.requires_grad_()
        y = torch.fft.irfft(torch.fft.rfft(x) * f, n=case["n"])
        gx, gf = torch.autograd.grad(y, (x, f), s["gy"].to(torch.float64))
        return y.detach(), gx, gf
    # ragged: the transforms of one size together
    gy = s["gy"].to(torch.complex128)
    y, gx = torch.empty_like(x), torch.empty_like(x)
    sizes = torch.tensor(_sizes(case))
    offsets = torch.cumsum(sizes, 0) - sizes
    for n in sorted(set(sizes.tolist())):
        at = offsets[sizes == n].cuda()
        for part in at.split(max(1, (1 << 25) // n)):
            i = part[:, None] + torch.arange(n, device="cuda")[None, :]
            y[i] = torch.fft.fft(x[i])
            gx[i] = torch.fft.ifft(gy[i], norm="forward")
    return y, gx
