"""Long transforms of a ragged batch on the pipelined passes: which batches
take them, against FFTs in 64 bits, and against the persistent kernel (input
off a 16-byte boundary takes it for every size)."""
import pytest

pytestmark = pytest.mark.gpu

POINTS = 1 << 23  # of one size, from which its transforms take the passes
MIX = ([64, 16] + [1 << 18] * (POINTS >> 18) + [32, 1 << 13] + [1 << 17] * (POINTS >> 17) + [4096] +
       [1 << 16] * ((POINTS >> 16) + 1) + [1 << 14, 1 << 15, 16])
BATCHES = [  # sizes, kernels of an exec
    (MIX, 7),
    ([1 << 17] * ((POINTS >> 17) + 3), 2),                 # nothing else
    ([48 // 3] + [1 << 16] * (POINTS >> 16), 3),
    ([1 << 18] * (POINTS >> 18) + [1 << 17, 2], 3),         # only one size has enough
    ([1 << 17] * ((POINTS >> 17) - 1), 1),                 # one too few
    ([8] + [1 << 16] * (POINTS >> 16), 1),                  # starts off multiples of 16
    ([16] + [1 << 14] * (POINTS >> 14) + [64] + [1 << 13] * ((POINTS >> 13) + 1), 3),  # the fused kernel
    ([1 << 13] * (POINTS >> 13), 1),
    ([16] + [1 << 14] * ((POINTS >> 14) - 1), 1),
    ([1] + [1 << 16] * (POINTS >> 16), 1),                  # one-point transforms: no copies at all
]


def check(plan, x, y, inverse):
    import math
    import torch
    for o, n in zip(plan.offsets, plan.sizes):
        a = x[o:o + n].to(torch.complex128)
        ref = torch.fft.ifft(a, norm="forward") if inverse else torch.fft.fft(a)
        err = float((y[o:o + n] - ref).norm() / ref.norm())
        assert err <= 2e-7 * max(1, math.log2(n)), (n, o, inverse, err)


@pytest.mark.parametrize("case", range(len(BATCHES)))
@pytest.mark.parametrize("inverse", [False, True])
def test_long_transforms(gfft, case, inverse):
    import torch
    sizes, launches = BATCHES[case]
    plan = gfft.RaggedPlan(sizes)
    assert plan.launches == launches
    g = torch.Generator(device="cuda").manual_seed(case)
    buf = torch.randn(plan.elements + 1, dtype=torch.complex64, device="cuda", generator=g)
    x, y = buf[:-1], torch.full((plan.elements + 4,), 7.0, dtype=torch.complex64, device="cuda")
    plan.exec(y[2:-2], x, inverse)
    check(plan, x, y[2:-2], inverse)
    assert bool((y[:2] == 7).all()) and bool((y[-2:] == 7).all())
    # the persistent kernel for all of them
    odd = torch.empty_like(buf)[1:]
    odd.copy_(x)
    z = torch.empty_like(x)
    plan.exec(z, odd, inverse)
    check(plan, x, z, inverse)
    # in place, twice through the same graph
    for _ in range(2):
        w = x.clone()
        plan.exec(w, w, inverse)
        assert torch.equal(w, y[2:-2])
    assert gfft.device_error() == 0
