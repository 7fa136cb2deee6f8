"""Which calls skip the autograd.Function (torchfft._plain), on the CPU."""
import torch

from genfft_gb300 import torchfft as GT


def test_traced_calls_are_not_plain():
    x = torch.ones(2)
    seen = []

    def f(v):
        seen.append(GT._plain(v))
        return v + 1

    torch.jit.trace(f, x, check_trace=False)
    assert GT._plain(x) and seen == [False]
