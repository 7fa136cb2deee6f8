"""Which plans the module functions keep from call to call (stand-ins for the
plan and the library, on the CPU)."""
import ctypes
import types

import pytest
import torch

import genfft_gb300 as G


@pytest.fixture
def made(monkeypatch):
    made = []

    class Plan:
        handle = None

        def __init__(self, *args):
            made.append(args)

    def workspace_size(handle, size):
        ctypes.cast(size, ctypes.POINTER(ctypes.c_size_t))[0] = 0
        return 0

    monkeypatch.setattr(G, "Plan", Plan)
    monkeypatch.setattr(G, "lib", lambda: types.SimpleNamespace(gfft_plan_workspace_size=workspace_size))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(G, "_STATELESS", type(G._STATELESS)())
    return made


@pytest.mark.parametrize("kind", [G.KIND_C2C_2D, G.KIND_R2C_2D])
@pytest.mark.parametrize("knob", ["GFFT_COL_SPLIT", "GFFT_COL_MAXC"])
def test_column_knobs_are_read_on_every_call(made, monkeypatch, kind, knob):
    monkeypatch.delenv(knob, raising=False)
    a = G._call_plan(kind, G.F32, 64, 2048, 1)
    assert G._call_plan(kind, G.F32, 64, 2048, 1) is a
    monkeypatch.setenv(knob, "1")
    b = G._call_plan(kind, G.F32, 64, 2048, 1)
    assert b is not a and G._call_plan(kind, G.F32, 64, 2048, 1) is b
    monkeypatch.delenv(knob)
    assert G._call_plan(kind, G.F32, 64, 2048, 1) is a
    assert len(made) == 2


def test_plans_are_told_apart_and_bounded(made):
    for i in range(G._STATELESS_MAX + 5):
        G._call_plan(G.KIND_R2C, G.F32, 64, 0, i + 1)
    assert len(G._STATELESS) == G._STATELESS_MAX and len(made) == G._STATELESS_MAX + 5
    G._call_plan(G.KIND_R2C, G.F32, 64, 0, G._STATELESS_MAX + 5)
    assert len(made) == G._STATELESS_MAX + 5
