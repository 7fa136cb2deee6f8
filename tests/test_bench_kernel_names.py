"""`roofline.kernel` names the kernels a workload's batch runs: the rule it
repeats is the library's own."""
import os
import re
import sys
import types

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
G = types.SimpleNamespace(F32=0, F64=1, max_fused_size=lambda d: (1 << 14) if d == 0 else (1 << 13))


@pytest.fixture(scope="module")
def bench():
    import bench as B
    return B


def test_the_rule_is_the_librarys(bench):
    """Waves and groups as csrc/fused_tma.cu spells them."""
    src = open(os.path.join(ROOT, "genfft_gb300", "csrc", "fused_tma.cu")).read()
    groups = {int(a): (int(b), int(c)) for a, b, c in re.findall(r"make_entry<(\d+), (\d+), (\d+)>\(\)", src)}
    assert "logn == 14 ? 1 : logn == 13 ? 3 : real ? 2 : 4" in src
    waves = {12: (4, 2), 13: (3, 3), 14: (1, 1)}
    assert {l: tuple(w * g for w, g in zip(waves[l], groups[l])) for l in groups} == bench.FUSED_TMA_WAVES


@pytest.mark.parametrize("args,name", [
    (("c2c", "f32", 4096, 0, 1, 16384), "k_fused_tma"), (("c2c", "f32", 4096, 0, 1, 1824), "k_c2c_fused"),
    (("c2c", "f32", 4096, 0, 1, 1825), "k_fused_tma"), (("c2c", "f32", 1024, 0, 1, 65536), "k_c2c_fused"),
    (("c2c", "f64", 4096, 0, 1, 8192), "k_c2c_fused"), (("c2c", "f32", 16384, 0, 1, 153), "k_fused_tma"),
    (("r2c", "f32", 1 << 20, 0, 2, 64), "k_colpass_tma + k_rowdit_pipe"),
    (("r2c", "f32", 1 << 17, 0, 2, 64), "k_colpass_tma + k_rowpass_dit"),
    (("r2c", "f32", 8192, 0, 1, 1217), "k_fused_tma"), (("r2c", "f32", 8192, 0, 1, 1216), "k_r2c_fused"),
    (("c2r", "f32", 1 << 20, 0, 2, 64), "k_c2rcol_pipe + k_rowpass_tma"),
    (("c2r", "f32", 1 << 23, 0, 3, 4), "C2R pre-pass + four-step inverse"),
    (("c2d", "f32", 4096, 0, 2, 1, 4096), "k_fused_tma (rows) + k_colpass_tma (columns)"),
    (("c2d", "f32", 512, 0, 2, 1, 512), "k_c2c_fused (rows) + k_colpass_tma (columns)"),
    (("r2d", "f32", 4096, 0, 2, 1, 4096), "k_r2c_fused (rows) + k_colpass_tma (columns)")])
def test_names(bench, args, name):
    assert bench.kernel_name(G, *args, sms=152) == name


def test_launch_counts_of_three_groups(bench):
    """Six launches at 2^22 are three groups of a pair unless GFFT_3PASS asks
    for three passes."""
    assert bench.kernel_name(G, "c2c", "f32", 1 << 22, 0, 6, 96, sms=152, three_pass=False).startswith("k_colpass_tma")
    assert bench.kernel_name(G, "c2c", "f32", 1 << 22, 0, 6, 96, sms=152, three_pass=True).startswith("k3_col")
