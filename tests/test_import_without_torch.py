"""The binding without torch: importing it, loading the library and calling
the ABI need no torch, whatever importing torch would do."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("error", ["RuntimeError", "ImportError", "OSError"])
def test_abi_without_torch(tmp_path, error):
    (tmp_path / "torch.py").write_text(f"raise {error}('torch cannot be imported')\n")
    code = ("import sys; import genfft_gb300 as G; assert 'torch' not in sys.modules; "
            "print(G.lib().gfft_version(), G.max_fused_size(G.F32))")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, PYTHONPATH=f"{tmp_path}{os.pathsep}{ROOT}"),
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split()[1] == str(1 << 14)


def test_torch_is_bound_on_first_use():
    code = ("import genfft_gb300 as G, torch\n"
            "z = torch.zeros(2, dtype=torch.complex64)\n"
            "assert G._dtype_code(z) == G.F32 and G.torch is torch\n"
            "for bad in (torch.float16, torch.int32):\n"
            "    try: G._dtype_code(torch.zeros(2, dtype=bad))\n"
            "    except TypeError: pass\n"
            "    else: raise AssertionError\n"
            "try: G.fft(z)\n"
            "except ValueError: pass\n"
            "else: raise AssertionError\n")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, PYTHONPATH=ROOT), capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stderr
