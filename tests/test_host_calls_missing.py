"""The package without its extension module, or with one built for another torch: it imports, says so, and every
native call declines, which leaves the call to the Python code behind it."""
import subprocess
import sys

import pytest

PACKAGE = "blackwell_diffusion_rtx6000_5090_i2v_b200"
CALLS = ["linear", "quantize", "norm_quantize", "dequantize", "gemm", "attention"]


def _run(prepare):
    code = f"""
import sys, types, warnings
import torch, {PACKAGE}
{prepare}
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    from {PACKAGE} import _native as N, nvfp4_linear_cpp, nvfp4, dit
assert any("native calls are not in use" in str(w.message) for w in seen), seen
assert all(getattr(N.host, n)(1, 2, 3) is None for n in {CALLS})
N.host.set_status(0, torch.zeros(1))
print("declined")
"""
    return subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)


@pytest.mark.parametrize("prepare", [
    f"sys.modules['{PACKAGE}._host_calls'] = None",                                     # not there, or not loadable
    f"m = sys.modules['{PACKAGE}._host_calls'] = types.ModuleType('m'); m.built_for = 'torch 1.0, Python 3.0'; "
    f"{PACKAGE}._host_calls = m",
    f"m = sys.modules['{PACKAGE}._host_calls'] = types.ModuleType('m'); {PACKAGE}._host_calls = m",
])
def test_every_call_declines(prepare):
    r = _run(prepare)
    assert r.returncode == 0 and "declined" in r.stdout, r.stderr


def test_the_built_module_is_in_use():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N, build
    assert N.host.built_for == build.host_built_for() and not build.host_is_stale()


def test_a_module_for_another_torch_is_stale(monkeypatch):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import build
    monkeypatch.setattr(build, "host_built_for", lambda: "torch 99.0, Python 3.99")
    assert build.host_is_stale()
