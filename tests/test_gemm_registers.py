"""The GEMM's kernels keep what they work on in registers: a spill costs the epilogue, which bounds short K (the one that
asks for its parts, with 16 bytes of spills and without: 27280 x 3072 x 3072 with bias, GELU and residual 148 and 141 us)."""
import os
import re
import subprocess

import pytest

from blackwell_diffusion_rtx6000_5090_i2v_b200 import build


def test_no_spills(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    log = subprocess.run([nvcc, *build._host_cxx(), *build.NVCC_FLAGS, "-Xptxas=-v", "-c",
                          os.path.join(build.CSRC, "gemm_sm100.cu"), "-o", str(tmp_path / "gemm.o")],
                         check=True, capture_output=True, text=True).stderr
    spills = re.findall(r"Function properties for (\S*nvfp4_gemm_kernel\S*)\n.*?(\d+) bytes spill stores", log)
    assert len(spills) >= 19                        # 3 tilings x 6 epilogues, and one that asks at least
    assert [s for s in spills if s[1] != "0"] == []
