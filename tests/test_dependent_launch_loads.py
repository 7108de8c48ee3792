"""Kernels that may start before their predecessor has finished (launched through launch_dependent) read
global memory with ordinary loads only: non-coherent ones (__ldg and its kin, or what the compiler makes
of a const __restrict__ pointer) are for memory that nobody writes while the kernel runs, and may be
moved ahead of the wait for the predecessor."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "blackwell_diffusion_rtx6000_5090_i2v_b200", "csrc")
NON_COHERENT = re.compile(r"__ld(?:g|ca|cg|cs)\b|ld\.global[\w.:]*\.nc|\bconst [^,;(){}]*\*\s*__restrict__")


def _source(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def _bodies(text):
    """(name, signature and body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        depth, i = 0, text.index("{", m.end())
        for j in range(i, len(text)):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            if depth == 0:
                yield m.group(1), text[m.start():j + 1]
                break


def _split():
    """Per file: the text of its dependent kernels with all helpers, and those kernels by name."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = _source(path)
        bodies = dict(_bodies(text))
        plain = {n for n in bodies if re.search(rf"\b{n}(?:<[^<>]*>)?<<<", text)
                 and not re.search(rf"launch_dependent\(\s*(?:\w+::)?{n}\b", text)}
        dependent = {n: b for n, b in bodies.items() if n not in plain}
        for n in plain:
            text = text.replace(bodies[n], "")
        yield os.path.basename(path), text, dependent


def test_the_scan_finds_the_kernels():
    found = {n for _, _, kernels in _split() for n in kernels}
    assert {"amax_bf16_kernel", "pack_rows_kernel", "quantize_small_kernel", "quantize_transposed_kernel",
            "norm_mod_kernel", "rope_warp_kernel", "rope_cta_kernel", "nvfp4_gemm_kernel"} == found


@pytest.mark.parametrize("name", [n for n, _, k in _split() if k])
def test_ordinary_loads_behind_the_wait(name):
    text, kernels = next((t, k) for n, t, k in _split() if n == name)
    assert not NON_COHERENT.findall(text)
    for kernel, body in kernels.items():
        assert "grid_dependency_wait()" in body, kernel


def test_shared_helpers():
    for path in glob.glob(os.path.join(CSRC, "*.cuh")):
        assert not NON_COHERENT.findall(_source(path)), path


def test_no_wait_where_nothing_is_overlapped():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = _source(path)
        for name, body in _bodies(text):
            if not re.search(rf"launch_dependent\(\s*(?:\w+::)?{name}\b", text) and f"{name}<<<" in text:
                assert "grid_dependency_wait" not in body, name
