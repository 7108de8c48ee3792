"""Kernels that may start before their predecessor has finished (launched with programmatic stream serialization)
read global memory with ordinary loads only: non-coherent ones (__ldg and its kin, or what the compiler makes
of a const __restrict__ pointer) are for memory that nobody writes while the kernel runs, and may be
moved ahead of the wait for the predecessor.  Which kernels these are is read off the launches: launch_dependent(),
a cudaLaunchKernelEx() in a file that asks for that attribute, <<<>>> for a plain one; a cooperative launch (a kernel
whose grid meets) is a plain one too."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "blackwell_diffusion_rtx6000_5090_i2v_b200", "csrc")
NON_COHERENT = re.compile(r"__ld(?:g|ca|cg|cs)\b|ld\.global[\w.:]*\.nc|\bconst [^,;(){}]*\*\s*__restrict__")
SERIALIZED = "cudaLaunchAttributeProgrammaticStreamSerialization"
MEETS = "this_grid().sync()"


def _source(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def _bodies(text):
    """(name, signature and body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?!\d)(?=[^()]*(?:const|\w+\s*\*))", text):
        depth, i = 0, text.index("{", m.end())
        for j in range(i, len(text)):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            if depth == 0:
                yield m.group(1), text[m.start():j + 1]
                break


def _launches(text, name):
    """How the kernel of this name is launched: a subset of {"plain", "dependent"}."""
    kinds = set()
    if re.search(rf"\b{name}(?:<[^<>]*>)?<<<", text):
        kinds.add("plain")
    if re.search(rf"launch_dependent\(\s*(?:\w+::)?{name}\b", text) or \
            re.search(rf"auto kernel = {name}\b[^;]*;(?:(?!auto kernel).)*?launch_dependent\(kernel", text, re.S):
        kinds.add("dependent")
    if re.search(rf"cudaLaunchKernelEx\(\s*&cfg,\s*{name}\b", text) or \
            re.search(rf"auto kernel = {name}\b[^;]*;(?:(?!auto kernel).)*?cudaLaunchKernelEx\(&cfg, kernel", text, re.S):
        kinds.add("dependent" if SERIALIZED in text else "plain")
    return kinds


def _files():
    """Per file: its name, its text and its kernels by name."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = _source(path)
        yield os.path.basename(path), text, dict(_bodies(text))


def _split():
    """Per file: the text of its dependent kernels with all helpers, and those kernels by name."""
    for name, text, bodies in _files():
        dependent = {n: b for n, b in bodies.items() if "dependent" in _launches(text, n)}
        for n in bodies.keys() - dependent.keys():
            text = text.replace(bodies[n], "")
        yield name, text, dependent


def test_the_scan_finds_the_kernels():
    found = {n for _, _, kernels in _split() for n in kernels}
    assert {"amax_bf16_kernel", "pack_rows_kernel", "quantize_small_kernel", "quantize_transposed_kernel",
            "norm_mod_kernel", "rope_warp_kernel", "rope_cta_kernel", "nvfp4_gemm_kernel", "attention_kernel"} == found
    for _, text, bodies in _files():
        assert len(bodies) == len(re.findall(r"__global__", text))
        for n in bodies.keys() - {"linear_scratch_anchor"}:      # never launched
            assert _launches(text, n), f"{n}: how it is launched is not seen"


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
    for _, text, bodies in _files():
        for name, body in bodies.items():
            if _launches(text, name) == {"plain"}:
                assert "grid_dependency_wait" not in body, name


def test_kernels_whose_grid_meets_are_launched_cooperatively():
    meeting = {n for _, _, bodies in _files() for n, b in bodies.items() if MEETS in b}
    assert meeting == {"norm_mod_resident_kernel", "quantize_resident_kernel"}
    for _, text, bodies in _files():
        for n in bodies.keys() & meeting:
            launch = text[text.index("int launch_resident("):]
            launch = launch[:launch.index("\n}\n")]
            assert n in launch and "cudaLaunchAttributeCooperative" in launch and SERIALIZED not in launch
            assert _launches(text, n) == {"plain"} and not re.search(rf"\b{n}(?:<[^<>]*>)?<<<", text)


def test_the_launch_that_may_start_early():
    """Attention's kernel alone lets the next launch start before its end, and only where the next is its own of the
    shared blocks, which waits for it before it ends itself."""
    for name, text, bodies in _files():
        for kernel, body in bodies.items():
            if "griddepcontrol.launch_dependents" in body:
                assert kernel == "attention_kernel"
                assert re.search(r"if \(p\.lets_next_start\) asm volatile\(\"griddepcontrol\.launch_dependents;", body)
                assert "if (p.follows) grid_dependency_wait();" in body
                assert "w.lets_next_start = parts > 1 && w.end == whole" in text
                assert re.search(r"numAttrs = p\.follows \? 1 : 0", text)
