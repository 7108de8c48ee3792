"""The norm's kernels for calls with both vectors of a kind against those that ask for each: a shift or bias of zeros
changes no value.  Widths whose threads all have blocks and widths that leave some without, odd row counts, both the one-launch
form and the two sweeps."""
import pytest
import torch

from helpers import student_t_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 512), (3, 3072), (65, 528), (301, 5120), (20001, 3072), (6001, 6384), (70001, 512)])
@pytest.mark.parametrize("kind", ["modulation", "affine", "rms", "all four"])
def test_zeros_change_nothing(rows, cols, kind):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), rows, scale=1.5, device="cuda") if rows * cols < 1 << 24 else \
        torch.randn(rows, cols, generator=torch.Generator("cuda").manual_seed(rows), device="cuda").to(torch.bfloat16)
    v = torch.randn(cols, generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    a, b = ("weight", "bias") if kind == "affine" else ("scale", "shift")
    rest = {"weight": 1 + v.flip(0) / 8, "bias": v.roll(1)} if kind == "all four" else {}
    one = nv.FP4Tensor.from_norm_mod(x, rms=kind == "rms", **{a: v}, **rest)
    both = nv.FP4Tensor.from_norm_mod(x, rms=kind == "rms", **{a: v, b: torch.zeros_like(v)}, **rest)
    nv.check_status()
    assert torch.equal(one.global_amax(), both.global_amax())
    assert torch.equal(one.scale_factors_swizzled(), both.scale_factors_swizzled())
    # a negative zero plus zero is a positive one: magnitudes, and signs of what is not zero
    d, e = one.quantized_data(), both.quantized_data()
    assert torch.equal(d & 0x77, e & 0x77)
    for shift in (0, 4):
        there = ((d >> shift) & 7) != 0
        assert torch.equal(((d >> shift) & 8)[there], ((e >> shift) & 8)[there])
