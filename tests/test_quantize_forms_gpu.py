"""The quantizer's three forms (one cluster, rows, flat) at the edges between them, all against the CPU
oracle, byte for byte, pad of the swizzled scales included."""
import numpy as np
import pytest
import torch

from helpers import bits_of, student_t_bf16

pytestmark = pytest.mark.gpu


def _check(oracle, x, t):
    packed, scales, amax = oracle.quantize(bits_of(x))
    assert float(t.global_amax()) == amax
    assert np.float32(t.global_scale().item()) == np.float32(oracle.global_decode_scale(amax))
    assert np.array_equal(t.quantized_data().cpu().numpy(), packed.reshape(-1))
    assert np.array_equal(t.scale_factors().cpu().numpy(), scales.reshape(-1))
    assert np.array_equal(t.scale_factors_swizzled().cpu().numpy(), oracle.swizzle_scales(scales, x.shape[1]))


@pytest.mark.parametrize("rows,cols", [
    (1, 16), (1, 18432), (2, 8192), (33, 512), (128, 64),                  # one CTA to eight
    (31, 16896), (32, 16384), (33, 15888),                                 # around 524288 elements
    (1, 131072), (1, 131088), (3, 131088), (1, 524288),                    # mostly pad: 2 MB of it, and past that
    (31, 17408), (32, 16912), (40, 13840), (200, 3072), (171, 3088),       # past it: flat / rows
    (1000, 1136), (1000, 1152), (1000, 1280), (1000, 1488),                # the narrowest rows of that form
    (1000, 1520), (1000, 1536), (1000, 1552), (4096, 144), (70000, 16)])   # narrow rows
def test_forms_against_the_oracle(oracle, rows, cols):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), rows + cols)
    t = nv.FP4Tensor.from_bfloat16(x.cuda())
    _check(oracle, x, t)
    # the same with the maximum already known (no amax pass)
    _check(oracle, x, nv.FP4Tensor.from_bfloat16(x.cuda(), amax=t.global_amax()))


# small, flat and, past 524288 elements and with 96 threads or more a row, rows form
@pytest.mark.parametrize("rows,cols", [(40, 512), (700, 1024), (1000, 1552), (200, 3072)])
def test_input_on_a_16_byte_boundary_only(oracle, rows, cols):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    buf = student_t_bf16((rows * cols + 8,), 5).cuda()
    x = buf[8:].view(rows, cols)
    assert x.data_ptr() % 32 == 16
    _check(oracle, x.cpu(), nv.FP4Tensor.from_bfloat16(x))


@pytest.mark.parametrize("rows,cols", [(2049, 1152), (5000, 1280), (5120, 1280), (300, 3072), (5376, 3072), (5632, 3072),
                                       (257, 2048)])
def test_known_maximum_fills_a_poisoned_buffer(oracle, rows, cols):
    """The packing kernel alone, through the entry point that takes the maximum: every byte of the
    swizzled layout is written, whichever form packs."""
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), 9)
    b = nv.PackedBuffers(rows, cols, "cuda", linear_scales=True)
    for t in (b.data, b.scales, b.scales_swz):
        t.fill_(0xAA)
    amax = x.float().abs().max().reshape(1).cuda()
    _check(oracle, x, nv.FP4Tensor.from_bfloat16(x.cuda(), amax=amax, out=b))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("with_partials", [False, True])
def test_c_entry_without_partials_and_with_odd_scale_pointers(oracle, offset, with_partials):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    for rows, cols in ((3, 256), (600, 1024), (1000, 1152), (1000, 1280), (1000, 1552), (200, 3072)):
        x = student_t_bf16((rows, cols), 6)
        xd = x.cuda()
        swz = torch.full((N.lib.nvfp4_swizzled_scale_bytes(rows, cols) + 16,), 0xAA, dtype=torch.uint8, device="cuda")
        lin = torch.empty(rows * cols // 16 + 16, dtype=torch.uint8, device="cuda")
        data = torch.empty(rows * cols // 2, dtype=torch.uint8, device="cuda")
        slots = torch.empty(2, device="cuda")
        part = torch.empty(N.AMAX_PARTIALS, device="cuda")
        rc = N.lib.nvfp4_amax_quantize_bf16(xd.data_ptr(), rows, cols, slots.data_ptr(), data.data_ptr(),
                                            lin.data_ptr() + offset, swz.data_ptr() + offset,
                                            slots.data_ptr() + 4, part.data_ptr() if with_partials else None,
                                            N.stream_ptr())
        assert rc == 0
        packed, scales, amax = oracle.quantize(bits_of(x))
        n = swz.numel() - 16
        assert float(slots[0]) == amax
        assert np.array_equal(data.cpu().numpy(), packed.reshape(-1))
        assert np.array_equal(lin[offset:offset + scales.size].cpu().numpy(), scales.reshape(-1))
        assert np.array_equal(swz[offset:offset + n].cpu().numpy(), oracle.swizzle_scales(scales, cols))
        assert bool((swz[offset + n:] == 0xAA).all()) and bool((swz[:offset] == 0xAA).all())


@pytest.mark.parametrize("rows,cols", [(33, 512), (600, 1024), (1000, 1536), (700, 4096)])
def test_given_buffers_nothing_is_allocated(rows, cols):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), 7, device="cuda")
    b = nv.PackedBuffers(rows, cols, "cuda", linear_scales=True)
    want = nv.FP4Tensor.from_bfloat16(x)
    count = lambda: torch.cuda.memory_stats()["allocation.all.allocated"]  # noqa: E731
    before = count()
    t = nv.FP4Tensor.from_bfloat16(x, out=b)
    nv.FP4Tensor.from_bfloat16(x, amax=t.global_amax(), out=b)
    nv.FP4Tensor.from_norm_mod(x, out=b)
    t = nv.FP4Tensor.from_bfloat16(x, out=b)
    assert count() == before
    assert torch.equal(t.quantized_data(), want.quantized_data())
    assert torch.equal(t.scale_factors_swizzled(), want.scale_factors_swizzled())


@pytest.mark.parametrize("rows,cols", [(33, 512), (700, 1024), (1000, 1280), (2000, 1536), (6000, 3072)])
@pytest.mark.parametrize("linear", [True, False])
def test_scale_layouts_that_are_not_wanted(oracle, rows, cols, linear):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), 8)
    packed, scales, amax = oracle.quantize(bits_of(x))
    for kw in ({}, {"amax": torch.full((1,), amax, device="cuda")}):
        t = nv.FP4Tensor.from_bfloat16(x.cuda(), linear_scales=linear, swizzled_scales=not linear, **kw)
        assert np.array_equal(t.quantized_data().cpu().numpy(), packed.reshape(-1))
        assert (t._scales is None, t._scales_swz is None) == (not linear, linear)
        assert np.array_equal(t.scale_factors_swizzled().cpu().numpy(), oracle.swizzle_scales(scales, cols))
        if linear:
            assert np.array_equal(t.scale_factors().cpu().numpy(), scales.reshape(-1))
