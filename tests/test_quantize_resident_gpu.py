"""The quantizer that holds the tensor in shared memory, and the sizes at which the forms meet: byte for byte the
maximum and the packing in two calls, over poisoned buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(one, x, rows, cols, linear=True, swizzled=True, shift=0):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    dev = x.device
    slots = torch.full((2,), float("nan"), device=dev)
    part = torch.full((N.AMAX_PARTIALS,), float("nan"), device=dev)
    data = torch.full((rows * cols // 2 + 16,), 0xA5, dtype=torch.uint8, device=dev)
    lin = torch.full((rows * cols // 16 + 16,), 0xA5, dtype=torch.uint8, device=dev) if linear else None
    swz = torch.full((N.swizzled_scale_bytes(rows, cols) + 16,), 0xA5, dtype=torch.uint8, device=dev)
    p_swz = swz.data_ptr() + shift if swizzled else None
    amax, gs, st = slots.data_ptr(), slots.data_ptr() + 4, N.stream_ptr()
    if one:
        rc = N.lib.nvfp4_amax_quantize_bf16(x.data_ptr(), rows, cols, amax, data.data_ptr(), N.ptr(lin), p_swz, gs,
                                            part.data_ptr(), st)
    else:
        rc = N.lib.nvfp4_amax_bf16(x.data_ptr(), rows * cols, amax, st)
        rc = rc or N.lib.nvfp4_quantize_bf16(x.data_ptr(), rows, cols, amax, data.data_ptr(), N.ptr(lin), p_swz, gs, st)
    assert rc == 0
    torch.cuda.synchronize()
    return [t for t in (data, lin, swz, slots) if t is not None]


@pytest.mark.parametrize("rows,cols", [
    (64, 4096), (65, 4096), (85, 3072), (86, 3072),      # either side of four blocks a thread of a cluster
    (128, 4096), (129, 4096), (1, 262160), (300, 272),
    (296, 8192), (296, 8208),                            # one block a thread of the grid, and a few over
    (1480, 9840), (1776, 8192), (1776, 8208),            # the last that fits, and the first that does not
    (700, 14336), (2500, 5120), (100, 13824),
])
def test_forms_agree_at_their_edges(rows, cols):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, cols, generator=g, device="cuda") * 3).bfloat16()
    x.view(-1)[-1] = 100.0                               # the maximum in the last block
    for a, b in zip(_run(True, x, rows, cols), _run(False, x, rows, cols)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", [dict(linear=False), dict(swizzled=False), dict(shift=1), dict(shift=4)])
@pytest.mark.parametrize("offset", [0, 8])
def test_buffers_a_caller_may_give(form, offset):
    x = torch.randn(600 * 4096 + 8, device="cuda").bfloat16()[offset:offset + 600 * 4096].view(600, 4096)
    for a, b in zip(_run(True, x, 600, 4096, **form), _run(False, x, 600, 4096, **form)):
        assert torch.equal(a, b)
