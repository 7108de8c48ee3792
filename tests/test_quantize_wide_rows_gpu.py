"""The rows form's wider CTAs (3088 to 5120 columns), alone and ahead of a GEMM, over poisoned buffers, against the form
that takes any width: one row of the same elements."""
import pytest
import torch

from helpers import student_t_bf16

pytestmark = pytest.mark.gpu


# edges of the widths (a CTA of 224 threads from 3088, one of 256 from 3600, one of 320 from 4624 columns; 3072 and 5136 take
# others), of the K padding (3328, 3344), of four-row groups and of the 256-row padding; both sides of the line below which
# a few wide rows alone take one launch (kAloneBlocks) and of the one above which long ones with a known maximum are flat
@pytest.mark.parametrize("rows,cols", [(32, 3456), (33, 3440), (129, 3600), (257, 4096), (1536, 5120), (1537, 5120),
                                       (2001, 4640), (5000, 5104), (300, 5136), (33, 3088), (2600, 3088), (2547, 3088),
                                       (129, 3328), (2601, 3328), (2560, 3344), (2500, 3584), (2500, 3600), (1800, 4608),
                                       (1800, 4624), (2500, 3072), (9830, 5120), (9831, 5120)])
@pytest.mark.parametrize("offset", [0, 8])
def test_bytes(rows, cols, offset):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = torch.empty(rows * cols + offset, dtype=torch.bfloat16, device="cuda")[offset:].view(rows, cols)
    x.copy_(student_t_bf16((rows, cols), rows) if rows * cols < 1 << 24 else
            torch.randn(rows, cols, generator=torch.Generator("cuda").manual_seed(rows), device="cuda"))
    flat = nv.FP4Tensor.from_bfloat16(x.reshape(-1))
    b = nv.PackedBuffers(rows, cols, "cuda", linear_scales=True)
    for t in b.tensors:
        t.view(torch.uint8).fill_(0xFF)
    got = nv.FP4Tensor.from_bfloat16(x, out=b)
    known = nv.FP4Tensor.from_bfloat16(x, amax=flat.global_amax())
    for t in (got, known):
        assert torch.equal(t.quantized_data(), flat.quantized_data())
        assert torch.equal(t.scale_factors(), flat.scale_factors())
        assert torch.equal(t.global_scale(), flat.global_scale())
    # the swizzled layout of the linear scales, its padding zeros
    sf = torch.zeros(-(-rows // 256) * 256, -(-cols // 256) * 16, dtype=torch.uint8, device="cuda")
    sf[:rows, :cols // 16] = flat.scale_factors().view(rows, cols // 16)
    want = sf.view(-1, 4, 32, sf.shape[1] // 4, 4).permute(0, 3, 2, 1, 4).reshape(-1)
    assert torch.equal(got.scale_factors_swizzled(), want) and torch.equal(known.scale_factors_swizzled(), want)


@pytest.mark.parametrize("m,k", [(40, 3456), (300, 4096), (1000, 5120), (2100, 4640), (85, 3104), (700, 3328), (701, 3360)])
def test_linear(m, k):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv, nvfp4_linear_cpp as lc
    x, w = student_t_bf16((m, k), m, device="cuda"), student_t_bf16((64, k), 2, device="cuda")
    want = nv.fp4_gemm(nv.FP4Tensor.from_bfloat16(x.reshape(-1, k)), nv.FP4Tensor.from_bfloat16(w))
    for _ in range(3):
        assert torch.equal(lc.linear(x, w), want)
    nv.check_status()
