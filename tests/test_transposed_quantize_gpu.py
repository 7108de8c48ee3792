"""The transposing quantizer against the plain one on a transposed copy, byte for byte, and the
gradients built on it against the products on transposed copies."""
import pytest
import torch

from helpers import randn_bf16, student_t_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 8), (16, 64), (31, 72), (32, 128), (127, 264), (128, 256), (129, 248),
                                       (1000, 1000), (2048, 3072), (4097, 520)])
def test_bytes_equal_those_of_a_transposed_copy(rows, cols):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = student_t_bf16((rows, cols), rows + cols, device="cuda")
    t = nv.FP4Tensor.from_bfloat16_transposed(x)
    c = torch.nn.functional.pad(x.t(), (0, -rows % 32)).contiguous()
    q = nv.FP4Tensor.from_bfloat16(c)
    assert t.shape() == list(c.shape) == q.shape()
    assert torch.equal(t.global_amax(), q.global_amax()) and torch.equal(t.global_scale(), q.global_scale())
    assert torch.equal(t.quantized_data(), q.quantized_data())
    assert torch.equal(t.scale_factors_swizzled(), q.scale_factors_swizzled())


def test_refusals():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x = randn_bf16((64, 64), 1, device="cuda")
    for bad in (x.t(), x[:, :12].contiguous(), x[:0], x[0], x.float(), x.cpu()):
        with pytest.raises(RuntimeError):
            nv.FP4Tensor.from_bfloat16_transposed(bad)
    with pytest.raises(RuntimeError, match="amax"):
        nv.FP4Tensor.from_bfloat16_transposed(x, torch.zeros(2, device="cuda"))


@pytest.mark.parametrize("m,n,k", [(64, 96, 128), (33, 64, 40), (100, 40, 72), (50, 36, 64), (64, 64, 36)])
def test_gradients_equal_the_products_on_copies(m, n, k):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = randn_bf16((m, k), 1, device="cuda"), randn_bf16((n, k), 2, device="cuda")
    go = randn_bf16((m, n), 3, device="cuda")
    one = torch.ones(1, device="cuda")
    dx, dw, db = lc.backward(go, x, w, one, one, one, True, True, True)
    assert torch.equal(dx, lc.gemm(go, w.t().contiguous()))
    assert torch.equal(dw, lc.gemm(go.t().contiguous(), x.t().contiguous()))
    assert torch.equal(db, go.sum(0))
    # a strided gradient, and the weight gradient alone
    wide = torch.cat([go, go], 1)[:, :n]
    assert torch.equal(lc.backward(wide, x, w, one, one, one, False, True, False)[1], dw)
    # a weight changed in place since it was packed: its maximum is taken anew
    lc.quantized_weight(w)
    w.mul_(3)
    dx3 = lc.backward(go, x, w, one, one, one, True, False, False)[0]
    assert torch.equal(dx3, lc.gemm(go, w.t().contiguous()))
    # also when the change went past the version count
    lc.quantized_weight(w)
    w.data.mul_(4)
    dx12 = lc.backward(go, x, w, one, one, one, True, False, False)[0]
    assert torch.equal(dx12, lc.gemm(go, w.t().contiguous()))
