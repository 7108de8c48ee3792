"""Norm + quantize in two sweeps while kernels on other streams share its SMs: byte for byte what it gives alone.
(Alone, the second sweep's reads of a row group are always done before the copy that takes its place arrives.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,kind", [(8192, 3072, 0), (8192, 3072, 2), (9000, 3072, 1), (5000, 5120, 2),
                                            (40000, 512, 2), (12000, 2064, 3), (2500, 14336, 2)])
def test_same_bytes_beside_other_kernels(rows, cols, kind):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N, dit
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4 import FP4Tensor
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(rows, cols, generator=g, device="cuda") * 1.5).bfloat16()
    v = [torch.randn(cols, generator=g, device="cuda") * 0.2 for _ in range(4)]
    kw = dict(weight=v[0], bias=v[1]) if kind & 1 else {}
    kw.update(dict(scale=v[2], shift=v[3]) if kind & 2 else {})
    other = torch.randn(8192, 3072, generator=g, device="cuda").bfloat16()
    heads = other.view(8192, 24, 128)
    want = FP4Tensor.from_norm_mod(x, **kw)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for _ in range(40):
        with torch.cuda.stream(streams[0]):
            FP4Tensor.from_bfloat16(other)
        with torch.cuda.stream(streams[1]):
            dit.attention_native(heads, heads[:256], heads[:256])
        with torch.cuda.stream(streams[2]):
            got.append(FP4Tensor.from_norm_mod(x, **kw))
    torch.cuda.synchronize()
    N.check_status()
    for t in got:
        assert torch.equal(t._amax, want._amax)
        assert torch.equal(t._data, want._data) and torch.equal(t._scales_swz, want._scales_swz)
