"""The dequantizer, tabulated and with a thread's own entries (up to a block per thread of one CTA per
SM): every scale byte with every code, at several tensor maxima, bit for bit against the formula in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


@pytest.mark.parametrize("amax", [0.0, 3.7, 2688.0, 1e-30, 3e38])
@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("copies", [1, 200])
def test_every_scale_byte_with_every_code(amax, shift, copies):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    codes = torch.arange(16, device="cuda", dtype=torch.uint8)
    byte = codes[0::2] | (codes[1::2] << 4)                              # sixteen codes = one block
    n = 256 * 16 * copies
    buf = torch.zeros(n // 2 + 8, dtype=torch.uint8, device="cuda")
    packed = buf[shift:shift + n // 2]
    packed.copy_(byte.repeat(256 * copies))
    sf = torch.arange(256, device="cuda", dtype=torch.int32).to(torch.uint8).repeat(copies)
    slot = torch.tensor([amax], device="cuda")
    out = torch.empty(n + 16, dtype=torch.bfloat16, device="cuda")[shift * 2:shift * 2 + n]
    rc = N.lib.nvfp4_dequantize_bf16(packed.data_ptr(), sf.data_ptr(), 256 * copies, 16, slot.data_ptr(), out.data_ptr(),
                                     N.stream_ptr())
    assert rc == 0
    big = torch.finfo(torch.float32).max
    s_enc = torch.clamp(torch.tensor(2688.0, device="cuda") / slot, max=big)
    s_enc = torch.where((slot == 0) | (s_enc == 0), torch.ones_like(s_enc), s_enc)
    d = sf.view(torch.float8_e4m3fn).float() / s_enc
    v = torch.tensor(_E2M1 + tuple(-e for e in _E2M1), device="cuda")
    want = (v.view(1, 16) * d.view(-1, 1)).to(torch.bfloat16).view(-1)
    nan = torch.isnan(want.float())
    assert torch.equal(torch.isnan(out.float()), nan)
    assert torch.equal(out.view(torch.int16)[~nan], want.view(torch.int16)[~nan])   # signs of zeros too


@pytest.mark.parametrize("n", [16, 16 * 511, 16 * 513, 16 * 37887, 16 * 37888, 16 * 37889, 16 * 700001])
def test_lengths(n):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4 as nv
    x = torch.randn(1, n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(torch.bfloat16)
    t = nv.FP4Tensor.from_bfloat16(x)
    assert torch.equal(t.to_bfloat16(), dit.dequant_f32(t).to(torch.bfloat16))
