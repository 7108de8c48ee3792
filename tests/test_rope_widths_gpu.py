"""q/k RMSNorm + rotation in both forms (a row per warp, a row per CTA), for every number of warps that
share a row and for heads whose width does not divide a team's: against the torch ops it replaces."""
import pytest
import torch

from helpers import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,heads,D", [
    (5, 1, 16), (9, 1, 128), (33, 24, 128), (65, 25, 128), (1, 40, 128), (130, 48, 128), (17, 49, 128),
    (3, 128, 128), (20, 10, 48), (11, 70, 80), (700, 3, 128),
    (1300, 3, 128), (1000, 12, 128), (1000, 24, 128), (1000, 30, 80), (1185, 12, 128), (12000, 20, 128)])   # rows at which the form changes
@pytest.mark.parametrize("gains", [True, False])
def test_widths_against_torch_ops(rows, heads, D, gains):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit
    dim = heads * D
    qkv = randn_bf16((rows, 3 * dim), rows + dim, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(dim)
    gq = 1 + 0.1 * torch.randn(dim, generator=g, device="cuda")
    gk = 1 + 0.1 * torch.randn(dim, generator=g, device="cuda")
    ang = torch.rand(rows, D // 2, generator=g, device="cuda") * 40
    cos, sin = ang.cos().repeat_interleave(2, 1), ang.sin().repeat_interleave(2, 1)
    q, k, v = dit.qk_norm_rope(qkv, heads, D, gq if gains else None, gk if gains else None, 1e-6,
                               dit.pack_rope_table(cos, sin))
    one = torch.ones(dim, device="cuda")
    for got, cols, gain in ((q, qkv[:, :dim], gq), (k, qkv[:, dim:2 * dim], gk)):
        n = dit.rms_norm(cols, gain if gains else one, 1e-6).view(rows, heads, D)
        want = dit.apply_rope(n, cos, sin)
        # the sum of squares in another order moves a bf16 rounding of n by one step (2^-8), which the
        # rotation carries into both elements of the pair: |dn| (|c| + |s|) <= 2^-8 * sqrt(2) * |n|,
        # plus the output's own rounding
        size = n.float().view(rows, heads, D // 2, 2).abs().amax(-1, keepdim=True).expand(-1, -1, -1, 2)
        bound = size.reshape(rows, heads, D) * (2.0 ** -8 * 1.4143 + 2.0 ** -7)
        assert bool(((got.float() - want.float()).abs() <= bound).all())
        assert float((got != want).float().mean()) < 5e-3
    assert torch.equal(v, qkv[:, 2 * dim:].view(rows, heads, D))
