"""The GEMM's epilogues that are fixed when its kernel is compiled against the one that reads its parameters, bit for bit:
a gate of ones, a residual and a bias of zeros take any call to the latter and change no value."""
import itertools

import pytest
import torch

from helpers import randn_bf16

pytestmark = pytest.mark.gpu


# one tile; 64- and 128-wide, 192-wide and 256-wide tilings, ragged in M and N
@pytest.mark.parametrize("m,n,k", [(1, 8, 32), (65, 200, 96), (300, 520, 1056), (1700, 3080, 288), (5000, 2056, 96)])
def test_every_combination_equals_the_general_epilogue(m, n, k):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    a = nv.FP4Tensor.from_bfloat16(randn_bf16((m, k), 1, device="cuda"), linear_scales=False)
    b = nv.FP4Tensor.from_bfloat16(randn_bf16((n, k), 2, 0.05, device="cuda"), linear_scales=False)
    bias, res = randn_bf16((n,), 3, device="cuda"), randn_bf16((m, n), 4, device="cuda")
    gate = torch.randn(n, generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    for with_bias, gelu, with_gate, with_c, with_amax in itertools.product([False, True], repeat=5):
        amax, amax_general = torch.full((1,), -1.0, device="cuda"), torch.full((1,), -1.0, device="cuda")
        y = nv.fp4_gemm(a, b, 1.0, 1.0 if with_c else 0.0, C=res if with_c else None, bias=bias if with_bias else None,
                        gate=gate if with_gate else None, gelu=gelu, out_amax=amax if with_amax else None)
        want = nv.fp4_gemm(a, b, 1.0, 1.0, C=res if with_c else torch.zeros_like(res),
                           bias=bias if with_bias else torch.zeros_like(bias),
                           gate=gate if with_gate else torch.ones_like(gate), gelu=gelu, out_amax=amax_general)
        assert torch.equal(y, want), (with_bias, gelu, with_gate, with_c, with_amax)
        assert float(amax_general) == float(want.abs().max())
        assert not with_amax or torch.equal(amax, amax_general)
    nv.check_status()
