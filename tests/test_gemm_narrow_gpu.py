"""The automatic choice of the GEMM's tile width: bit-identical to 256-wide tiles wherever it picks
narrower ones (the K order of every sum is the same), epilogues and ragged edges included."""
import pytest
import torch

from helpers import randn_bf16, student_t_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 32), (1, 64, 256), (3, 200, 512), (1, 3072, 512), (31, 1536, 512), (31, 1600, 512), (32, 1600, 512),
    (31, 6272, 256), (31, 6400, 256), (32, 6400, 256), (63, 13824, 256), (64, 13824, 256), (8, 5120, 8192), (512, 3072, 1024), (512, 3080, 4096), (257, 1096, 2048),
    (1760, 3072, 512), (1760, 9216, 256), (1760, 14336, 256), (2048, 1032, 14336), (900, 5120, 96),
    (4095, 5120, 288)])
@pytest.mark.parametrize("epilogue", [False, True])
def test_auto_tiling_equals_uniform(M, N, K, epilogue):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    a = nv.FP4Tensor.from_bfloat16(student_t_bf16((M, K), M + N, device="cuda"), linear_scales=False)
    b = nv.FP4Tensor.from_bfloat16(randn_bf16((N, K), K, 0.02, device="cuda"), linear_scales=False)
    kw = {}
    if epilogue:
        kw = dict(bias=randn_bf16((N,), 1, device="cuda"), gelu=True, C=randn_bf16((M, N), 2, device="cuda"),
                  gate=torch.randn(N, generator=torch.Generator("cuda").manual_seed(3), device="cuda"), beta=1.0,
                  out_amax=torch.empty(1, device="cuda"))
    beta = kw.pop("beta", 0.0)
    nv.set_gemm_tiling("uniform")
    try:
        want = nv.fp4_gemm(a, b, 1.0, beta, **kw)
        amax = kw["out_amax"].clone() if epilogue else None
    finally:
        nv.set_gemm_tiling("auto")
    for _ in range(3):
        y = nv.fp4_gemm(a, b, 1.0, beta, **kw)
        assert torch.equal(y, want)
        if epilogue:
            assert torch.equal(kw["out_amax"], amax)
            assert float(amax) == float(want.abs().max())
    nv.check_status()
