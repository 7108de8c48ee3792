"""The linear that goes through one library call equals quantize + GEMM called one by one, for every
combination of its epilogue and for operands that it has to leave to the general path."""
import itertools

import pytest
import torch

from helpers import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 3072, 3072), (7, 64, 32), (300, 520, 1056), (3000, 1024, 512)])
def test_equals_the_separate_calls(m, n, k):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv, nvfp4_linear_cpp as lc
    x, w = randn_bf16((m, k), 1, device="cuda"), randn_bf16((n, k), 2, 0.02, device="cuda")
    bias, res = randn_bf16((n,), 3, device="cuda"), randn_bf16((m, n), 4, device="cuda")
    gate = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    a, b = nv.FP4Tensor.from_bfloat16(x), nv.FP4Tensor.from_bfloat16(w)
    for use in itertools.product([False, True], repeat=4):
        kw = dict(bias=bias if use[0] else None, gelu=use[1], gate=gate if use[2] else None)
        want = nv.fp4_gemm(a, b, 1.0, 1.0 if use[3] else 0.0, C=res if use[3] else None, **kw)
        got = lc.linear(x.view(1, m, k), w, kw["bias"], gelu=use[1], gate=kw["gate"],
                        residual=res.view(1, m, n) if use[3] else None)
        assert got.shape == (1, m, n) and torch.equal(got[0], want), use
    nv.check_status()


def test_operands_for_the_general_path():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = randn_bf16((40, 64), 1, device="cuda"), randn_bf16((48, 64), 2, device="cuda")
    want = lc.linear(x, w)
    assert torch.equal(lc.linear(torch.cat([x, x], 1)[:, :64], w), want)               # strided rows
    out = torch.empty(40, 48, dtype=torch.bfloat16, device="cuda")
    assert lc.linear(x, w, out=out).data_ptr() == out.data_ptr() and torch.equal(out, want)
    with pytest.raises(RuntimeError, match="C must be contiguous"):
        lc.linear(x, w, residual=randn_bf16((40, 96), 3, device="cuda")[:, :48])
    with pytest.raises(RuntimeError):
        lc.linear(x, w, torch.zeros(48, device="cuda"))                                # fp32 bias
    with pytest.raises(RuntimeError):
        lc.linear(x.float(), w)
    w.mul_(2)                                                                          # packed anew
    assert torch.equal(lc.linear(x, w), lc.gemm(x, w))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = lc.linear(x, w)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(y, lc.gemm(x, w))


def test_a_strided_residual_is_copied_once():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = randn_bf16((4, 10, 64), 1, device="cuda"), randn_bf16((48, 64), 2, device="cuda")
    res = randn_bf16((10, 4, 48), 3, device="cuda").transpose(0, 1)
    out = torch.empty(4, 10, 48, dtype=torch.bfloat16, device="cuda")

    def allocations(r):
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        lc.linear(x, w, residual=r, out=out)
        return torch.cuda.memory_stats()["allocation.all.allocated"] - before
    lc.linear(x, w, residual=res, out=out)
    want = out.clone()
    plain = res.contiguous()
    assert allocations(res) == allocations(plain) + 1
    assert torch.equal(lc.linear(x, w, residual=res.contiguous()), want)
