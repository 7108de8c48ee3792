"""The maximum ahead of packing, wherever it lies: first and last pieces, pieces of a thread's last round that are there or
not, rows that start off a 32-byte boundary, a tensor larger than L2."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


# the rows form (more than 262144 elements; two kernels): whole rounds of 1024 pieces, one piece more, one round of all CTAs
# and a little more (592 CTAs of 1024 pieces), more than L2
@pytest.mark.parametrize("rows,cols", [(128, 2176), (129, 2048), (1023, 1168), (4736, 2048), (4737, 2048), (2547, 5104),
                                       (21600, 3072)])
@pytest.mark.parametrize("offset", [0, 8])
def test_planted(rows, cols, offset):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    n = rows * cols
    x = torch.randn(n + offset, device="cuda").bfloat16()[offset:].view(rows, cols)
    flat, out, rng = x.view(-1), nv.PackedBuffers(rows, cols, "cuda"), random.Random(rows)
    at = [0, 7, 8, 15, 16, n - 1, n - 8, n - 9, n - 17, 1024 * 16 - 1, 1024 * 16] + [rng.randrange(n) for _ in range(25)]
    for i in at:
        was = flat[i].clone()
        flat[i] = -77.5 if i % 2 else 77.5
        got = nv.FP4Tensor.from_bfloat16(x, linear_scales=False, out=out)
        assert float(got.global_scale()) == pytest.approx(77.5 / 2688, rel=1e-6) and float(got.global_amax()) == 77.5
        flat[i] = was


def test_planted_in_an_operand_of_the_backward():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    one, rng = torch.ones(1, device="cuda"), random.Random(3)
    m, n, k = 520, 96, 136
    for i in [0, 8, m * k - 1, m * k - 9] + [rng.randrange(m * k) for _ in range(6)]:
        go, x, w = (torch.randn(s, device="cuda").bfloat16() for s in ((m, n), (m, k), (n, k)))
        x.view(-1)[i] = 300.0
        go.view(-1)[i * (m * n - 1) // (m * k)] = -200.0
        dx, dw, _ = lc.backward(go, x, w, one, one, one, True, True, False)
        assert torch.equal(dx, lc.gemm(go, w.t().contiguous()))
        assert torch.equal(dw, lc.gemm(go.t().contiguous(), x.t().contiguous()))
