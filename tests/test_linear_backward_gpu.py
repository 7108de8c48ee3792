"""The backward of a linear in four launches: its gradients against the products on transposed copies, the bias
gradient against a float64 sum, in every combination of what is wanted."""
import itertools

import pytest
import torch

from helpers import randn_bf16, student_t_bf16

pytestmark = pytest.mark.gpu


def _backward(go, x, w, dx=True, dw=True, db=True, w_amax=None):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    (m, n), k = go.shape, 8 if w is None else w.shape[1]
    new = lambda *s: torch.full(s, float("nan"), dtype=torch.bfloat16, device="cuda")  # noqa: E731
    out = [new(m, k) if dx else None, new(n, k) if dw else None, new(n) if db else None]
    ws = torch.full((N.lib.nvfp4_linear_backward_workspace_bytes(m, n, k),), 0xA5, dtype=torch.uint8, device="cuda")
    N.check(N.lib.nvfp4_linear_backward_bias_bf16(
        go.data_ptr(), N.ptr(x), N.ptr(w), N.ptr(w_amax), m, n, k, *(N.ptr(t) for t in out), ws.data_ptr(),
        N.status_word(go.device).data_ptr(), N.stream_ptr()), "backward")
    return out


# one row; edges of the 128 x 64 tiles and of the 256-element padding; several row tiles per column sum
@pytest.mark.parametrize("m,n,k", [(1, 32, 8), (31, 64, 72), (128, 256, 64), (129, 288, 264), (1000, 1056, 1000),
                                   (4100, 96, 520)])
def test_every_combination(m, n, k):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = student_t_bf16((m, k), m, device="cuda"), randn_bf16((n, k), 2, device="cuda")
    go = student_t_bf16((m, n), 3, device="cuda")
    want_dx, want_dw = lc.gemm(go, w.t().contiguous()), lc.gemm(go.t().contiguous(), x.t().contiguous())
    want_db = go.double().sum(0)
    # sums of m terms in float32, then the bf16 rounding
    bound = go.double().abs().sum(0) * m * 2.0 ** -24 + want_db.abs() * 2.0 ** -8
    w_amax = w.float().abs().max().reshape(1)
    first = None
    for dx, dw, db in itertools.product((True, False), repeat=3):
        for known in (None, w_amax):
            got = _backward(go, x, w, dx, dw, db, known)
            assert got[0] is None or torch.equal(got[0], want_dx)
            assert got[1] is None or torch.equal(got[1], want_dw)
            if db:
                assert ((got[2].double() - want_db).abs() <= bound).all()
                first = got[2] if first is None else first
                assert torch.equal(got[2], first)      # whoever adds the partial sums


def test_infinities_and_nans_reach_the_bias_gradient():
    go = randn_bf16((300, 64), 1, device="cuda")
    go[7, 3], go[290, 4], go[0, 5], go[299, 5] = float("nan"), float("inf"), float("inf"), -float("inf")
    db = _backward(go, None, None, False, False, True)[2]
    assert db[3].isnan() and db[4] == float("inf") and db[5].isnan()
    assert db.isfinite().sum() == 61


def test_repeated_beside_another_stream():
    go, x, w = (student_t_bf16(s, i, device="cuda") for i, s in enumerate([(2048, 1024), (2048, 768), (1024, 768)]))
    want = _backward(go, x, w)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(30):
        with torch.cuda.stream(side):
            other = _backward(go, x, w)
        got = _backward(go, x, w)
        torch.cuda.synchronize()
        for a, b, c in zip(want, got, other):
            assert torch.equal(a, b) and torch.equal(a, c)


def test_refusals():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    go, w = randn_bf16((32, 64), 1, device="cuda"), randn_bf16((64, 32), 2, device="cuda")
    ws = torch.empty(N.lib.nvfp4_linear_backward_workspace_bytes(32, 64, 32), dtype=torch.uint8, device="cuda")
    y = torch.empty((32, 32), dtype=torch.bfloat16, device="cuda")

    def call(dy, wt, m, n, k, dx, work):
        return N.lib.nvfp4_linear_backward_bias_bf16(dy, None, wt, None, m, n, k, dx, None, None, work, None, None)
    good = (go.data_ptr(), w.data_ptr(), 32, 64, 32, y.data_ptr(), ws.data_ptr())
    for i, bad in ((0, None), (1, None), (2, 0), (3, 60), (3, 48), (4, 36), (6, None)):
        assert call(*good[:i], bad, *good[i + 1:]) == 1
    for i in (0, 1, 6):
        assert call(*good[:i], good[i] + 8, *good[i + 1:]) == 2
