"""The bias gradient of a linear where something follows what is done to the output's gradient: a forward-mode tangent, a
second derivative, a dispatch mode, a trace.  There it is a sum of torch, whichever code makes the other gradients."""
import pytest
import torch
from torch.autograd import forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

from helpers import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["native", "python"])
def operands(request, monkeypatch):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    if request.param == "python":
        monkeypatch.setattr(N, "host", N._Declines())
    return randn_bf16((48, 64), 1, device="cuda"), randn_bf16((96, 64), 2, device="cuda")


def _backward(go, x, w, dx=True, dw=True):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    one = torch.ones(1, device="cuda")
    return lc.backward(go, x, w, one, one, one, dx, dw, True)


@pytest.mark.parametrize("wanted", [(True, True), (False, True), (True, False), (False, False)])
@pytest.mark.parametrize("shape", [(48, 96), (2, 24, 96)])
def test_tangent(operands, wanted, shape):
    x, w = operands
    go, t = randn_bf16(shape, 3, device="cuda"), randn_bf16(shape, 4, device="cuda")
    x = x.view(*shape[:-1], 64)
    plain = _backward(go, x, w, *wanted)
    with forward_ad.dual_level():
        got = _backward(forward_ad.make_dual(go, t), x, w, *wanted)
        db, tangent = forward_ad.unpack_dual(got[2])
        assert tangent is not None and torch.equal(tangent, t.reshape(-1, 96).sum(0))
        assert torch.equal(db, go.reshape(-1, 96).sum(0))
        for a, b in zip(got[:2], plain[:2]):
            assert (a is None) == (b is None) and (a is None or torch.equal(forward_ad.unpack_dual(a).primal, b))


def test_second_derivative(operands):
    x, w = operands
    go = randn_bf16((48, 96), 3, device="cuda").requires_grad_(True)
    assert torch.equal(torch.autograd.grad(_backward(go, x, w)[2].sum(), go)[0], torch.ones_like(go))
    with torch.no_grad():
        assert not _backward(go, x, w)[2].requires_grad


def test_dispatch_mode(operands):
    x, w = operands
    go = randn_bf16((48, 96), 3, device="cuda")

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.made = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            if func.overloadpacket is torch.ops.aten.sum:
                self.made.append(out)
            return out
    with Seen() as seen:
        db = _backward(go, x, w)[2]
    assert any(db is t for t in seen.made) and torch.equal(db, go.sum(0))


def test_trace(operands):
    x, w = operands
    go, other = (randn_bf16((48, 96), s, device="cuda") for s in (3, 4))
    traced = torch.jit.trace(lambda g: _backward(g, x, w)[2], go, check_trace=False)
    assert torch.equal(traced(other), other.sum(0))
