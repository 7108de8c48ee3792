"""The native calls of the backward, the quantizer with given buffers or a known maximum, and the q/k norms against the
Python code that they spare: the same results, and the same answers to what they leave to it."""
import pytest
import torch

from helpers import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture
def both(monkeypatch):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N

    def run(call, name, native=True):
        """call() with the native function, and without; whether that took the call."""
        real, took = N.host, []

        class Spy:
            def __getattr__(self, attr):
                fn = getattr(real, attr)
                if attr != name:
                    return fn

                def spied(*a):
                    r = fn(*a)
                    took.append(r is not None)
                    return r
                return spied

        def outcome():
            try:
                return call()
            except Exception as e:           # the same refusal from both
                return type(e)
        monkeypatch.setattr(N, "host", Spy())
        a = outcome()
        monkeypatch.setattr(N, "host", N._Declines())
        b = outcome()
        monkeypatch.setattr(N, "host", real)
        assert took == [native], took
        return a, b
    return run


def _same(a, b):
    if isinstance(a, type) or a is None or b is None:
        return a is b
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("shape,n,k,native", [((64,), 96, 128, True), ((2, 33), 64, 40, True), ((1,), 32, 8, True),
                                              ((50,), 36, 64, False), ((20,), 40, 64, False), ((0,), 64, 64, False)])
@pytest.mark.parametrize("want", [(True, True, True), (True, False, False), (False, True, True), (False, False, True)])
def test_backward(both, shape, n, k, native, want):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = randn_bf16((*shape, k), 1, device="cuda"), randn_bf16((n, k), 2, device="cuda")
    go, one = randn_bf16((*shape, n), 3, device="cuda"), torch.ones(1, device="cuda")
    a, b = both(lambda: lc.backward(go, x, w, one, one, one, *want), "linear_backward",
                native and (want[0] or want[1]))
    assert _same(a, b)


def test_backward_leaves_to_python(both):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as lc
    x, w = randn_bf16((64, 64), 1, device="cuda"), randn_bf16((64, 64), 2, device="cuda")
    go, one = randn_bf16((64, 64), 3, device="cuda"), torch.ones(1, device="cuda")
    for g, i, v in ((go.t(), x, w), (go, x.t(), w), (go, x, w.t()), (go[:1].expand(64, 64), x, w), (go.float(), x, w),
                    (go, x[:32], w), (go, x[:, :32].contiguous(), w)):
        assert _same(*both(lambda: lc.backward(g, i, v, one, one, one, True, True, True), "linear_backward", False))


def test_a_differentiated_backward_keeps_the_bias_sum():
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4_linear_module import NVFP4Linear
    lin = NVFP4Linear(64, 32).cuda()
    x, g = randn_bf16((16, 64), 1, device="cuda"), randn_bf16((16, 32), 2, device="cuda").requires_grad_(True)
    db, = torch.autograd.grad(lin(x), [lin.bias], g, create_graph=True)
    assert torch.equal(torch.autograd.grad(db.sum(), g)[0], torch.ones_like(g))


@pytest.mark.parametrize("rows,cols,linear", [(3, 64, True), (300, 3072, False), (1, 16, False)])
def test_quantizer_with_buffers_or_maximum(both, rows, cols, linear):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    x, amax = randn_bf16((rows, cols), 1, device="cuda"), torch.full((1,), 7.0, device="cuda")
    bufs = [nv.PackedBuffers(rows, cols, "cuda", linear_scales=linear) for _ in range(2)]

    def call(out, known):
        t = nv.FP4Tensor.from_bfloat16(x, linear_scales=linear, amax=known, out=out)
        return [t.quantized_data().clone(), t.scale_factors_swizzled().clone(), t.global_amax().clone(), t.global_scale().clone(),
                t.scale_factors().clone() if linear else None]
    for out in (None, bufs[0]):
        for known in (None, amax):
            if out is None and known is None:
                continue
            assert _same(*both(lambda: call(out, known), "quantize_into"))
    # another tensor's buffers, a maximum of another type: refused by both
    other = nv.PackedBuffers(rows + 1, cols, "cuda", linear_scales=linear)
    with pytest.raises(RuntimeError):
        nv.FP4Tensor.from_bfloat16(x, linear_scales=linear, out=other)
    assert _same(*both(lambda: call(bufs[0], amax.double()), "quantize_into", False))
    assert _same(*both(lambda: call(bufs[0], torch.zeros(2, device="cuda")), "quantize_into", False))


@pytest.mark.parametrize("L,heads", [(1, 1), (65, 24), (300, 5)])
def test_norms(both, L, heads):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit
    dim = heads * 128
    qkv, gain = randn_bf16((L, 3 * dim), 1, device="cuda"), torch.randn(dim, device="cuda")
    cs = torch.randn(L, 64, 2, device="cuda")
    for g in (gain, None):
        assert _same(*both(lambda: dit.qk_norm_rope(qkv, heads, 128, g, g, 1e-6, cs), "qk_norm_rope"))
        assert _same(*both(lambda: dit.rms_norm_fused(qkv[:, dim:2 * dim], heads, 128, g, 1e-6), "rms_norm"))
    for bad in (lambda: dit.qk_norm_rope(qkv.float(), heads, 128, gain, gain, 1e-6, cs),
                lambda: dit.qk_norm_rope(qkv, heads, 128, gain, gain, 1e-6, cs.double()),
                lambda: dit.qk_norm_rope(qkv, heads + 1, 128, gain, gain, 1e-6, cs)):
        assert _same(*both(bad, "qk_norm_rope", False))
    assert _same(*both(lambda: dit.rms_norm_fused(qkv, heads, 128, gain, 1e-6), "rms_norm", False))
