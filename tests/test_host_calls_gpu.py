"""The native calls of the Python layer against the general path they stand in for: the same outputs for what
they take, and None for the rest, which the general path then takes or refuses as before."""
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("linear", "quantize", "norm_quantize", "dequantize", "gemm", "attention")


class _Off:
    """The module with every call declined."""

    def __init__(self, real):
        self.set_status = real.set_status
        for n in NAMES:
            setattr(self, n, lambda *a: None)


def _both(call):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    real, res = N.host, []
    for host in (real, _Off(real)):
        N.host = host
        try:
            res.append(call())
        except Exception as e:                     # noqa: BLE001 -- refusals are compared as well
            res.append((type(e), str(e)))
        finally:
            N.host = real
    torch.cuda.synchronize()
    return res


def _same(a, b):
    if isinstance(a, torch.Tensor):
        return (a.shape, a.dtype, a.stride(), a.requires_grad) == (b.shape, b.dtype, b.stride(), b.requires_grad) \
            and torch.equal(a, b)
    if isinstance(a, (list, tuple)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a == b


def _bf(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").bfloat16()


def _packed(t):
    return [t._data, t._scales, t._scales_swz, t._amax, t._gscale, t._rows, t._cols, t._shape, t._numel]


@pytest.mark.parametrize("shape", [(5, 64), (2, 3, 64), (300, 256), (1, 1, 1, 96), (0, 64), (64,), (4, 48), (7, 33)])
@pytest.mark.parametrize("kw", ["plain", "bias", "empty_bias", "gelu", "gate", "residual", "all", "float_bias",
                                "residual_3d", "strided_residual", "bias_2d"])
def test_linear(shape, kw):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as L
    k, n = shape[-1], 72
    x, w = _bf(*shape, seed=1), _bf(n, k, seed=2)
    out = shape[:-1] + (n,)
    a = {"plain": {}, "bias": dict(bias=_bf(n)), "empty_bias": dict(bias=_bf(0)), "gelu": dict(gelu=True),
         "gate": dict(gate=_bf(n).float()), "residual": dict(residual=_bf(*out)),
         "all": dict(bias=_bf(n), gelu=True, gate=_bf(n).float(), residual=_bf(*out)),
         "float_bias": dict(bias=_bf(n).float()), "residual_3d": dict(residual=_bf(1, *out)),
         "strided_residual": dict(residual=_bf(n, *shape[:-1]).movedim(0, -1)), "bias_2d": dict(bias=_bf(1, n))}[kw]
    try:
        L.quantized_weight(w)
    except RuntimeError:
        pass
    with torch.no_grad():
        assert _same(*_both(lambda: L.linear(x, w, **a)))


def test_linear_sees_a_changed_weight_and_strides():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4_linear_cpp as L
    x, w = _bf(40, 128), _bf(64, 128, seed=3)
    L.quantized_weight(w)
    before = L.linear(x, w)
    w.mul_(2)
    assert _same(L.linear(x, w), _both(lambda: L.linear(x, w))[1]) and not torch.equal(L.linear(x, w), before)
    for v in (x.t().contiguous().t(), x[::2], x[:, :128], _bf(40, 130)[:, 1:129], x.cpu(), x.float(), x[:, :96]):
        L.quantized_weight(w)
        assert _same(*_both(lambda: L.linear(v, w)))


@pytest.mark.parametrize("make", [lambda: _bf(7, 64), lambda: _bf(16), lambda: _bf(3, 5), lambda: _bf(0, 16),
                                  lambda: _bf(4, 33, 32)[:, 1:], lambda: _bf(64, 48).t(), lambda: _bf(4, 8, 16),
                                  lambda: _bf(64).view(-1)[1:33], lambda: _bf(1000, 5120), lambda: _bf(8, 16).float(),
                                  lambda: _bf(8, 16).cpu(), lambda: _bf(1)[0]])
@pytest.mark.parametrize("kw", [{}, dict(linear_scales=False), dict(swizzled_scales=False)])
def test_quantize_and_back(make, kw):
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4 import FP4Tensor
    x = make()
    assert _same(*_both(lambda: _packed(FP4Tensor.from_bfloat16(x, **kw))[:3]))
    first = 5 if x.numel() == 0 else 3             # an empty tensor's slots are not written
    assert _same(*_both(lambda: _packed(FP4Tensor.from_bfloat16(x, **kw))[first:]))
    assert _same(*_both(lambda: FP4Tensor.from_bfloat16(x, **kw).to_bfloat16()))


@pytest.mark.parametrize("rows,cols", [(5, 64), (0, 64), (300, 3072), (3, 24), (2, 16400)])
@pytest.mark.parametrize("vecs", [{}, {"scale": 0, "shift": 0}, {"weight": 0}, {"scale": 1}, {"scale": 2},
                                  {"bias": 3}])
@pytest.mark.parametrize("given", [False, True])
def test_norm(rows, cols, vecs, given):
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4 import FP4Tensor, PackedBuffers
    x = _bf(rows, cols)
    shape = {0: lambda: torch.ones(cols, device="cuda"), 1: lambda: torch.ones(1, cols, device="cuda"),
             2: lambda: torch.ones(cols, device="cuda", dtype=torch.float64),
             3: lambda: torch.ones(2 * cols, device="cuda")[::2]}
    v = {k: shape[i]() for k, i in vecs.items()}

    def call():
        out = PackedBuffers(rows, cols, "cuda") if given else None
        t = FP4Tensor.from_norm_mod(x, out=out, **v)
        slots = [t._gscale, t._amax] if rows else []      # an empty tensor's scale is not written
        return [t._data, *slots, t._rows, t._cols, t._shape, t._scales, t._scales_swz]
    if cols % 16 or (given and rows == 0):
        with pytest.raises(Exception):
            call()
            raise RuntimeError
    else:
        assert _same(*_both(call))


def test_gemm_and_attention():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4 as nv
    a, b = nv.FP4Tensor.from_bfloat16(_bf(100, 256)), nv.FP4Tensor.from_bfloat16(_bf(72, 256))
    y = _bf(100, 72)
    for kw in ({}, dict(bias=_bf(72)), dict(C=y, beta=0.5), dict(out=torch.empty_like(y)), dict(gelu=True),
               dict(gate=_bf(72).float()), dict(bias=_bf(71)), dict(C=y.t(), beta=1.0), dict(out=y.float()),
               dict(bias=_bf(72).float()), dict(out=torch.empty(72, 100, device="cuda", dtype=torch.bfloat16)),
               dict(C=y), dict(out_amax=torch.zeros(1, device="cuda"))):
        assert _same(*_both(lambda: nv.fp4_gemm(a, b, **kw)))
    q, k, v = _bf(130, 2, 384).split(128, dim=-1)
    for args in ((q, k, v), (q, k.contiguous(), v), (q.float(), k, v), (q[:, :, ::2], k, v), (q[:, :1], k, v),
                 (q, k, v[:-1]), (q, k[:-1], v), (q, k.cpu(), v), (q.cpu(), k.cpu(), v.cpu())):
        assert _same(*_both(lambda: dit.attention_native(*args)))
    for slot in (torch.zeros(1, device="cuda"), torch.zeros(9, device="cuda")[3:4], torch.zeros(1), y,
                 torch.zeros(0, device="cuda"), torch.zeros(1, device="cuda", dtype=torch.float64)):
        assert _same(*_both(lambda: (dit.attention_native(q, k, v, amax=slot.zero_()), slot.clone())))


def test_dispatch_modes_and_function_transforms_are_left_alone():
    from torch._subclasses.fake_tensor import FakeTensorMode
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    x = _bf(32, 64)
    with FakeTensorMode(allow_non_fake_inputs=True):
        assert N.host.quantize(x, True, True) is None

    def probe(t):
        assert N.host.quantize(t, True, True) is None
        return t.sum()
    torch.vmap(probe)(torch.stack([x, x]))
