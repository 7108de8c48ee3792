"""The quantizer that holds the tensor in shared memory, and the sizes at which the forms meet: byte for byte the
maximum and the packing in two calls, over poisoned buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(one, x, rows, cols, linear=True, swizzled=True, shift=0, part=None, check=True):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    dev = x.device
    slots = torch.full((2,), float("nan"), device=dev)
    part = torch.full((N.AMAX_PARTIALS,), float("nan"), device=dev) if part is None else part
    data = torch.full((rows * cols // 2 + 16,), 0xA5, dtype=torch.uint8, device=dev)
    lin = torch.full((rows * cols // 16 + 16,), 0xA5, dtype=torch.uint8, device=dev) if linear else None
    swz = torch.full((N.swizzled_scale_bytes(rows, cols) + 16,), 0xA5, dtype=torch.uint8, device=dev)
    p_swz = swz.data_ptr() + shift if swizzled else None
    amax, gs, st = slots.data_ptr(), slots.data_ptr() + 4, N.stream_ptr()
    if one:
        rc = N.lib.nvfp4_amax_quantize_bf16(x.data_ptr(), rows, cols, amax, data.data_ptr(), N.ptr(lin), p_swz, gs,
                                            part.data_ptr(), st)
    else:
        rc = N.lib.nvfp4_amax_bf16(x.data_ptr(), rows * cols, amax, st)
        rc = rc or N.lib.nvfp4_quantize_bf16(x.data_ptr(), rows, cols, amax, data.data_ptr(), N.ptr(lin), p_swz, gs, st)
    assert rc == 0
    if check:
        torch.cuda.synchronize()
    return [t for t in (data, lin, swz, slots) if t is not None]


@pytest.mark.parametrize("rows,cols", [
    (64, 4096), (65, 4096), (85, 3072), (86, 3072),      # either side of four blocks a thread of a cluster
    (128, 4096), (129, 4096), (1, 262160), (300, 272),
    (296, 8192), (296, 8208),                            # one block a thread of the grid, and a few over
    (1480, 9840), (1776, 8192), (1776, 8208),            # the last that fits, and the first that does not
    (700, 14336), (1700, 8192), (900, 14336), (100, 13824),
    (1536, 5120), (1537, 5120), (2500, 5120),            # rows of a CTA's width: the last that take one launch, and rows
])
def test_forms_agree_at_their_edges(rows, cols):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, cols, generator=g, device="cuda") * 3).bfloat16()
    x.view(-1)[-1] = 100.0                               # the maximum in the last block
    for a, b in zip(_run(True, x, rows, cols), _run(False, x, rows, cols)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", [dict(linear=False), dict(swizzled=False), dict(shift=1), dict(shift=4)])
@pytest.mark.parametrize("offset", [0, 8])
def test_buffers_a_caller_may_give(form, offset):
    x = torch.randn(600 * 4096 + 8, device="cuda").bfloat16()[offset:offset + 600 * 4096].view(600, 4096)
    for a, b in zip(_run(True, x, 600, 4096, **form), _run(False, x, 600, 4096, **form)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("rows,cols,ctas", [
    (64, 4096, 0),                          # the one-cluster form
    (128, 4096, 64), (600, 4096, 150), (1536, 5120, 240), (700, 14336, 245), (900, 14336, 263), (1700, 8192, 284), (1776, 8192, 296),
    (1480, 9840, 0), (1776, 8208, 0), (27280, 14336, 0),    # more than the shared memory holds: the maximum in a pass of its own
])
def test_which_form_is_taken(rows, cols, ctas, graph):
    """Each CTA of the one-launch form leaves its maximum among the partial ones, and nothing else does at these
    widths."""
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    part = torch.full((N.AMAX_PARTIALS,), float("nan"), device="cuda")
    want = _run(False, x, rows, cols)
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = _run(True, x, rows, cols, part=part, check=False)
        for _ in range(3):
            g.replay()
    else:
        got = _run(True, x, rows, cols, part=part)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert int((~torch.isnan(part)).sum()) == ctas and not bool(torch.isnan(part[:ctas]).any())


@pytest.mark.parametrize("what", ["inf", "-inf", "nan", "nan block", "largest", "all nan"])
@pytest.mark.parametrize("rows,cols", [(600, 4096), (50, 16400)])
def test_special_values(rows, cols, what):
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    if what == "nan block":
        x[rows // 2, 32:48] = float("nan")
    elif what == "all nan":
        x[:] = float("nan")
    elif what == "largest":
        x[3], x[4, ::2] = torch.finfo(torch.bfloat16).max, torch.finfo(torch.bfloat16).min
    else:
        x[rows // 3, cols // 2] = float(what)
    for a, b in zip(_run(True, x, rows, cols), _run(False, x, rows, cols)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


def test_beside_other_kernels_that_want_the_whole_gpu():
    """Two one-launch quantizers, a one-launch norm and an attention on a stream each: the grids that meet share
    the GPU with one another and with a kernel that does not."""
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N, dit
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4 import FP4Tensor, PackedBuffers
    sizes = {(1700, 8192): 284, (900, 14336): 263}       # and the CTAs of their one launch
    xs = [torch.randn(s, device="cuda").bfloat16() for s in sizes]
    y = torch.randn(4096, 3072, device="cuda").bfloat16()
    heads = y.view(4096, 24, 128)
    partials = [[], []]

    def quantize(i):
        out = PackedBuffers(*xs[i].shape, "cuda", linear_scales=True)
        partials[i].append(out.partials.fill_(float("nan")))
        return FP4Tensor.from_bfloat16(xs[i], out=out)
    calls = [lambda: quantize(0), lambda: quantize(1),
             lambda: FP4Tensor.from_norm_mod(y), lambda: dit.attention_native(heads, heads, heads)]
    want = [c() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    got = []
    for _ in range(30):
        for st, c in zip(streams, calls):
            with torch.cuda.stream(st):
                got.append(c())
    torch.cuda.synchronize()
    N.check_status()
    for i, t in enumerate(got):
        w = want[i % len(calls)]
        if isinstance(t, torch.Tensor):
            assert torch.equal(t, w)
        else:
            assert torch.equal(t._data, w._data) and torch.equal(t._scales_swz, w._scales_swz)
            assert torch.equal(t._gscale, w._gscale)
    # that each quantizer was one launch: its CTAs alone leave partial maxima
    for parts, ctas in zip(partials, sizes.values()):
        assert len(parts) == 31 and all(int((~torch.isnan(p)).sum()) == ctas for p in parts)
