"""The norm + quantize call that keeps its rows in shared memory (``nvfp4_norm_mod_bf16``) against the two sweeps,
byte for byte: row counts at the edges of a group, of a CTA's share and of what fits, widths with and without
a pad of K-blocks and with one and two blocks a thread, and buffers that send it to the two sweeps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(one, x, vecs, rms, linear=True, swizzled=True, shift_swz=0, partials=True, stats=None, check=True):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    rows, cols = x.shape
    dev = x.device
    f32 = dict(dtype=torch.float32, device=dev)
    stats = torch.empty(rows, 2, **f32) if stats is None else stats
    slots = torch.full((2,), float("nan"), **f32)
    part = torch.full((N.AMAX_PARTIALS,), float("nan"), **f32)
    data = torch.full((rows * cols // 2 + 16,), 0xA5, dtype=torch.uint8, device=dev)
    lin = torch.full((rows * cols // 16 + 16,), 0xA5, dtype=torch.uint8, device=dev) if linear else None
    n_swz = N.swizzled_scale_bytes(rows, cols)
    swz = torch.full((n_swz + 16,), 0xA5, dtype=torch.uint8, device=dev) if swizzled else None
    p_swz = swz.data_ptr() + shift_swz if swizzled else None
    w, b, sc, sh = (N.ptr(v) for v in vecs)
    st, status = N.stream_ptr(), N.status_word(dev).data_ptr()
    amax, gs = slots.data_ptr(), slots.data_ptr() + 4
    if one:
        rc = N.lib.nvfp4_norm_mod_bf16(x.data_ptr(), rows, cols, w, b, sc, sh, rms, 1e-6, stats.data_ptr(), amax,
                                       data.data_ptr(), N.ptr(lin), p_swz, gs,
                                       part.data_ptr() if partials else None, status, st)
    else:
        rc = N.lib.nvfp4_norm_mod_amax_bf16(x.data_ptr(), rows, cols, w, b, sc, sh, rms, 1e-6, stats.data_ptr(), amax,
                                            None, status, st)
        rc = rc or N.lib.nvfp4_norm_mod_quantize_bf16(x.data_ptr(), rows, cols, w, b, sc, sh, stats.data_ptr(), amax,
                                                      data.data_ptr(), N.ptr(lin), p_swz, gs, status, st)
    assert rc == 0
    if check:
        N.check_status()
    return [t for t in (data, lin, swz, slots) if t is not None]


def _inputs(rows, cols, kind, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn(rows, cols, generator=g, device="cuda") * 1.5 + 0.2).bfloat16()
    v = [torch.randn(cols, generator=g, device="cuda") * 0.2 for _ in range(4)]
    return x, [1 + v[0] if kind & 1 else None, v[1] if kind & 1 else None, v[2] if kind & 2 else None,
               v[3] if kind & 2 else None]


@pytest.mark.parametrize("rows,cols,kind", [
    (1, 16, 0), (1, 3072, 2), (2, 3072, 1), (3, 3072, 3), (147, 272, 2), (149, 2528, 3), (255, 4096, 2), (257, 5120, 1),
    (740, 3072, 2), (1481, 3072, 2), (1222, 3936, 2), (4436, 3072, 2), (4445, 3072, 1),    # the last of the full share
    (4730, 3072, 2), (4800, 3072, 2),                                                    # what fits, and does not
    (64, 6400, 3), (33, 16384, 2), (130, 16368, 0), (20001, 128, 1),
])
@pytest.mark.parametrize("rms", [0, 1])
def test_one_launch_equals_two_sweeps(rows, cols, kind, rms):
    x, vecs = _inputs(rows, cols, kind, rows + cols)
    for a, b in zip(_run(True, x, vecs, rms), _run(False, x, vecs, rms)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", [dict(linear=False), dict(swizzled=False), dict(shift_swz=1), dict(shift_swz=4),
                                  dict(partials=False)])
def test_buffers_a_caller_may_give(form):
    x, vecs = _inputs(300, 1040, 2, 5)
    for a, b in zip(_run(True, x, vecs, 0, **form), _run(False, x, vecs, 0, **form)):
        assert torch.equal(a, b)


def test_rows_of_zeros():
    x, vecs = _inputs(200, 3072, 2, 6)
    x[17] = 0
    for a, b in zip(_run(True, x, vecs, 0), _run(False, x, vecs, 0)):
        assert torch.equal(a, b)
    z = torch.zeros(64, 1024, device="cuda", dtype=torch.bfloat16)
    for a, b in zip(_run(True, z, [None] * 4, 1), _run(False, z, [None] * 4, 1)):
        assert torch.equal(a, b)


def test_two_streams_and_a_graph():
    from blackwell_diffusion_rtx6000_5090_i2v_b200.nvfp4 import FP4Tensor
    xs = [_inputs(1500, 3072, 0, s)[0] for s in (1, 2)]
    want = [FP4Tensor.from_norm_mod(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(10):
        got = []
        for st, x in zip(streams, xs):
            with torch.cuda.stream(st):
                got.append(FP4Tensor.from_norm_mod(x))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a._data, b._data) and torch.equal(a._scales_swz, b._scales_swz)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        t = FP4Tensor.from_norm_mod(xs[0])
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(t._data, want[0]._data) and torch.equal(t._gscale, want[0]._gscale)


def _one_launch(rows, cols, kind, graph=False):
    """Whether the call took the one-launch form, which leaves the row statistics alone; the same bytes either way."""
    x, vecs = _inputs(rows, cols, kind, rows)
    want = _run(False, x, vecs, 0)
    stats = torch.full((rows, 2), float("nan"), device="cuda")
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = _run(True, x, vecs, 0, stats=stats, check=False)
        g.replay()
    else:
        got = _run(True, x, vecs, 0, stats=stats)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    untouched = torch.isnan(stats)
    assert bool(untouched.all()) or not bool(untouched.any())
    return bool(untouched.all())


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("rows,cols,kind,one", [
    # two CTAs an SM by their rows alone, one with their own shared memory and the reserve added
    (3552, 4096, 2, True), (3553, 4096, 2, False), (4144, 4096, 2, False),
    (7992, 2048, 1, True), (7993, 2048, 1, False), (8288, 2048, 2, False),
    (4441, 3584, 2, False), (4736, 3584, 2, False),
    (1776, 7168, 2, True), (1777, 7168, 2, True), (2072, 7168, 2, True), (2073, 7168, 2, False),    # seven groups a CTA
    (593, 14336, 0, True), (888, 14336, 0, True), (889, 14336, 0, False),
    (4737, 3072, 0, True), (5328, 3072, 0, True), (5329, 3072, 0, False),                    # three CTAs an SM, not six
    (1, 16, 0, True), (20001, 128, 1, True), (27280, 3072, 2, False),
])
def test_where_the_rows_fit(rows, cols, kind, one, graph):
    assert _one_launch(rows, cols, kind, graph) == one


@pytest.mark.parametrize("rows,cols", [(300, 3072), (257, 5120), (70, 1536), (64, 10240), (1900, 272)])
@pytest.mark.parametrize("kind", [0, 2, 3])
@pytest.mark.parametrize("rms", [0, 1])
@pytest.mark.parametrize("what", ["inf", "-inf", "nan", "nan row", "largest", "all nan"])
def test_special_values(rows, cols, kind, rms, what):
    x, vecs = _inputs(rows, cols, kind, rows)
    if what == "nan row":
        x[rows // 2] = float("nan")
    elif what == "all nan":
        x[:] = float("nan")
    elif what == "largest":
        x[3] = torch.finfo(torch.bfloat16).max
        x[4, ::2] = torch.finfo(torch.bfloat16).min
    else:
        x[rows // 3, cols // 2] = float(what)
        x[rows - 1, 0] = float(what)                  # the row's first element, which the sums are taken around
    for a, b in zip(_run(True, x, vecs, rms), _run(False, x, vecs, rms)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
