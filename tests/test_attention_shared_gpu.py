"""Attention blocks whose keys several CTA pairs share (few blocks, or the blocks behind full waves of pairs),
and the walk of a pair from block to block: odd and even tile counts, one tile a block, ragged ends.
Bound as in test_attention_gpu: twice the library kernel's own error, 1e-2 at least."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v):
    o = torch.empty(q.shape, device="cuda", dtype=torch.float32)
    for h in range(q.shape[1]):
        s = q[:, h].float() @ k[:, h].float().t() / q.shape[-1] ** 0.5
        o[:, h] = torch.softmax(s, -1) @ v[:, h].float()
    return o


def _inputs(Lq, Lk, H, rise, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(L, H, 128, generator=g, device="cuda") for L in (Lq, Lk, Lk))
    if rise:       # the maximum of some rows rises by `rise` nats a key tile, so that every part has its own
        q[::3, :, 0] = 8.0
        k[:, :, 0] = (torch.arange(Lk, device="cuda") // 128 * (rise * 128 ** 0.5 / 8.0))[:, None]
    return q.bfloat16(), k.bfloat16(), v.bfloat16()


@pytest.mark.parametrize("Lq,Lk,H,rise", [
    (1000, 1000, 5, 0.0),          # 20 blocks by two pairs each, the last tile ragged
    (2500, 4096, 2, 0.0),          # 20 blocks of 32 tiles: by three
    (1000, 4000, 2, 0.0),          # 8 blocks of 32 tiles: by four
    (1000, 4000, 2, 9.0),          # ... whose maxima rise from part to part
    (9979, 2950, 2, 0.0),          # four blocks behind a wave of 74
    (9979, 2950, 2, -9.0),
    (9979, 1, 4, 0.0),             # one tile a block: each group of warps has every other block
    (20011, 300, 3, 5.0),          # three tiles a block: a block begins with either group
    (20011, 640, 2, 0.0),          # five
    (129, 1000, 1, 0.0),           # the pair's second CTA has one row
    (128, 1000, 1, 0.0),           # ... none
])
def test_shared_and_walked_blocks(Lq, Lk, H, rise):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4
    q, k, v = _inputs(Lq, Lk, H, rise, Lq + Lk + H)
    out = torch.full((Lq + 1, H, 128), 7.0, device="cuda", dtype=torch.bfloat16)   # a row that stays
    amax = torch.zeros(1, device="cuda")
    o = dit.attention_native(q, k, v, amax=amax, out=out[:Lq])
    nvfp4.check_status()
    r = _ref(q, k, v)
    old = dit.ATTENTION_BACKEND
    dit.ATTENTION_BACKEND = "library"
    try:
        err_lib = (dit.attention(q, k, v).float() - r).abs().max().item()
    finally:
        dit.ATTENTION_BACKEND = old
    err = (o.float() - r).abs().max().item()
    assert err <= max(2 * err_lib, 1e-2), (err, err_lib)
    assert amax.item() == o.float().abs().max().item()
    assert bool((out[Lq] == 7.0).all())
    # the parts are added in their order: the same bits every time
    again = torch.empty_like(o)
    for _ in range(8):
        dit.attention_native(q, k, v, out=again)
        assert torch.equal(again, o)


def test_strided_output_and_its_neighbours():
    """The output leaves in boxes of 32 rows: rows and columns beside a strided view stay as they are."""
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4
    q, k, v = _inputs(300, 700, 2, 0.0, 3)
    want = dit.attention_native(q, k, v)
    buf = torch.full((310, 5, 384), 7.0, device="cuda", dtype=torch.bfloat16)
    got = dit.attention_native(q, k, v, out=buf[4:304, 1:4:2, 128:256])
    nvfp4.check_status()
    assert torch.equal(got, want)
    buf[4:304, 1:4:2, 128:256] = 7.0
    assert bool((buf == 7.0).all())


def test_two_streams_and_a_graph():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4
    sets = [_inputs(2300, 2300, 9, 0.0, s) for s in (1, 2)]        # 81 blocks: a wave and seven shared ones
    want = [dit.attention_native(*s) for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for st, s in zip(streams, sets):
            with torch.cuda.stream(st):
                got.append(dit.attention_native(*s))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        x = dit.attention_native(*sets[0])
        y = dit.attention_native(x, x, x)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    nvfp4.check_status()
    assert torch.equal(x, want[0]) and torch.equal(y, dit.attention_native(want[0], want[0], want[0]))
