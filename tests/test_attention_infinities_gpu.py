"""Keys whose scores are -inf (a mask carried by one dimension of q and k), in whole key tiles: at the start of a
block's keys, at the start of a part of them that a pair of CTAs has, in all but one key.  Bound as in
test_attention_gpu: twice the library kernel's own error, 1e-2 at least; NaN where softmax is one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(q, k, v):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4
    o = dit.attention_native(q, k, v)
    nvfp4.check_status()
    want, err_lib = torch.empty(q.shape, device="cuda", dtype=torch.float64), 0.0
    lib = torch.nn.functional.scaled_dot_product_attention(*(t.transpose(0, 1).unsqueeze(0) for t in (q, k, v)))
    lib = lib.squeeze(0).transpose(0, 1).double()
    for h in range(q.shape[1]):
        s = (q[:, h].float() @ k[:, h].float().t()).double() / q.shape[-1] ** 0.5     # scores of 32 bits, as everywhere
        want[:, h] = torch.softmax(s, -1) @ v[:, h].double()
    assert torch.equal(torch.isnan(o), torch.isnan(want))
    ok = ~torch.isnan(want)
    if bool(ok.any()):
        both = ok & ~torch.isnan(lib)
        if bool(both.any()):
            err_lib = (lib[both] - want[both]).abs().max().item()
        assert (o.double()[ok] - want[ok]).abs().max().item() <= max(2 * err_lib, 1e-2)
    return o


def _inputs(Lq, Lk, H, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(L, H, 128, generator=g, device="cuda").bfloat16() for L in (Lq, Lk, Lk))
    q[:, :, 0] = 1.0
    return q, k, v


SHAPES = [(1000, 1000, 5),        # by two pairs, eight tiles
          (2500, 4096, 2),        # by three
          (1000, 4000, 2),        # by four
          (9979, 2950, 2),        # walked, and four shared blocks behind
          (20011, 300, 3),        # three tiles a block
          (100, 100, 1), (300, 129, 2)]


@pytest.mark.parametrize("Lq,Lk,H", SHAPES)
@pytest.mark.parametrize("mask", ["second half", "first tile", "first two tiles", "tiles by turns", "all but the last",
                                  "all but the first", "a tile in the middle", "all"])
@pytest.mark.parametrize("low", [float("-inf"), torch.finfo(torch.bfloat16).min])
def test_masked_keys(Lq, Lk, H, mask, low):
    q, k, v = _inputs(Lq, Lk, H)
    n = torch.arange(Lk, device="cuda")
    masked = {"second half": n >= Lk // 2 - 20, "first tile": n < 128, "first two tiles": n < 256,
              "tiles by turns": n // 128 % 2 == 0, "all but the last": n < Lk - 1, "all but the first": n > 0,
              "a tile in the middle": n // 128 == Lk // 256, "all": n >= 0}[mask]
    if low != float("-inf"):
        q[:, :, 0] = 4.0                                # the product overflows
    k[:, :, 0] = torch.where(masked, low, 0.0).bfloat16()[:, None]
    _check(q, k, v)


@pytest.mark.parametrize("Lq,Lk,H", SHAPES)
def test_rows_of_infinite_scores_keep_to_themselves(Lq, Lk, H):
    q, k, v = _inputs(Lq, Lk, H)
    k[:, :, 0] = 0.0
    k[Lk // 2:, :, 0] = float("-inf")
    q[::3, :, 0] = -1.0                                 # +inf there: NaN in these rows alone
    o = _check(q, k, v)
    assert bool(torch.isnan(o[::3]).all())


@pytest.mark.parametrize("Lq,Lk,H", [(130, 128, 1), (130, 300, 2), (1000, 1000, 5)])
def test_a_key_with_nan_reaches_every_row(Lq, Lk, H):
    """Whichever way its exponential takes: most element pairs through the special-function unit, some through a
    polynomial."""
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit, nvfp4
    q, k, v = _inputs(Lq, Lk, H)
    for key in [*range(128), Lk - 1]:
        bad = k.clone()
        bad[key, :, 5] = float("nan")
        o = dit.attention_native(q, bad, v)
        assert bool(torch.isnan(o).all()), key
    nvfp4.check_status()
