"""What ``attention_native`` refuses before any address reaches the kernel: on stand-ins for CUDA tensors, with
the library replaced by one that must not be called, so that it runs without a GPU."""
import math

import pytest
import torch

from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
from blackwell_diffusion_rtx6000_5090_i2v_b200 import dit


class Fake:
    """The attributes of a contiguous tensor that the checks look at."""

    def __init__(self, *shape, dtype=torch.bfloat16, device="cuda:0", inner=1):
        self.shape, self.dtype, self.device, self.inner = shape, dtype, torch.device(device), inner
        self.is_cuda = self.device.type == "cuda"

    def dim(self):
        return len(self.shape)

    def numel(self):
        return math.prod(self.shape)

    def stride(self, i):
        return math.prod(self.shape[i + 1:]) * self.inner

    def data_ptr(self):
        return 4096


class Called(Exception):
    pass


class Lib:
    def __getattr__(self, name):
        raise Called(name)


class Declines:
    def attention(self, *a):
        return None


@pytest.fixture(autouse=True)
def no_gpu(monkeypatch):
    import contextlib
    monkeypatch.setattr(N, "lib", Lib())
    monkeypatch.setattr(N, "host", Declines())
    monkeypatch.setattr(N, "status_word", lambda device: Fake(1))
    monkeypatch.setattr(N, "stream_ptr", lambda: 0)
    monkeypatch.setattr(N, "device_guard", lambda device: contextlib.nullcontext(), raising=False)


def _qkv(Lk=20, Lv=20):
    return Fake(10, 2, 128), Fake(Lk, 2, 128), Fake(Lv, 2, 128)


@pytest.mark.parametrize("args,kw", [
    (_qkv(Lv=19), {}), (_qkv(Lk=19), {}),
    ((Fake(10, 2, 128), Fake(20, 2, 128, device="cpu"), Fake(20, 2, 128)), {}),
    ((Fake(10, 2, 128), Fake(20, 2, 128), Fake(20, 2, 128, device="cuda:1")), {}),
    (tuple(Fake(20, 2, 128, device="cpu") for _ in range(3)), {}),
    (_qkv(), dict(out=Fake(9, 2, 128))), (_qkv(), dict(out=Fake(10, 1, 128))), (_qkv(), dict(out=Fake(10, 2, 64))),
    (_qkv(), dict(out=Fake(10, 256))), (_qkv(), dict(out=Fake(10, 2, 128, dtype=torch.float32))),
    (_qkv(), dict(out=Fake(10, 2, 128, device="cpu"))), (_qkv(), dict(out=Fake(10, 2, 128, inner=2))),
    (_qkv(), dict(amax=Fake(1))), (_qkv(), dict(amax=Fake(0, dtype=torch.float32))),
    (_qkv(), dict(amax=Fake(1, dtype=torch.float32, device="cpu"))),
])
def test_refused(args, kw):
    with pytest.raises(ValueError):
        dit.attention_native(*args, **kw)


@pytest.mark.parametrize("kw", [dict(), dict(amax=Fake(1, dtype=torch.float32)), dict(out=Fake(10, 2, 128)),
                                dict(out=Fake(11, 2, 128))])
def test_still_taken(kw):
    kw.setdefault("out", Fake(10, 2, 128))
    with pytest.raises(Called):
        dit.attention_native(*_qkv(), **kw)
