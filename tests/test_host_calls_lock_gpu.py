"""The native calls and the interpreter: other threads run while a call waits, and errors are torch's."""
import sys
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ["linear", "quantize", "norm_quantize", "dequantize", "gemm", "attention"]


def _operands():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N, nvfp4 as nv, nvfp4_linear_cpp as L
    N.status_word(torch.device("cuda", torch.cuda.current_device()))
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(8192, 3072, generator=g, device="cuda").bfloat16()
    w = torch.randn(3072, 3072, generator=g, device="cuda").bfloat16()
    q = L.quantized_weight(w)
    p = nv.FP4Tensor.from_bfloat16(x)
    heads = x.view(8192, 24, 128)
    calls = [
        lambda: N.host.linear(x, w, q._data, q._scales_swz, q._gscale, None, None, None, False),
        lambda: N.host.quantize(x, True, True),
        lambda: N.host.norm_quantize(x, None, None, None, None, False, 1e-6, False, None),
        lambda: N.host.dequantize(p._data, p._scales, p._amax, 8192, 3072, [8192, 3072]),
        lambda: N.host.gemm(p._data, q._data, p._scales_swz, q._scales_swz, p._gscale, q._gscale, 8192, 3072, 3072, 1.0,
                            0.0, None, None, None, False, None, None),
        lambda: N.host.attention(heads, heads[:1024], heads[:1024], None, None),
    ]
    return dict(zip(NAMES, calls))


@pytest.mark.parametrize("name", NAMES)
def test_other_threads_run_while_a_launch_waits(name):
    """With a switch interval of an hour a thread gets the interpreter only where another one lets go of it; the
    calls outrun the GPU until the queue of launches is full and each of them waits for a free place."""
    call = _operands()[name]
    assert call() is not None
    torch.cuda.synchronize()
    ran, stop = [0], threading.Event()

    def other():
        while not stop.is_set():
            ran[0] += 1
            time.sleep(0)                    # lets go of the interpreter

    interval = sys.getswitchinterval()
    t = threading.Thread(target=other)
    t.start()
    try:
        sys.setswitchinterval(3600.0)
        before = ran[0]
        for _ in range(2500):
            call()
        during = ran[0] - before
    finally:
        sys.setswitchinterval(interval)
        stop.set()
        t.join()
        torch.cuda.synchronize()
    assert during > 0


def test_threads_with_a_stream_each():
    calls = _operands()
    streams = {name: torch.cuda.Stream() for name in calls}
    want = {name: call() for name, call in calls.items()}
    torch.cuda.synchronize()
    wrong = []

    def work(name):
        with torch.cuda.stream(streams[name]):
            for _ in range(20):
                got = calls[name]()
                streams[name].synchronize()
                pairs = zip(got, want[name]) if isinstance(got, tuple) else [(got, want[name])]
                if not all(torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b for a, b in pairs):
                    wrong.append(name)
    threads = [threading.Thread(target=work, args=(n,)) for n in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_an_allocation_that_does_not_fit():
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    x = torch.randn(4096, 3072, device="cuda").bfloat16()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _, total = torch.cuda.mem_get_info()
    torch.cuda.set_per_process_memory_fraction(min(1.0, (torch.cuda.memory_reserved() + (1 << 20)) / total))
    try:
        with pytest.raises(torch.OutOfMemoryError):
            held = [N.host.quantize(x, True, True) for _ in range(64)]
            del held
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    with pytest.raises(RuntimeError, match="not 16-byte aligned"):
        N.host.quantize(x.view(-1)[12:12 + 3072], True, True)
