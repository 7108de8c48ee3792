"""The status word of a device is one tensor for good: kernels and the native calls keep its address."""
import threading
import time

import torch

from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N


def test_threads_that_ask_first_get_the_same_word(monkeypatch):
    zeros, told = torch.zeros, []

    class Torch:
        int32, device = torch.int32, torch.device

        @staticmethod
        def zeros(n, dtype, device):
            time.sleep(0.05)                       # an allocation lets other threads run
            return zeros(n, dtype=dtype)

    class Host:
        @staticmethod
        def set_status(device, word):
            time.sleep(0.01)
            told.append((device, word))
    monkeypatch.setattr(N, "torch", Torch)
    monkeypatch.setattr(N, "host", Host)
    monkeypatch.setattr(N, "_status_words", {})
    got = []
    threads = [threading.Thread(target=lambda: got.append(N.status_word(torch.device("cuda", 3)))) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 8 and all(w is got[0] for w in got)
    assert len(told) == 1 and told[0][0] == 3 and told[0][1] is got[0]
    assert N.status_word(torch.device("cuda", 3)) is got[0]
