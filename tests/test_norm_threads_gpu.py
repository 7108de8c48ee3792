"""Norm + quantize from several threads with rows of different widths: what one thread asks of the runtime for its width
changes nothing for another's launch."""
import threading

import pytest
import torch

from helpers import student_t_bf16

pytestmark = pytest.mark.gpu


# of each pair one variant of the kernels; too many rows for one launch, or as many as fit
@pytest.mark.parametrize("sizes", [((5400, 3072), (3400, 5120)), ((1000, 3072), (600, 5120))])
def test_widths_of_a_thread_each(sizes):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import nvfp4 as nv
    xs = [student_t_bf16(s, s[1], device="cuda") for s in sizes]
    want = [nv.FP4Tensor.from_norm_mod(x) for x in xs]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for n in range(400):
                try:
                    got = nv.FP4Tensor.from_norm_mod(xs[i])
                except RuntimeError as e:
                    wrong.append((i, n, str(e)))
                    continue
                if n % 40 == 0:
                    stream.synchronize()
                    if not (torch.equal(got.quantized_data(), want[i].quantized_data())
                            and torch.equal(got.scale_factors_swizzled(), want[i].scale_factors_swizzled())):
                        wrong.append((i, n, "bytes"))
            stream.synchronize()
    threads = [threading.Thread(target=work, args=(i % 2,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    nv.check_status()
    assert not wrong, (len(wrong), wrong[:3])
