"""Arguments that the one-call norm + quantize refuses on any machine, before it looks at the device."""
import pytest

BAD_ARG = 1


@pytest.mark.parametrize("rows", [0, 1, 64, 4000, 27280])        # of either form
@pytest.mark.parametrize("missing", ["row_stats", "amax"])
def test_missing_buffers(rows, missing):
    from blackwell_diffusion_rtx6000_5090_i2v_b200 import _native as N
    assert N.status_string(BAD_ARG) == "bad argument"
    stats, amax = (None if missing == "row_stats" else 4096), (None if missing == "amax" else 4096)
    assert N.lib.nvfp4_norm_mod_bf16(4096, rows, 3072, None, None, None, None, 0, 1e-6, stats, amax, 4096, None, None,
                                     None, 4096, None, None) == BAD_ARG
