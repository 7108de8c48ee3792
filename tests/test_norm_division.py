"""The norm's division by the row length (csrc/norm_quantize.cu: div_by), a product and a residual correction, is the
IEEE quotient for every row length that it takes."""
import numpy as np


def test_product_and_correction_equal_the_quotient():
    rng = np.random.default_rng(1)
    for n in range(16, 16385, 16):
        x = np.ldexp(rng.uniform(1, 2, 3000), rng.integers(-80, 120, 3000)).astype(np.float32)
        x *= rng.choice(np.array([-1, 1], np.float32), x.size)
        nf = np.float32(n)
        inv = np.float32(1) / nf
        q0 = x * inv
        # both fused operations: the products are exact in 64 bits, the sums in the extended type
        r = (x.astype(np.float64) - n * q0.astype(np.float64)).astype(np.float32)
        q = (r.astype(np.longdouble) * np.longdouble(inv) + q0).astype(np.float32)
        assert np.array_equal(q, x / nf), n
